"""Rows of logits without a number have no candidates: no word or hypothesis outside the vocabulary and the beam leaves the n-best merge."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beam,batch,vocab,k", [(1, 2, 300, 2), (2, 3, 300, 2), (4, 2, 1003, 4), (3, 1, 100, 8)])
@pytest.mark.parametrize("all_rows", [True, False])
def test_rows_without_a_number(cuda_device, beam, batch, vocab, k, all_rows):
    from marian_dev_b200.binding import check, lib
    L = lib()
    rng = np.random.default_rng(vocab + k)
    rows = beam * batch
    logits = rng.standard_normal((rows, vocab)).astype(np.float32)
    prev = rng.standard_normal(rows).astype(np.float32)
    bad = np.arange(rows) < (rows if all_rows else (rows + 1) // 2)      # the first hypotheses of the sentences
    logits[bad] = np.nan
    stream = torch.cuda.current_stream().cuda_stream

    def merged(x, p):
        ld, pd = torch.from_numpy(x).to(cuda_device), torch.from_numpy(p).to(cuda_device)
        cs = torch.empty(rows, k, device=cuda_device)
        cw = torch.empty(rows, k, dtype=torch.int32, device=cuda_device)
        arrivals = torch.zeros(batch, dtype=torch.int32, device=cuda_device)
        outs = [torch.full((batch, k), 7, dtype=t, device=cuda_device) for t in (torch.float32, torch.int32, torch.int32) * 2]
        check(L.mi8g_lse_topk_nbest(ld.data_ptr(), beam, batch, vocab, k, pd.data_ptr(), cs.data_ptr(), cw.data_ptr(), arrivals.data_ptr(),
                                    *[o.data_ptr() for o in outs[:3]], stream))
        check(L.mi8g_nbest_merge(cs.data_ptr(), cw.data_ptr(), beam, batch, vocab, k, *[o.data_ptr() for o in outs[3:]], stream))
        torch.cuda.synchronize()
        return [o.cpu().numpy() for o in outs]
    got = merged(logits, prev)
    # a hypothesis without a number is as good as none: the same rows as dummies (score -inf)
    x, p = logits.copy(), prev.copy()
    x[bad], p[bad] = 0.0, -np.inf
    for a, b in zip(got, merged(x, p)):
        assert np.array_equal(a, b)
    if all_rows:
        assert np.all(got[0] == -np.inf) and not got[1].any() and not got[2].any()
