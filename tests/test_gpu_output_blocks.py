"""The output layer of up to 32 rows, whose write-back leaves the blocks' maxima and sums of the log-softmax: the step's n-best lists against
mi8g_lse_topk_nbest, which scans the step's own logits.  Scores, hypotheses and words are the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 16 and of 32 rows, full and not; vocabularies that end inside a block of 128 and at its edge, of one block, and of more blocks than there
# are SMs (several tiles per CTA); words that a bias of -inf rules out, a whole block of them among them
@pytest.mark.parametrize("rows", [1, 2, 16, 17, 31, 32])
@pytest.mark.parametrize("scheme,vocab", [("intgemm8", 100), ("intgemm8", 128), ("intgemm8", 1003), ("intgemm8", 21504), ("intgemm8", 32001),
                                          ("packed8avx512", 128), ("packed8avx512", 544), ("packed8avx512", 32000)])
def test_blocks_of_the_write_back(cuda_device, scheme, vocab, rows):
    from marian_dev_b200 import decoder, model, ops
    from marian_dev_b200.binding import check, lib
    L = lib()
    cfg = model.TransformerConfig(dim_emb=256, dim_ffn=256, heads=8, enc_depth=1, dec_depth=1, vocab=vocab)
    params = model.random_init(cfg, vocab + rows)
    bias = params["decoder_ff_logit_out_b"]
    bias[0, 3::17] = -np.inf
    if vocab > 300:
        bias[0, 128:256] = -np.inf
    net = decoder.Int8Transformer(cfg, params, cuda_device, scheme=scheme)
    beam = 2 if rows == 32 else 1
    batch = rows // beam
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=8, max_steps=8)
    check(L.mi8d_keep_logits(stepper.h, 1))
    g = torch.Generator(device="cuda").manual_seed(rows)
    stepper.start(torch.randn(batch, 7, cfg.dim_emb, generator=g, device=cuda_device), torch.zeros(batch, 7, device=cuda_device))
    k = 1 + rows % 8
    first = stepper.step(None, None, None, None, 1, batch, k)
    prev = np.random.default_rng(rows).standard_normal(rows).astype(np.float32)
    prev[batch:] = -np.inf                                    # (the second hypotheses are dummies)
    for step in range(2):
        if step == 0:
            n, b, scores, got = batch, 1, None, first
        else:
            n, b, scores = rows, beam, prev
            got = stepper.step(np.arange(rows) % batch, np.resize(first[2][:, 0], rows), np.arange(batch), scores, beam, batch, k)
        assert ops.poll_status() == 0
        cs, cw = torch.empty(n, k, device=cuda_device), torch.empty(n, k, dtype=torch.int32, device=cuda_device)
        arrivals = torch.zeros(batch, dtype=torch.int32, device=cuda_device)
        want = [torch.empty(batch, k, dtype=t, device=cuda_device) for t in (torch.float32, torch.int32, torch.int32)]
        prev_d = torch.zeros(n, device=cuda_device) if scores is None else torch.from_numpy(scores).to(cuda_device)
        check(L.mi8g_lse_topk_nbest(L.mi8d_last_logits(stepper.h), b, batch, vocab, k, prev_d.data_ptr(), cs.data_ptr(), cw.data_ptr(),
                                    arrivals.data_ptr(), *[w.data_ptr() for w in want], torch.cuda.current_stream().cuda_stream))
        for x, y in zip(got[:3], want):
            assert np.array_equal(x, y.cpu().numpy())
        assert np.isfinite(got[0][:, 0]).all()
