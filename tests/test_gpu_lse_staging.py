"""mi8g_lse_topk copies a warp's 1024 entries at a time to shared memory: rows that end inside, at and after such a piece and after
the pass of a whole block (32768, 16384 and 8192 entries), by 16 bytes and by the word, bit for bit the oracle's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 149, 300])   # 1024, 512 and 256 threads per row
@pytest.mark.parametrize("vocab", [1, 31, 1023, 1024, 1028, 8193, 16388, 32772, 33797])
@pytest.mark.parametrize("shift", [0, 1])         # the logits' first entry on and off a 16-byte boundary
def test_rows_that_end_at_the_edges_of_the_pieces(cuda_device, oracle, rows, vocab, shift):
    from marian_dev_b200.binding import check, lib
    rng = np.random.default_rng(vocab + rows)
    x = (4 * rng.standard_normal((rows, vocab))).astype(np.float32)
    x[-1, -1] = 30.0                              # the very last entry is the best of its row
    k = min(vocab, 6)
    room = torch.full((rows * vocab + 8,), np.inf, dtype=torch.float32, device=cuda_device)   # an entry read from beyond a row's end shows
    logits = room[shift:shift + rows * vocab]
    logits.copy_(torch.from_numpy(x).flatten())
    cs = torch.empty(rows, k, device=cuda_device)
    cw = torch.empty(rows, k, dtype=torch.int32, device=cuda_device)
    check(lib().mi8g_lse_topk(logits.data_ptr(), rows, vocab, k, None, cs.data_ptr(), cw.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    cs_w, cw_w = oracle.lse_topk(x, k)
    assert np.array_equal(cs.cpu().numpy(), cs_w)
    assert np.array_equal(cw.cpu().numpy(), cw_w)
