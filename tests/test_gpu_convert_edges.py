"""Weight conversion at the edges of its 128 x 32 tiles, with rows of W that are and are not 16-byte aligned and with K that is and is not a multiple of four,
against torch's arithmetic in float32 (one product, rounded half to even: exact)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [(4, 1), (6, 10), (127, 4), (128, 32), (128, 33), (129, 36), (130, 34), (132, 31), (252, 68), (257, 28), (1024, 124), (384, 4100)])
def test_prepare_b(cuda_device, k, n):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    w = torch.randn(k, n, generator=torch.Generator(device=cuda_device).manual_seed(k + n), device=cuda_device)
    bt = torch.full((k * n + 64,), 99, dtype=torch.int8, device=cuda_device)
    mult = torch.zeros(1, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    check(lib().mi8_prepare_b_f32(w.data_ptr(), k, n, 0, bt.data_ptr(), mult.data_ptr(), ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream))
    want_mult = torch.tensor([127.0], device=cuda_device) / w.abs().max()
    assert torch.equal(mult, want_mult)
    assert torch.equal(bt[:k * n].view(n, k), torch.clamp(torch.round(w * want_mult), -127, 127).to(torch.int8).T) and bool((bt[k * n:] == 99).all())
    assert ops.poll_status() == 0
