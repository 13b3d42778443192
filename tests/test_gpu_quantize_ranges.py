"""Quantisation with a given abs-max, a warp's lanes side by side: lengths around a vector, a block's share and more than the grid takes in one turn, against
torch's arithmetic in float32 (one product, rounded half to even, saturated: exact)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 7, 16, 20, 1023, 4096, 4100, 3 * 4096 + 8, 1184 * 4096 + 4, 1200 * 4096 + 4095])
def test_lengths(cuda_device, n):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    g = torch.Generator(device=cuda_device).manual_seed(n)
    x = torch.randn(n, generator=g, device=cuda_device)
    slot = (x.abs().max() * 0.9).reshape(1)          # (some values saturate)
    q = torch.full((n + 64,), 99, dtype=torch.int8, device=cuda_device)
    mult = torch.zeros(1, device=cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    check(lib().mi8g_quantize_slot(x.data_ptr(), n, slot.data_ptr(), q.data_ptr(), mult.data_ptr(), stream))
    want_mult = torch.tensor(127.0, device=cuda_device) / slot
    assert torch.equal(mult, want_mult)
    assert torch.equal(q[:n], torch.clamp(torch.round(x * want_mult), -127, 127).to(torch.int8)) and bool((q[n:] == 99).all())
    q.fill_(99)
    check(lib().mi8_quantize_f32_i8(x.data_ptr(), n, mult.data_ptr(), q.data_ptr(), stream))
    assert torch.equal(q[:n], torch.clamp(torch.round(x * want_mult), -127, 127).to(torch.int8)) and bool((q[n:] == 99).all())
    assert ops.poll_status() == 0


# one CTA, the cluster with one and with two chunks per thread, threads and whole warps beyond the end; the maximum in the first or the last float
@pytest.mark.parametrize("n16", [1, 2, 31, 32, 33, 63, 511, 512, 513, 520, 1000, 4097, 8191, 8192, 8193, 9000, 12345, 16383, 16384])
@pytest.mark.parametrize("last", [False, True])
def test_maximum_and_quantisation_in_one_launch(cuda_device, n16, last):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    n = 16 * n16
    x = torch.rand(n, generator=torch.Generator(device=cuda_device).manual_seed(n16), device=cuda_device) - 0.5
    x[-1 if last else 0] = -0.75
    q = torch.full((n + 64,), 99, dtype=torch.int8, device=cuda_device)
    mult = torch.zeros(1, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    check(lib().mi8_prepare_a_f32(x.data_ptr(), n16, 16, q.data_ptr(), mult.data_ptr(), ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream))
    want_mult = torch.tensor([127.0], device=cuda_device) / x.abs().max()     # (by a tensor: torch divides by a number as a product with its reciprocal)
    assert torch.equal(mult, want_mult)
    assert torch.equal(q[:n], torch.clamp(torch.round(x * want_mult), -127, 127).to(torch.int8)) and bool((q[n:] == 99).all())
    assert ops.poll_status() == 0
