"""CTA-pair GEMM whose last wave of tiles is dealt out in halves, against 128-row tiles (exact: integer sums, the same two roundings): waves with one tile and with
half a wave of them, and the first count that is not halved; last tiles without a second half; odd columns and strides; several weights; both result types."""
import ctypes

import pytest
import torch

from tests.kernel_args import arguments

pytestmark = pytest.mark.gpu


def _names(call):
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    check(lib().mi8_kernel_times_begin())
    try:
        call()
    finally:
        records, count = (Mi8KernelTime * 4)(), ctypes.c_int(0)
        check(lib().mi8_kernel_times_end(records, 4, ctypes.byref(count)))
    return [r.name.decode() for r in records[:count.value]]


# pairs of SMs + 1, + half, + half and one tiles; two waves and some; M that ends in a tile's first and second half; N that ends inside a pair's first and second CTA
@pytest.mark.parametrize("tiles,n_tiles,m_cut,n_cut,k,half,halved", [
    (lambda p: p + 1, 1, 0, 0, 128, False, True), (lambda p: p + p // 2, 1, 0, 0, 272, False, True), (lambda p: p + p // 2 + 1, 1, 0, 0, 128, False, False),
    (lambda p: 2 * p, 1, 0, 0, 128, False, False), (lambda p: p, 1, 0, 0, 128, False, False), (lambda p: p + 5, 1, 200, 0, 1024, False, True),
    (lambda p: p + 5, 1, 60, 130, 1040, False, True), (lambda p: 2 * p + 8, 3, 129, 3, 384, False, True), (lambda p: 2 * p + 8, 3, 128, 1, 384, True, True),
    (lambda p: p + 9, 5, 1, 200, 2064, True, True)])
@pytest.mark.parametrize("relu", [False, True])
def test_last_wave(cuda_device, tiles, n_tiles, m_cut, n_cut, k, half, halved, relu):
    from marian_dev_b200 import ops
    pairs = torch.cuda.get_device_properties(cuda_device).multi_processor_count // 2
    count = tiles(pairs)
    m_tiles = -(-count // n_tiles)
    if (m_tiles * n_tiles) % pairs > pairs // 2 and halved:
        m_tiles -= 1
    m, n = 256 * m_tiles - m_cut, 256 * n_tiles - n_cut
    g = torch.Generator(device=cuda_device).manual_seed(m + k)
    x = ops.prepareA(torch.randn(m, k, generator=g, device=cuda_device))
    w = ops.prepareB(torch.randn(k, n, generator=g, device=cuda_device))
    b = torch.randn(n, generator=g, device=cuda_device)
    dtype = torch.float16 if half else torch.float32
    room = torch.full((m + 8, n), 7.0, dtype=dtype, device=cuda_device)
    names = _names(lambda: ops.multiply(x, w, b, relu=relu, out=room[:m], out_dtype=dtype, tile_m=512))
    assert len(names) == 1 and bool(arguments("mi8_gemm_pair_kernel", names[0])["kHalves"]) == halved
    assert torch.equal(room[:m], ops.multiply(x, w, b, relu=relu, out_dtype=dtype, tile_m=128)) and bool((room[m:] == 7.0).all())
    for _ in range(3):      # (launches that overlap)
        ops.multiply(x, w, b, relu=relu, out=room[:m], out_dtype=dtype, tile_m=512)
    assert torch.equal(room[:m], ops.multiply(x, w, b, relu=relu, out_dtype=dtype, tile_m=128)) and ops.poll_status() == 0


@pytest.mark.parametrize("n_each", [256, 384])
def test_several_weights(cuda_device, n_each):
    """Three weights in one launch; 384 columns each: a pair's CTAs in different segments."""
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import check, lib
    pairs = torch.cuda.get_device_properties(cuda_device).multi_processor_count // 2
    m, k, n_tiles = 256 * (-(-(pairs + 3) // (-(-3 * n_each // 256)))) - 100, 1024, -(-3 * n_each // 256)
    assert 0 < (-(-m // 256) * n_tiles) % pairs <= pairs // 2
    g = torch.Generator(device=cuda_device).manual_seed(n_each)
    x = ops.prepareA(torch.randn(m, k, generator=g, device=cuda_device))
    ws = [ops.prepareB(torch.randn(k, n_each, generator=g, device=cuda_device) * (i + 1)) for i in range(3)]
    all_w = torch.cat([w.data.reshape(-1) for w in ws])
    outs = [torch.empty(m, n_each, device=cuda_device) for _ in range(3)]
    biases = [torch.randn(n_each, generator=g, device=cuda_device) for _ in range(3)]
    space = ops.default_workspace(cuda_device)
    pointers = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])
    check(lib().mi8_multiply_i8_multi(x.data.data_ptr(), all_w.data_ptr(), m, n_each, k, 3, x.quant_mult.data_ptr(), pointers([w.quant_mult for w in ws]), 1.0,
                                      pointers(biases), 0, pointers(outs), 0, space.ptr, space.nbytes, torch.cuda.current_stream().cuda_stream))
    for i in range(3):
        assert torch.equal(outs[i], ops.multiply(x, ws[i], biases[i], tile_m=128))
    assert ops.poll_status() == 0
