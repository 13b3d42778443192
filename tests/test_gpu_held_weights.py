"""The CTA-pair kernel that holds its weights' tile in shared memory (results of 144 MB and more, K of up to 1024) against the same product in blocks of
rows, which are too small for it and take the general route: the results are whole sums and two roundings, so they are equal bit for bit."""
import ctypes
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(dev, m, k, n, unsigned=False):
    g = torch.Generator(device=dev).manual_seed(m + k + n)
    a = torch.randint(0, 256, (m, k), generator=g, device=dev, dtype=torch.uint8) if unsigned else torch.randint(-127, 128, (m, k), generator=g, device=dev).to(torch.int8)
    w = torch.randint(-127, 128, (n, k), generator=g, device=dev).to(torch.int8)
    return g, a, w, torch.randn(n, generator=g, device=dev)


def _route(call):
    """The kernel of the one product that `call` launches: "held", "pair" (the CTA-pair kernel that streams both operands) or its name."""
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    check(lib().mi8_kernel_times_begin())
    try:
        call()
    finally:
        records, count = (Mi8KernelTime * 4)(), ctypes.c_int(0)
        check(lib().mi8_kernel_times_end(records, 4, ctypes.byref(count)))
    assert count.value == 1 and records[0].launches == 1
    name = records[0].name.decode()
    pair = re.search(r"mi8_gemm_pair_kernelILb[01]ELi\dELb([01])E", name)
    return name if pair is None else "held" if pair.group(1) == "1" else "pair"


def _status():
    from marian_dev_b200 import ops
    return ops.poll_status()


# K blocks: fewer than the ring has stages, an odd number, a ragged last one, all eight; one and several activation tiles of a share; N odd (no paired stores);
# M of one row more than a tile
@pytest.mark.parametrize("m,k,n,half", [(1300, 80, 29101, False), (1281, 272, 30720, False), (2049, 1024, 37002, True), (6100, 640, 6200, False), (1200, 896, 63000, True)])
@pytest.mark.parametrize("relu", [False, True])
def test_equals_blocks_of_rows(cuda_device, m, k, n, half, relu):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    _, a, w, bias = _operands(cuda_device, m, k, n)
    q = torch.tensor([31.7, 211.3], device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    dtype = torch.float16 if half else torch.float32

    def product(rows, out):
        assert out.numel() * out.element_size() >= 144 << 20 or rows.shape[0] < m
        check(lib().mi8_multiply_i8(rows.data_ptr(), w.data_ptr(), rows.shape[0], n, k, q.data_ptr(), q[1:].data_ptr(), 1.0, bias.data_ptr(), int(relu),
                                    out.data_ptr(), 1 if half else 0, None, ws.ptr, ws.nbytes, stream))

    got = torch.full((m, n), float("nan"), dtype=dtype, device=cuda_device)
    product(a, got)
    want = torch.full((m, n), float("nan"), dtype=dtype, device=cuda_device)
    for r in range(0, m, 500):
        product(a[r:r + 500], want[r:r + 500])
    assert torch.equal(got, want) and _status() == 0


@pytest.mark.parametrize("limit", [0, 255, 256, 1300, 2300])
def test_rows_below_a_limit_are_kept(cuda_device, limit):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    m, k, n = 2300, 384, 17000
    _, a, w, bias = _operands(cuda_device, m, k, n)
    q = torch.tensor([31.7, 211.3], device=cuda_device)
    words = torch.tensor([7, 7, 8], dtype=torch.int32, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream

    def product(rows, out, other, below):
        check(lib().mi8_multiply_i8_rows_from(rows.data_ptr(), w.data_ptr(), rows.shape[0], n, k, q.data_ptr(), q[1:].data_ptr(), 1.0, bias.data_ptr(), 0,
                                              out.data_ptr(), 0, ws.ptr, ws.nbytes, stream, words.data_ptr(), other.data_ptr(), below, 0))

    want = torch.empty((m, n), device=cuda_device)
    for r in range(0, m, 500):
        product(a[r:r + 500], want[r:r + 500], words[2:], 0)
    for other, kept in ((words[1:], limit // 256 * 256), (words[2:], 0)):
        got = torch.full((m, n), 12345.0, device=cuda_device)
        product(a, got, other, limit)
        assert bool((got[:kept] == 12345.0).all()) and torch.equal(got[kept:], want[kept:])
    assert _status() == 0


def test_packed8(cuda_device):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    m, k, n = 1400, 768, 28000
    g, a, w, bias = _operands(cuda_device, m, k, n, unsigned=True)
    scale_a, scale_b = torch.rand(m, generator=g, device=cuda_device), torch.rand(n, generator=g, device=cuda_device)
    zp_a, sum_a = (torch.randint(0, 256, (m,), generator=g, device=cuda_device, dtype=torch.int32) for _ in range(2))
    zp_b, off_b = (torch.randint(-63, 64, (n,), generator=g, device=cuda_device, dtype=torch.int32) for _ in range(2))
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream

    def product(first, last, out):
        check(lib().mi8p_multiply(a[first:].data_ptr(), scale_a[first:].data_ptr(), zp_a[first:].data_ptr(), sum_a[first:].data_ptr(), w.data_ptr(),
                                  scale_b.data_ptr(), zp_b.data_ptr(), off_b.data_ptr(), last - first, n, k, bias.data_ptr(), 1, out[first:].data_ptr(), None,
                                  ws.ptr, ws.nbytes, stream, 0, 0))

    got, want = torch.empty((m, n), device=cuda_device), torch.empty((m, n), device=cuda_device)
    product(0, m, got)
    for r in range(0, m, 448):
        product(r, min(m, r + 448), want)
    assert torch.equal(got, want) and _status() == 0


# held only where every row of the results is whole 32-byte sectors, the parts of other rows' sectors at the tiles' edges being written too far apart (`shift`:
# bytes between a sector's start and the results'), and where no more than a ninth of the activation tiles is padding
@pytest.mark.parametrize("m,n,half,shift,route", [(1536, 25000, False, 0, "held"), (1536, 25004, False, 0, "pair"), (1536, 25001, False, 0, "pair"),
                                                  (1536, 25000, False, 16, "pair"), (2560, 31984, True, 0, "held"), (2560, 31992, True, 0, "pair"),
                                                  (2560, 31985, True, 0, "pair"), (2560, 31984, True, 2, "pair"),
                                                  (1366, 29104, False, 0, "held"), (1365, 29104, False, 0, "pair"), (1281, 30720, False, 0, "pair")])
def test_which_results(cuda_device, m, n, half, shift, route):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    k = 1024
    _, a, w, bias = _operands(cuda_device, m, k, n)
    q = torch.tensor([31.7, 211.3], device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    dtype, skip = (torch.float16, shift // 2) if half else (torch.float32, shift // 4)

    def product(rows, out):
        check(lib().mi8_multiply_i8(rows.data_ptr(), w.data_ptr(), rows.shape[0], n, k, q.data_ptr(), q[1:].data_ptr(), 1.0, bias.data_ptr(), 0,
                                    out.data_ptr(), 1 if half else 0, None, ws.ptr, ws.nbytes, stream))

    got = torch.full((m * n + skip,), float("nan"), dtype=dtype, device=cuda_device)[skip:].view(m, n)
    assert got.data_ptr() % 32 == shift
    assert _route(lambda: product(a, got)) == route
    want = torch.empty((m, n), dtype=dtype, device=cuda_device)
    for r in range(0, m, 512):
        product(a[r:r + 512], want[r:r + 512])
    assert torch.equal(got, want) and _status() == 0
