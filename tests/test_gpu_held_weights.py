"""The CTA-pair kernel that holds its weights' tile in shared memory (results of 144 MB and more, K of up to 1024) against the same product in blocks of
rows, which are too small for it and take the general route: the results are whole sums and two roundings, so they are equal bit for bit.  Every test looks at
the name of the kernel that ran.  The plan chooses the CTA-pair kernel itself from eight K blocks on; with fewer it is asked for."""
import ctypes
import re

import pytest
import torch

pytestmark = pytest.mark.gpu
PAIR = 512        # the tile width that asks for the CTA-pair kernel
ONE_WARP = -2


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


class _Products:
    """Products of int8 operands of one shape, a call of mi8_multiply_i8_ex each."""

    def __init__(self, dev, m, k, n, half=False, relu=False, tile=0):
        from marian_dev_b200 import ops
        self.shape, self.dtype, self.relu, self.tile = (m, k, n), torch.float16 if half else torch.float32, relu, tile
        _, self.a, self.w, self.bias = _operands(dev, m, k, n)
        self.q = torch.tensor([31.7, 211.3], device=dev)
        self.ws = ops.default_workspace(dev)

    def empty(self, skip=0):
        m, _, n = self.shape
        return torch.full((m * n + skip,), float("nan"), dtype=self.dtype, device=self.a.device)[skip:].view(m, n)

    def call(self, rows, out, tile=None):
        from marian_dev_b200.binding import check, lib
        _, k, n = self.shape
        check(lib().mi8_multiply_i8_ex(rows.data_ptr(), self.w.data_ptr(), rows.shape[0], n, k, self.q.data_ptr(), self.q[1:].data_ptr(), 1.0, self.bias.data_ptr(),
                                       int(self.relu), out.data_ptr(), 1 if self.dtype == torch.float16 else 0, None, self.ws.ptr, self.ws.nbytes,
                                       torch.cuda.current_stream().cuda_stream, self.tile if tile is None else tile, 0))

    def whole(self, out):
        self.call(self.a, out)
        return out

    def by_blocks(self, rows=512):
        out = self.empty()
        for r in range(0, self.shape[0], rows):
            self.call(self.a[r:r + rows], out[r:r + rows], 0)
        return out


# asked for: one K block and fewer blocks than the ring has, an odd number, a ragged last one; the plan's own choice: eight blocks, full and ragged.  One and
# several activation tiles of a share, M of one row more than a tile
@pytest.mark.parametrize("m,k,n,half,tile", [(1400, 80, 27008, False, PAIR), (2305, 272, 16400, False, PAIR), (6100, 640, 6200, False, PAIR), (1200, 896, 63008, True, PAIR),
                                             (2049, 1024, 36992, True, 0), (1400, 912, 27008, False, 0), (2305, 1008, 16400, False, 0)])
@pytest.mark.parametrize("relu", [False, True])
def test_equals_blocks_of_rows(cuda_device, m, k, n, half, tile, relu):
    p = _Products(cuda_device, m, k, n, half, relu, tile)
    assert _route(lambda: p.whole(p.empty())) == "held"
    got, want = p.whole(p.empty()), p.by_blocks()
    assert torch.equal(got, want) and _status() == 0


@pytest.mark.parametrize("k,tile", [(384, PAIR), (1024, 0)])
@pytest.mark.parametrize("limit", [0, 255, 256, 1300, 2300])
def test_rows_below_a_limit_are_kept(cuda_device, k, tile, limit):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    m, n = 2300, 17000
    _, a, w, bias = _operands(cuda_device, m, k, n)
    q = torch.tensor([31.7, 211.3], device=cuda_device)
    words = torch.tensor([7, 7, 8], dtype=torch.int32, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream

    def product(rows, out, other, below, tile=0):
        check(lib().mi8_multiply_i8_rows_from(rows.data_ptr(), w.data_ptr(), rows.shape[0], n, k, q.data_ptr(), q[1:].data_ptr(), 1.0, bias.data_ptr(), 0,
                                              out.data_ptr(), 0, ws.ptr, ws.nbytes, stream, words.data_ptr(), other.data_ptr(), below, tile))

    want = torch.empty((m, n), device=cuda_device)
    for r in range(0, m, 500):
        product(a[r:r + 500], want[r:r + 500], words[2:], 0)
    for other, kept in ((words[1:], limit // 256 * 256), (words[2:], 0)):
        got = torch.full((m, n), 12345.0, device=cuda_device)
        assert _route(lambda: product(a, got, other, limit, tile)) == "held"
        product(a, got.fill_(12345.0), other, limit, tile)
        assert bool((got[:kept] == 12345.0).all()) and torch.equal(got[kept:], want[kept:])
    assert _status() == 0


@pytest.mark.parametrize("k,tile", [(768, PAIR), (1024, 0)])
def test_packed8(cuda_device, k, tile):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    m, n = 1400, 28000
    g, a, w, bias = _operands(cuda_device, m, k, n, unsigned=True)
    scale_a, scale_b = torch.rand(m, generator=g, device=cuda_device), torch.rand(n, generator=g, device=cuda_device)
    zp_a, sum_a = (torch.randint(0, 256, (m,), generator=g, device=cuda_device, dtype=torch.int32) for _ in range(2))
    zp_b, off_b = (torch.randint(-63, 64, (n,), generator=g, device=cuda_device, dtype=torch.int32) for _ in range(2))
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream

    def product(first, last, out, tile=0):
        check(lib().mi8p_multiply(a[first:].data_ptr(), scale_a[first:].data_ptr(), zp_a[first:].data_ptr(), sum_a[first:].data_ptr(), w.data_ptr(),
                                  scale_b.data_ptr(), zp_b.data_ptr(), off_b.data_ptr(), last - first, n, k, bias.data_ptr(), 1, out[first:].data_ptr(), None,
                                  ws.ptr, ws.nbytes, stream, tile, 0))

    got, want = torch.empty((m, n), device=cuda_device), torch.empty((m, n), device=cuda_device)
    assert _route(lambda: product(0, m, got, tile)) == "held"
    product(0, m, got.fill_(0), tile)
    for r in range(0, m, 448):
        product(r, min(m, r + 448), want)
    assert torch.equal(got, want) and _status() == 0


@pytest.mark.parametrize("half", [False, True])
def test_several_matrices(cuda_device, half):
    """Three matrices of an odd number of 128-row tiles: a pair's CTAs hold rows of two matrices, the last pair's second CTA holds none."""
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    m, k, n = 4096, 1024, 51 * 128
    _, a, w, bias = _operands(cuda_device, m, k, 3 * n)
    q = torch.tensor([31.7, 211.3, 95.1, 400.7], device=cuda_device)
    dtype = torch.float16 if half else torch.float32
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    got = [torch.full((m, n), float("nan"), dtype=dtype, device=cuda_device) for _ in range(3)]
    pointers = ctypes.c_void_p * 3
    qb, bp, cp = (pointers(*[x.data_ptr() for x in xs]) for xs in ([q[1:], q[2:], q[3:]], [bias, bias[n:], bias[2 * n:]], got))

    def products():
        check(lib().mi8_multiply_i8_multi(a.data_ptr(), w.data_ptr(), m, n, k, 3, q.data_ptr(), qb, 1.0, bp, 0, cp, int(half), ws.ptr, ws.nbytes, stream))

    assert _route(products) == "held"
    for x in got:
        x.fill_(float("nan"))
    products()
    for i in range(3):
        want = torch.empty((m, n), dtype=dtype, device=cuda_device)
        for r in range(0, m, 512):
            check(lib().mi8_multiply_i8(a[r:].data_ptr(), w[i * n:].data_ptr(), 512, n, k, q.data_ptr(), q[1 + i:].data_ptr(), 1.0, bias[i * n:].data_ptr(), 0,
                                        want[r:].data_ptr(), int(half), None, ws.ptr, ws.nbytes, stream))
        assert torch.equal(got[i], want)
    assert _status() == 0


# held only where every row of the results is whole 32-byte sectors, the parts of other rows' sectors at the tiles' edges being written too far apart (`shift`:
# bytes between a sector's start and the results'), and where no more than a ninth of the activation tiles is padding
@pytest.mark.parametrize("m,n,half,shift,route", [(1536, 25000, False, 0, "held"), (1536, 25004, False, 0, "pair"), (1536, 25001, False, 0, "pair"),
                                                  (1536, 25000, False, 16, "pair"), (2560, 31984, True, 0, "held"), (2560, 31992, True, 0, "pair"),
                                                  (2560, 31985, True, 0, "pair"), (2560, 31984, True, 2, "pair"),
                                                  (1366, 29104, False, 0, "held"), (1365, 29104, False, 0, "pair"), (1281, 30720, False, 0, "pair")])
def test_which_results(cuda_device, m, n, half, shift, route):
    p = _Products(cuda_device, m, 1024, n, half)
    got = p.empty(shift // (2 if half else 4))
    assert got.data_ptr() % 32 == shift
    assert _route(lambda: p.whole(got)) == route
    assert torch.equal(p.whole(got.fill_(0)), p.by_blocks()) and _status() == 0


# a block of a pair's first tile and one of its second that never arrive, with one ring stage and with three, and one write-back warp that gives up
@pytest.mark.parametrize("k,tile", [(80, PAIR), (640, PAIR), (1024, 0)])
@pytest.mark.parametrize("item", [0, "second tile", ONE_WARP])
def test_waits_run_out(cuda_device, k, tile, item):
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import check, lib
    p = _Products(cuda_device, 1536, k, 25000, tile=tile)
    got, want = p.empty(), p.by_blocks()
    assert _route(lambda: p.whole(got)) == "held" and _status() == 0
    blocks = (k + 127) // 128
    try:
        lib().mi8_test_wait_fault(2 * blocks - 1 if item == "second tile" else item, 1 << 14)
        p.whole(got)
        torch.cuda.synchronize()                      # the kernel returned by itself
    finally:
        lib().mi8_test_wait_fault(-1, 0)
    assert _status() in (101, 102, 103, 104)
    check(lib().mi8_workspace_init(p.ws.ptr, p.ws.nbytes, torch.cuda.current_stream().cuda_stream))
    ops.clear_status()
    for _ in range(2):
        assert torch.equal(p.whole(got.fill_(0)), want) and _status() == 0
