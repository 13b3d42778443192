"""Affines of few floats in one launch, every CTA finding the activation's maximum itself, against the quantisation and the product apart (bit for bit, the scratch
included): rows, inner dimensions, float counts and widths around the rule's limits, the maximum anywhere, zeros, what is not a number, launches that overlap."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _affine(x, w, b, scale, relu, half, ws, scratch, out):
    from marian_dev_b200.binding import lib
    m, k = x.shape
    return lib().mi8_affine_f32(x.data_ptr(), m, k, w.data.data_ptr(), w.quant_mult.data_ptr(), out.shape[1], b.data_ptr() if b is not None else None, scale, relu,
                                out.data_ptr(), 1 if half else 0, scratch.data_ptr(), ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream)


def _launches(call):
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    check(lib().mi8_kernel_times_begin())
    try:
        call()
    finally:
        records, n = (Mi8KernelTime * 8)(), ctypes.c_int(0)
        check(lib().mi8_kernel_times_end(records, 8, ctypes.byref(n)))
    return sum(r.launches for r in records[:n.value])


@pytest.mark.parametrize("m,k,n,one", [(1, 16, 129, True), (1, 1024, 300, True), (4, 256, 1536, True), (3, 272, 300, True), (16, 256, 512, True), (15, 272, 200, True),
                                       (16, 272, 200, False), (4, 1024, 256, True), (4, 1040, 256, False), (17, 16, 256, False), (16, 16, 256, True),
                                       (2, 512, 128, False), (2, 512, 18944, True), (2, 512, 18945, False)])
@pytest.mark.parametrize("where", ["first", "last", "zero"])
def test_bits(cuda_device, m, k, n, one, where):
    from marian_dev_b200 import ops
    g = torch.Generator(device=cuda_device).manual_seed(m * k + n)
    x = torch.randn(m, k, generator=g, device=cuda_device)
    if where == "zero":
        x.zero_()
    else:
        x.view(-1)[0 if where == "first" else -1] = -9.5
    w = ops.prepareB(torch.randn(k, n, generator=g, device=cuda_device) * 0.05)
    ws = ops.default_workspace(cuda_device)
    for half, b, relu in ((False, torch.randn(n, generator=g, device=cuda_device), 1), (True, None, 0)):
        dtype = torch.float16 if half else torch.float32
        room = torch.full((m + 1, n), 7.0, dtype=dtype, device=cuda_device)
        scratch = torch.full((m * k + 64,), 99, dtype=torch.int8, device=cuda_device)
        assert _launches(lambda: _affine(x, w, b, 1.5, relu, half, ws, scratch, room[:m])) == (1 if one else 2)
        aq = ops.prepareA(x)
        want = ops.multiply(aq, w, b, scale=1.5, relu=bool(relu), out_dtype=dtype)
        assert torch.equal(room[:m], want) and bool((room[m] == 7.0).all())
        assert torch.equal(scratch[:m * k].view(m, k), aq.data.view(m, k)) and bool((scratch[m * k + 4:] == 99).all())
        assert torch.equal(scratch[m * k:m * k + 4].view(torch.float32), aq.quant_mult)
        for i in range(4):
            _affine(x, w, b, 1.5, relu, half, ws, scratch, room[:m])
        assert torch.equal(room[:m], want) and ops.poll_status() == 0


def test_refused_and_reported(cuda_device):
    from marian_dev_b200 import ops
    x = torch.randn(4, 256, device=cuda_device)
    w = ops.prepareB(torch.randn(256, 512, device=cuda_device))
    ws, scratch, out = ops.default_workspace(cuda_device), torch.empty(4 * 256 + 64, dtype=torch.int8, device=cuda_device), torch.empty(4, 512, device=cuda_device)
    from marian_dev_b200.binding import lib
    args = [x.data_ptr(), 4, 256, w.data.data_ptr(), w.quant_mult.data_ptr(), 512, None, 1.0, 0, out.data_ptr(), 0, scratch.data_ptr(), ws.ptr, ws.nbytes, None]
    for place, value, status in ((0, None, 1), (3, None, 1), (4, None, 1), (9, None, 1), (10, 7, 1), (11, None, 1), (0, x.data_ptr() + 4, 2), (3, w.data.data_ptr() + 4, 2),
                                 (11, scratch.data_ptr() + 4, 2), (12, None, 4), (13, 64, 4)):
        assert lib().mi8_affine_f32(*[value if i == place else a for i, a in enumerate(args)]) == status, (place, status)
    x[2, 5] = float("nan")
    assert _affine(x, w, None, 1.0, 0, False, ws, scratch, out) == 0
    assert ops.poll_status() == 110
    ops.clear_status()
    torch.cuda.synchronize()
    assert ops.poll_status() == 0


def test_wait_that_runs_out(cuda_device):
    """A K block that never comes, a write-back warp that gives up in front of the maximum's barrier: reported, and the next call is right."""
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import lib
    x = torch.randn(4, 256, device=cuda_device)
    w = ops.prepareB(torch.randn(256, 512, device=cuda_device))
    want = ops.affine(x, w, None)
    assert ops.poll_status() == 0
    for item in (0, 1, -2):     # (-2: one write-back warp)
        try:
            lib().mi8_test_wait_fault(item, 1 << 14)
            ops.affine(x, w, None)
            torch.cuda.synchronize()
        finally:
            lib().mi8_test_wait_fault(-1, 0)
        assert ops.poll_status() in (101, 102, 103, 104)
        ops.clear_status()
        assert torch.equal(ops.affine(x, w, None), want) and ops.poll_status() == 0
