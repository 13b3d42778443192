"""The native per-call host path (host/ops_native.cpp): what it declines goes through the general Python route with that route's results and
errors, and no argument ends the process."""
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_DECLINED = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from marian_dev_b200 import ops
n = ops.native()
with FakeTensorMode():                                     # CUDA tensors without memory (and here without a GPU)
    a, w, f, i = (torch.empty(s, dtype=t, device="cuda") for s, t in (((4, 256), torch.float32), (32 * 256 + 256, torch.uint8), (32, torch.float32),
                                                                     (32, torch.int32)))
    bt = torch.empty(32, 256, dtype=torch.int8, device="cuda")
for a, w, f, i, bt in ((a, w, f, i, bt), [torch.empty(x.shape, dtype=x.dtype) for x in (a, w, f, i, bt)], ["a", None, 3, 4.0, []]):
    assert n.affine(a, w, 256, 32, f, 1.0, False, False) is None
    assert n.prepare_b(a, 4, 256, False) is None
    assert n.p8_prepare_b(a) is None
    assert n.p8_gemm(a, bt, f, i, i, f) is None
print("declined")
"""


def test_tensors_without_device_memory_are_declined():
    """In a process of its own: an exception that leaves the extension ends the process."""
    r = subprocess.run([sys.executable, "-c", _DECLINED], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "declined", r.stderr[-2000:]


def test_packed8_general_route_rejects_bad_operands():
    """What the native route declines is checked again before any address is taken: fake CUDA tensors have none."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from marian_dev_b200 import ops, packed8
    with FakeTensorMode():
        new = lambda *s, dtype=torch.float32, device="cuda": torch.empty(s, dtype=dtype, device=device)
        w = packed8.Packed8Weight.__new__(packed8.Packed8Weight)
        w.K, w.N, w.item = 256, 32, new(256 * 32 + 384, dtype=torch.int8)
        w.bt, w.scale_b, w.zp_b, w.off_b = new(32, 256, dtype=torch.int8), new(32), new(32, dtype=torch.int32), new(32, dtype=torch.int32)
        bad = [(new(4, 128), None), (new(4, 512), None), (new(), None), (new(4, 256, dtype=torch.float16), None), (new(4, 256, dtype=torch.float64), None),
               (new(4, 256, device="cpu"), None), (new(4, 256), new(31)), (new(4, 256), new(33)), (new(4, 256), new(32, dtype=torch.float16)),
               (new(4, 256), new(32, dtype=torch.int32)), (new(4, 256), new(32, device="cpu"))]
        outs = [new(4, 31), new(4, 32, dtype=torch.float16), new(32, 4).t(), new(4, 32, device="cpu")]
    for a, bias in bad:
        with pytest.raises(ops.Mi8Error):
            packed8.gemmInt8Packed(a, w, bias)
    for out in outs:
        with pytest.raises(ops.Mi8Error):
            packed8.gemmInt8Packed(bad[6][0], w, None, out=out)
    for a in (bad[3][0], bad[4][0]):
        with pytest.raises(ops.Mi8Error):
            packed8.quantize_rows(a)
    aq, f, i = w.bt.view(torch.uint8)[:4], w.scale_b, w.zp_b
    for bias in (b for _, b in bad if b is not None):
        with pytest.raises(ops.Mi8Error):
            packed8.multiply(aq, f, i, i, w, bias)


def _operands(device, m=6, k=64, n=40):
    from marian_dev_b200 import ops
    g = torch.Generator(device=device).manual_seed(m * k + n)
    x = torch.randn(m, k, generator=g, device=device)
    return x, ops.prepareB(torch.randn(k, n, generator=g, device=device) * 0.05), torch.randn(n, generator=g, device=device)


@pytest.mark.gpu
def test_vmapped_operands_raise(cuda_device):
    from marian_dev_b200 import ops, packed8
    x, w, b = _operands(cuda_device)
    w8 = packed8.prepareB(torch.randn(256, 32, device=cuda_device))
    x8, b8 = torch.randn(6, 256, device=cuda_device), torch.randn(32, device=cuda_device)
    for f, arg in ((lambda t: ops.affine(x, w, t), b), (lambda t: ops.affine(t, w, b), x), (lambda t: ops.prepareB(t).storage, x),
                   (lambda t: packed8.gemmInt8Packed(x8, w8, t), b8), (lambda t: packed8.gemmInt8Packed(t, w8, b8), x8),
                   (lambda t: packed8.prepareB(t).item, torch.randn(256, 32, device=cuda_device))):
        with pytest.raises(RuntimeError):
            torch.func.vmap(f)(torch.stack([arg, arg]))
    torch.cuda.synchronize()
    assert ops.affine(x, w, b).shape == (6, 40) and ops.poll_status() == 0


@pytest.mark.gpu
def test_declined_operands_take_the_general_route(cuda_device):
    """Layouts that the native route leaves alone give the bits of the contiguous operands; refused ones raise as they do with an explicit
    workspace, which always takes the general route."""
    from marian_dev_b200 import ops
    x, w, b = _operands(cuda_device)
    want = ops.affine(x, w, b)
    assert torch.equal(ops.affine(x, w, b, ws=ops.default_workspace(cuda_device)), want)
    assert torch.equal(ops.affine(x.t().contiguous().t(), w, b), want)
    assert torch.equal(ops.affine(x, w, torch.stack([b, b], 1)[:, 0]), want)
    assert torch.equal(ops.affine(x.t().contiguous(), w, b, transA=True), want)
    assert ops.affine(x.reshape(2, 3, 64), w, b).shape == (2, 3, 40) and ops.affine(x[0], w, b).shape == (40,)
    for args in ((x.half(), w, b), (x[:, :32].contiguous(), w, b), (x, w, b[:39]), (x, w, b.half()), (x.cpu(), w, b), (x, w, b.cpu()), (x, w.data, b)):
        for kw in ({}, {"ws": ops.default_workspace(cuda_device)}):
            with pytest.raises(ops.Mi8Error):
                ops.affine(*args, **kw)
    assert ops.poll_status() == 0


@pytest.mark.gpu
def test_packed8_general_route_gives_the_same_bits(cuda_device):
    from marian_dev_b200 import ops, packed8
    g = torch.Generator(device=cuda_device).manual_seed(5)
    x, b = torch.randn(6, 256, generator=g, device=cuda_device), torch.randn(32, generator=g, device=cuda_device)
    w = packed8.prepareB(torch.randn(256, 32, generator=g, device=cuda_device))
    want = packed8.gemmInt8Packed(x, w, b)
    out = torch.empty(6, 32, device=cuda_device)
    assert torch.equal(packed8.gemmInt8Packed(x, w, b, out=out), want) and torch.equal(out, want)
    assert torch.equal(packed8.gemmInt8Packed(x.t().contiguous().t(), w, torch.stack([b, b], 1)[:, 0]), want)
    assert torch.equal(packed8.gemmInt8Packed(x, w, b, ws=ops.default_workspace(cuda_device)), want)
    assert packed8.gemmInt8Packed(x.reshape(2, 3, 256), w).shape == (2, 3, 32) and packed8.gemmInt8Packed(x[0], w).shape == (32,)
    assert packed8.gemmInt8Packed(x[:0], w, b).shape == (0, 32)
    assert torch.equal(packed8.multiply(*packed8.quantize_rows(x), w, torch.stack([b, b], 1)[:, 0]), want)
    assert ops.poll_status() == 0


@pytest.mark.gpu
def test_failed_allocation_raises_torchs_error(cuda_device):
    from marian_dev_b200 import ops
    n = 1 << 24
    w = ops.prepareB(torch.zeros(16, n, device=cuda_device))
    with pytest.raises(torch.OutOfMemoryError):          # 4 TB of output
        ops.affine(torch.zeros(1 << 16, 16, device=cuda_device), w, None)


def test_documented_build_makes_the_extension():
    """`make -C marian-dev_b200/csrc` and build_library() are the documented builds of all that the Python operators need."""
    out = subprocess.run(["make", "-n", "-B", "-C", os.path.join(ROOT, "marian-dev_b200", "csrc")], capture_output=True, text=True, check=True).stdout
    assert "-o ../libmarian_i8.so" in out and "-o ../_ops_native.so" in out and "-D_GLIBCXX_USE_CXX11_ABI=" in out


def test_missing_or_foreign_extension_names_the_build(monkeypatch):
    from marian_dev_b200 import ops
    ops.native()
    monkeypatch.setattr(ops, "_native_ext", None)
    with monkeypatch.context() as m, pytest.raises(ImportError, match="built for torch .*make -C .*host ops"):
        m.setattr(torch, "__version__", "1.0.0")
        ops.native()
    pkg = sys.modules[ops.__name__.rpartition(".")[0]]
    with monkeypatch.context() as m, pytest.raises(ImportError, match="make -C .*host ops"):
        m.setitem(sys.modules, pkg.__name__ + "._ops_native", None)
        m.delattr(pkg, "_ops_native")
        ops.native()
    assert ops.native().affine


@pytest.mark.parametrize("storage", [torch.zeros(300, dtype=torch.uint8)[1:], torch.zeros(600, dtype=torch.uint8)[::2], torch.zeros(300), torch.zeros(20, 16, dtype=torch.uint8)],
                         ids=["off a word boundary", "strided", "float", "matrix"])
def test_given_storage_that_cannot_be_viewed_is_refused(storage):
    from marian_dev_b200 import ops
    with pytest.raises(RuntimeError):
        ops.IntgemmTensor(16, 16, "cpu", storage=storage)
    ok = ops.IntgemmTensor(16, 16, "cpu", storage=torch.arange(260, dtype=torch.uint8))
    assert ok.data.shape == (16, 16) and ok.data.dtype == torch.int8 and int(ok.data[1, 2]) == 18
    assert ok.quant_mult.shape == (1,) and torch.equal(ok.quant_mult.view(torch.uint8), ok.storage[256:260])


@pytest.mark.gpu
def test_weight_whose_shape_is_not_its_width_is_refused(cuda_device):
    from marian_dev_b200 import ops
    x, w, b = _operands(cuda_device)
    other = ops.IntgemmTensor(w.rows, w.cols, cuda_device, storage=w.storage)      # shape [N,K]: not a weight's
    for kw in ({}, {"ws": ops.default_workspace(cuda_device)}):
        with pytest.raises(RuntimeError):
            ops.affine(x, other, b, **kw)
