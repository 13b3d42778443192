"""Affines of few floats under stream capture: two launches as before there was one, since a graph has no host launches to save; the replay gives the same bits as
the call, with other values in the same buffers too.  Long rows against weights that fill the chip are two launches in any case."""
import pytest
import torch

from tests.test_gpu_affine_one_launch import _affine, _launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,half", [(4, 256, 1536, False), (1, 16, 129, False), (16, 256, 512, True), (4, 1024, 1024, False)])
def test_replay(cuda_device, m, k, n, half):
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import lib
    g = torch.Generator(device=cuda_device).manual_seed(n)
    x = torch.randn(m, k, generator=g, device=cuda_device)
    w = ops.prepareB(torch.randn(k, n, generator=g, device=cuda_device))
    b = torch.randn(n, generator=g, device=cuda_device)
    dtype = torch.float16 if half else torch.float32
    out, want = (torch.empty(m, n, dtype=dtype, device=cuda_device) for _ in range(2))
    scratch = torch.empty(m * k + 64, dtype=torch.int8, device=cuda_device)
    ws = ops.Workspace(cuda_device)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        before = lib().mi8_launch_count()
        assert _affine(x, w, b, 1.0, 1, half, ws, scratch, out) == 0
        captured = lib().mi8_launch_count() - before
    assert captured == 2
    before = lib().mi8_launch_count()
    assert _affine(x, w, b, 1.0, 1, half, ws, scratch, want) == 0 and lib().mi8_launch_count() - before == 1
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and ops.poll_status() == 0
        x.normal_(generator=g)
        assert _affine(x, w, b, 1.0, 1, half, ws, scratch, want) == 0


@pytest.mark.parametrize("m,k,n,one", [(4, 1024, 8192, True), (4, 1024, 8193, False), (4, 528, 8193, False), (4, 512, 8193, True)])
def test_wide_weights(cuda_device, m, k, n, one):
    from marian_dev_b200 import ops
    x = torch.randn(m, k, device=cuda_device)
    w = ops.prepareB(torch.randn(k, n, device=cuda_device))
    ws, scratch, out = ops.default_workspace(cuda_device), torch.empty(m * k + 64, dtype=torch.int8, device=cuda_device), torch.empty(m, n, device=cuda_device)
    assert _launches(lambda: _affine(x, w, None, 1.0, 0, False, ws, scratch, out)) == (1 if one else 2)
    assert torch.equal(out, ops.multiply(ops.prepareA(x), w, None)) and ops.poll_status() == 0
