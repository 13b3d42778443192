"""Abs-max and quantisation in two launches that overlap, and the conversion of a weight behind the same search: lengths around the routes' limits (the wide
cluster, one to eight vectors per thread, more blocks than are resident, 256, 512 and 1024 threads), with and without a ragged end, the maximum anywhere;
against torch's arithmetic in float32 (one product, rounded half to even, saturated: exact)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(x):
    m = x.abs().max()
    mult = torch.tensor([127.0], device=x.device) / m if m > 0 else torch.ones(1, device=x.device)
    return mult, torch.clamp(torch.round(x * mult), -127, 127).to(torch.int8)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4099, 32752, 32768, 32784, 65552, 262128, 262144, 262160, 262147, 454656, 454672, 909312, 1310720, 1310736, 1363970,
                               1818640, 2727936, 3637264, 3932160, 3932176, 4194307])
@pytest.mark.parametrize("where", ["first", "middle", "last", "zero"])
def test_prepare(cuda_device, n, where):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    x = torch.rand(n, generator=torch.Generator(device=cuda_device).manual_seed(n), device=cuda_device) - 0.5
    if where == "zero":
        x.zero_()
    else:
        x[{"first": 0, "middle": n // 2, "last": -1}[where]] = -0.75
    q = torch.full((n + 64,), 99, dtype=torch.int8, device=cuda_device)
    mult = torch.zeros(1, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    want_mult, want = _want(x)
    for _ in range(2):   # (the second beside the first's end)
        check(lib().mi8_prepare_a_f32(x.data_ptr(), 1, n, q.data_ptr(), mult.data_ptr(), ws.ptr, ws.nbytes, stream))
    assert torch.equal(mult, want_mult)
    assert torch.equal(q[:n], want) and bool((q[n:] == 99).all())
    assert ops.poll_status() == 0


def test_input_of_the_kernel_in_front(cuda_device):
    """Launches whose input the kernel before them writes: nothing of it is read early, back to back and replayed from a graph."""
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    n = 1 << 20
    src = [torch.randn(n, device=cuda_device) * (i + 1) for i in range(4)]
    x = torch.empty(n, device=cuda_device)
    q = torch.empty(4, n, dtype=torch.int8, device=cuda_device)
    mult = torch.empty(4, 1, device=cuda_device)

    def run(ws):
        for i in range(4):
            x.copy_(src[i])
            check(lib().mi8_prepare_a_f32(x.data_ptr(), 1, n, q[i].data_ptr(), mult[i].data_ptr(), ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream))

    def right():
        return all(torch.equal(q[i], _want(src[i])[1]) and torch.equal(mult[i], _want(src[i])[0]) for i in range(4))

    run(ops.default_workspace(cuda_device))
    assert right()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        ws = ops.default_workspace(cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        run(ws)
    q.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert right() and ops.poll_status() == 0


@pytest.mark.parametrize("k,n", [(1, 4), (3, 1), (128, 32), (1000, 1001), (1282, 1024), (1024, 4100), (3841, 1024), (129, 32000)])
@pytest.mark.parametrize("last", [False, True])
def test_convert(cuda_device, k, n, last):
    from marian_dev_b200.binding import check, lib
    from marian_dev_b200 import ops
    w = torch.rand(k, n, generator=torch.Generator(device=cuda_device).manual_seed(k + n), device=cuda_device) - 0.5
    w.view(-1)[-1 if last else 0] = 0.75
    bt = torch.full((k * n + 64,), 99, dtype=torch.int8, device=cuda_device)
    mult = torch.zeros(1, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    for _ in range(2):
        check(lib().mi8_prepare_b_f32(w.data_ptr(), k, n, 0, bt.data_ptr(), mult.data_ptr(), ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream))
    want_mult, want = _want(w)
    assert torch.equal(mult, want_mult)
    assert torch.equal(bt[:k * n].view(n, k), want.T) and bool((bt[k * n:] == 99).all())
    assert ops.poll_status() == 0
