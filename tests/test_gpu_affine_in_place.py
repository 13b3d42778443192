"""Affines of few floats whose results or scratch lie over the activation (whole, its end, its start): two launches, which have read the activation before
anything is stored, against the same call with buffers of its own (bit for bit); buffers that touch without sharing a byte keep the one launch."""
import pytest
import torch

from tests.test_gpu_affine_one_launch import _affine, _launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,half", [(8, 512, 512, False), (4, 1024, 1024, False), (1, 256, 256, False), (16, 256, 256, True), (3, 272, 200, False)])
@pytest.mark.parametrize("where", ["result", "result from the last row on", "result up to the first row", "scratch", "results behind", "scratch behind"])
def test_over_the_activation(cuda_device, m, k, n, half, where):
    from marian_dev_b200 import ops
    g = torch.Generator(device=cuda_device).manual_seed(m + k)
    x = torch.randn(m, k, generator=g, device=cuda_device)
    w = ops.prepareB(torch.randn(k, n, generator=g, device=cuda_device) * 0.05)
    b = torch.randn(n, generator=g, device=cuda_device)
    ws = ops.default_workspace(cuda_device)
    dtype, size = (torch.float16, 2) if half else (torch.float32, 4)
    want = torch.empty(m, n, dtype=dtype, device=cuda_device)
    scratch = torch.empty(m * k + 64, dtype=torch.int8, device=cuda_device)
    assert _launches(lambda: _affine(x, w, b, 1.0, 1, half, ws, scratch, want)) == 1
    quantised = scratch[:m * k + 4].clone()
    in_bytes, out_bytes = 4 * m * k, size * m * n
    lead = (out_bytes + 255) // 256 * 256
    room = torch.zeros(lead + in_bytes + lead + 64, dtype=torch.int8, device=cuda_device)
    a = room[lead:lead + in_bytes].view(torch.float32).view(m, k)
    place = {"result": lead, "result from the last row on": lead + in_bytes - 4 * k, "result up to the first row": lead + 4 * k - out_bytes,
             "results behind": lead + in_bytes}.get(where)
    out = room[place:place + out_bytes].view(dtype).view(m, n) if place is not None else torch.empty_like(want)
    aq = scratch if place is not None else room[lead:] if where == "scratch" else room[lead + in_bytes:]
    call = lambda: _affine(a, w, b, 1.0, 1, half, ws, aq, out)
    for i in range(4):
        a.copy_(x)
        if i == 0:
            assert _launches(call) == (1 if "behind" in where else 2)
        else:
            assert call() == 0
        assert torch.equal(out, want) and torch.equal(aq[:m * k + 4], quantised) and ops.poll_status() == 0
