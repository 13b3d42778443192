"""Encoder self-attention, 32 query positions a block: lengths around a block's queries, a warp's key positions, a head's interleaved sums and what shared memory
holds (the lengths beyond take the one-row kernel), with and without a mask; bit for bit the oracle's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 65, 97, 205, 300, 316, 317, 330])
@pytest.mark.parametrize("dh,heads", [(32, 3), (64, 2)])
@pytest.mark.parametrize("with_mask", [True, False])
def test_bits(cuda_device, oracle, length, dh, heads, with_mask):
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import check, lib
    batch = 3 if length < 200 else 1
    rows, dim = batch * length, heads * dh
    rng = np.random.default_rng(length + dh)
    q, k, v = (rng.standard_normal((rows, dim)).astype(np.float32) for _ in range(3))
    mask = None
    if with_mask:
        lens = rng.integers(1, length + 1, size=batch)
        mask = np.where(np.arange(length)[None, :] < lens[:, None], 0.0, -99999999.0).astype(np.float32)
    want = oracle.attention1(q, k, v, mask, rows, heads, dh, length, batch, 2)
    d = [torch.from_numpy(a).to(cuda_device) for a in (q, k, v)]
    m = torch.from_numpy(mask).to(cuda_device) if with_mask else None
    out = torch.full((rows + 1, dim), 7.0, device=cuda_device)
    slot = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    check(lib().mi8g_attention1(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), m.data_ptr() if with_mask else None, rows, heads, dh, length, batch, 2,
                                out.data_ptr(), slot.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(out[:rows].cpu().numpy(), want) and bool((out[rows] == 7.0).all())
    assert slot.view(torch.float32).item() == np.abs(want).max() and ops.poll_status() == 0
