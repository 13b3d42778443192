"""One write-back warp whose bounded wait runs out while the others' do not: all eight leave the tile together (they meet at barriers of the
block, which have no bound), the launch returns, and the status word says so.  mi8_test_wait_fault(MI8_TEST_ONE_WARP, ...) makes one warp of
every CTA give up; nothing faults or spins for ever."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ONE_WARP = -2


def _expect_status_then_clear(L, ops, ws):
    from marian_dev_b200.binding import check
    status = ops.poll_status()
    v = ctypes.c_int(0)
    assert L.mi8_poll_status(ctypes.byref(v)) == 6      # MI8_ERR_DEVICE until the word is cleared
    check(L.mi8_workspace_init(ws.ptr, ws.nbytes, torch.cuda.current_stream().cuda_stream))
    ops.clear_status()
    return status


# a tile per CTA without and with several splits of K, several tiles per CTA, the CTA-pair kernel, two CTAs that share a tile's K
@pytest.mark.parametrize("m,k,n,tile,kind", [(48, 512, 384, 0, "plain"), (40, 4096, 256, 0, "splits"), (300, 512, 20000, 64, "plain"),
                                             (300, 1024, 512, 512, "pair"), (700, 512, 32000, 512, "pair"), (200, 2048, 1664, 0, "duo")])
def test_multiply(cuda_device, oracle, m, k, n, tile, kind):
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import lib, multiply_plan
    L = lib()
    plan = multiply_plan(m, n, k, tile, 0)
    duo = plan["splits"] == 2 and plan["tile_m"] == 64 and plan["grid"] == 2 * plan["n_tiles"] * plan["m_tiles"] and k > 1920 and m > 64
    assert kind == ("pair" if plan["tile_m"] == 512 else "duo" if duo else "splits" if plan["splits"] > 1 else "plain")
    rng = np.random.default_rng(m + n)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((k, n)) * 0.02).astype(np.float32)
    bt, qb = oracle.prepare_b(w)
    want = oracle.affine(a, bt, qb, None, 1.0, False)
    aq = ops.prepareA(torch.from_numpy(a).to(cuda_device))
    b = ops.prepareB(torch.from_numpy(w).to(cuda_device))
    ws = ops.default_workspace(cuda_device)
    torch.cuda.synchronize()
    assert ops.poll_status() == 0
    try:
        L.mi8_test_wait_fault(ONE_WARP, 1 << 14)
        ops.multiply(aq, b, None, tile_m=tile)
        torch.cuda.synchronize()                      # the kernel returned by itself
    finally:
        L.mi8_test_wait_fault(-1, 0)
    assert _expect_status_then_clear(L, ops, ws) in (101, 102, 103, 104)
    for _ in range(2):
        out = ops.multiply(aq, b, None, tile_m=tile)
        torch.cuda.synchronize()
        assert ops.poll_status() == 0 and np.array_equal(out.cpu().numpy(), want)


# the first step of up to 32 rows: its output layer reduces the blocks of the log-softmax at such barriers (tiles of 16 and of 32 rows, both schemes)
# the first step of a few rows of an SSRU decoder: the cluster launch of all layers, one warp giving up or a unit of every warp's weights never arriving (with
# and without units behind it that are waited for before the CTA leaves)
@pytest.mark.parametrize("scheme,rnn,rows,items", [("intgemm8", False, 3, (ONE_WARP,)), ("intgemm8", False, 20, (ONE_WARP,)),
                                                   ("packed8avx512", False, 5, (ONE_WARP,)), ("intgemm8", True, 1, (ONE_WARP, 0, 1)),
                                                   ("intgemm8", True, 30, (ONE_WARP, 2))])
def test_decoder_step(cuda_device, scheme, rnn, rows, items):
    from marian_dev_b200 import decoder, model, ops
    from marian_dev_b200.binding import lib
    L = lib()
    cfg = model.TransformerConfig(dim_emb=256, dim_ffn=512, heads=8, enc_depth=1, dec_depth=2, vocab=30016,
                                  decoder_autoreg="rnn" if rnn else "self-attention")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, rows), cuda_device, scheme=scheme)
    stepper = decoder.NativeStepper(net, max_batch=rows, beam=2, max_src=8, max_steps=8)
    g = torch.Generator(device="cuda").manual_seed(rows)
    context = torch.randn(rows, 7, cfg.dim_emb, generator=g, device=cuda_device)
    log_mask = torch.zeros(rows, 7, device=cuda_device)

    def first_step():
        stepper.start(context, log_mask)
        return stepper.step(None, None, None, None, 1, rows, 2)
    want = first_step()
    assert ops.poll_status() == 0
    if rnn:                                           # (all layers in one launch)
        first_step()
        L.mi8_launch_count_reset()
        first_step()
        assert L.mi8_launch_count() < 12
    for item in items:
        try:
            L.mi8_test_wait_fault(item, 1 << 14)
            first_step()
        finally:
            L.mi8_test_wait_fault(-1, 0)
        assert _expect_status_then_clear(L, ops, stepper.ws) in (101, 102, 103, 104)
        got = first_step()
        assert ops.poll_status() == 0
        for a, b in zip(got[:3], want[:3]):
            assert np.array_equal(a, b)
