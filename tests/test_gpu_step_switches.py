"""Which of two routes a decoder step takes, by its sizes and by the switch that chooses: both give the same bits."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernels(run):
    """What `run` returns, and the launches per kernel that it made."""
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    L = lib()
    check(L.mi8_kernel_times_begin())
    out = run()
    buf = (Mi8KernelTime * 64)()
    n = ctypes.c_int(0)
    check(L.mi8_kernel_times_end(buf, 64, ctypes.byref(n)))
    return out, {r.name.decode(): r.launches for r in buf[:n.value]}


def _searches(cuda_device, dim, heads, rnn, beam, batch, switch, values, width=9):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=heads, enc_depth=1, dec_depth=2, vocab=515,
                                  decoder_autoreg="rnn" if rnn else "self-attention")
    params = model.random_init(cfg, dim + beam)
    net = decoder.Int8Transformer(cfg, params, cuda_device)
    rng = np.random.default_rng(batch)
    ids = torch.from_numpy(rng.integers(4, cfg.vocab, size=(batch, width)))
    ids[:, -1] = cfg.eos_id
    out = []
    for value in values:
        stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=width, max_steps=2 * width)
        if value is not None:
            stepper.set_option(switch, value)
        res, names = _kernels(lambda: decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper).search(ids, torch.ones(batch, width)))
        assert ops.poll_status() == 0
        out.append(([(list(t), np.float32(s)) for t, s in res], names))
    return out


# hypotheses per sentence x sentences on both sides of the rule
@pytest.mark.parametrize("dim,heads,beam,batch,shared", [(64, 1, 1, 3, False), (64, 2, 2, 40, True), (192, 3, 4, 70, True), (128, 2, 5, 32, True),
                                                         (128, 4, 5, 33, False), (64, 1, 6, 32, True), (64, 1, 6, 33, False), (64, 1, 7, 2, False)])
def test_hypotheses_share_their_history(cuda_device, dim, heads, beam, batch, shared):
    on, off = _searches(cuda_device, dim, heads, False, beam, batch, "shared_history", (None, 0))
    assert on[0] == off[0]
    assert any("attention_hist_kernel" in n for n in on[1]) == shared
    assert not any("attention_hist_kernel" in n for n in off[1])


# rows around what the cluster launch takes, and around the limit that a pool of several searches sets
@pytest.mark.parametrize("dim,batch,limit,one", [(256, 32, None, True), (256, 33, None, False), (256, 24, 24, True), (256, 25, 24, False), (512, 16, None, True),
                                                 (512, 17, None, False), (256, 1, 0, False)])
def test_layers_of_a_step_in_one_launch(cuda_device, dim, batch, limit, one):
    got, apart = _searches(cuda_device, dim, 8, True, 1, batch, "one_launch_rows", (limit, 0))
    assert got[0] == apart[0]
    # (sentences end, so later steps may be of few rows again: the first step decides, by its embedding)
    steps = [n for k, n in got[1].items() if "decoder_rows_kernel" in k]
    if limit == 0:
        assert not steps
    elif one:
        assert sum(n for k, n in got[1].items() if "embed_kernel" in k) == 1     # (the encoder's only)
    else:
        assert sum(n for k, n in got[1].items() if "embed_kernel" in k) > 1
    assert not any("decoder_rows_kernel" in k for k in apart[1])


@pytest.mark.parametrize("workers,rows", [(2, 32), (3, 24), (4, 24)])
def test_pools_limit_the_rows(cuda_device, workers, rows):
    """Several searches on one GPU: from three on the cluster launch is for up to 24 rows (a step of 25 rows takes a launch per operation)."""
    from marian_dev_b200 import decoder, model
    cfg = model.TransformerConfig(dim_emb=256, dim_ffn=512, heads=8, enc_depth=1, dec_depth=2, vocab=515, decoder_autoreg="rnn")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, 1), cuda_device)
    pool = decoder.SearchPool(net, workers, beam=1, max_batch=32, max_src=9, max_steps=18)
    for batch in (24, 25, 32):
        for stepper in pool.steppers:
            stepper.start(torch.randn(batch, 7, cfg.dim_emb, device=cuda_device), torch.zeros(batch, 7, device=cuda_device))
            _out, names = _kernels(lambda: stepper.step(None, None, None, None, 1, batch, 1))
            assert any("decoder_rows_kernel" in n for n in names) == (batch <= rows)
