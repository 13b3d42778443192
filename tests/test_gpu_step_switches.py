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
