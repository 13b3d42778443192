"""Parameters that a caller rewrites in place count from the next step on: the driver reads them where they were registered.  (Matrices that share an
intgemm8 launch are copied one behind the other at the first step; those stay as they are here.)"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(cfg, batch, longest, seed):
    rng = np.random.default_rng(seed)
    lens = np.sort(rng.integers(max(1, longest - 3), longest + 1, size=batch))[::-1]
    ids = np.full((batch, int(lens[0]) + 1), cfg.eos_id, np.int64)
    mask = np.zeros(ids.shape, np.float32)
    for row, n in enumerate(lens):
        ids[row, :n] = rng.integers(4, cfg.vocab, size=n)
        mask[row, :n + 1] = 1.0
    return torch.from_numpy(ids), torch.from_numpy(mask)


def _stepper(net, batch, beam, longest):
    from marian_dev_b200 import decoder
    return decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=longest + 1, max_steps=longest + 12)


def _search(net, stepper, beam, ids, mask):
    from marian_dev_b200 import decoder, ops
    out = decoder.BeamSearch(net, beam, 1.1, 1.0, native=stepper).search(ids, mask)
    assert ops.poll_status() == 0
    return [(list(t), np.float32(s)) for t, s in out]


def _models(cuda_device, scheme, rnn, dim):
    from marian_dev_b200 import decoder, model
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=8 if dim <= 512 else dim // 64, enc_depth=1, dec_depth=2, vocab=1024,
                                  decoder_autoreg="rnn" if rnn else "self-attention")
    nets = []
    for seed in (3, 4):
        params = model.random_init(cfg, seed)
        rng = np.random.default_rng(seed)
        for name, val in params.items():
            if "_ln_" in name or "_b" in name:
                params[name] = (val + 0.2 * rng.standard_normal(val.shape)).astype(np.float32)
        nets.append(decoder.Int8Transformer(cfg, params, cuda_device, scheme=scheme))
    return cfg, nets


# few rows (all layers of an SSRU decoder in one launch) and more (a launch per operation); models with self-attention
@pytest.mark.parametrize("dim,rnn,batch,beam", [(256, True, 1, 1), (256, True, 8, 4), (512, True, 16, 1), (256, True, 33, 1), (256, False, 4, 2)])
def test_rewritten_in_place(cuda_device, dim, rnn, batch, beam):
    cfg, (net, other) = _models(cuda_device, "intgemm8", rnn, dim)
    ids, mask = _batch(cfg, batch, 9, batch)
    stepper = _stepper(net, batch, beam, 9)
    before = _search(net, stepper, beam, ids, mask)
    alone = ("ffn_W1", "ffn_W2", "_Wo", "context_Wq")          # (matrices with a launch of their own; their multipliers lie behind them)
    for name, p in net.p.items():
        if name != "Wemb":
            p.copy_(other.p[name])
    for name, w in net.w.items():
        if name.endswith(alone):
            w.storage.copy_(other.w[name].storage)
    after = _search(net, stepper, beam, ids, mask)
    assert after != before
    assert after == _search(net, _stepper(net, batch, beam, 9), beam, ids, mask)


def test_parameters_at_any_float_address(cuda_device):
    """Biases that lie on 4-byte boundaries only are read all the same."""
    from marian_dev_b200.binding import check, lib
    cfg, (net, _) = _models(cuda_device, "intgemm8", True, 256)
    ids, mask = _batch(cfg, 4, 9, 1)
    want = _search(net, _stepper(net, 4, 2, 9), 2, ids, mask)
    stepper = _stepper(net, 4, 2, 9)
    moved = []
    for name, p in net.p.items():
        if "_b" in name and "_ln_" not in name:
            room = torch.empty(p.numel() + 1, device=cuda_device)
            room[1:] = p.reshape(-1)
            moved.append(room)
            check(lib().mi8d_set_param(stepper.h, name.encode(), room[1:].data_ptr()))
    assert len(moved) > 8
    assert _search(net, stepper, 2, ids, mask) == want


# packed8avx512: matrices that share a launch stay where they are, with their columns' scales, zero points and offsets (a tile per CTA and the CTA-pair
# kernel: the encoder of 40 sentences x 50 tokens; an odd number of weight tiles)
@pytest.mark.parametrize("dim,rnn,batch,beam,longest", [(256, True, 3, 1, 9), (256, False, 4, 2, 9), (256, False, 40, 1, 49), (768, False, 60, 1, 49)])
def test_packed8_rewritten_in_place(cuda_device, dim, rnn, batch, beam, longest):
    cfg, (net, other) = _models(cuda_device, "packed8avx512", rnn, dim)
    ids, mask = _batch(cfg, batch, longest, batch)
    stepper = _stepper(net, batch, beam, longest)
    before = _search(net, stepper, beam, ids, mask)
    for name, p in net.p.items():
        if name != "Wemb":
            p.copy_(other.p[name])
    for name, w in net.w.items():
        w.item.copy_(other.w[name].item)          # (scales, zero points and offsets are its tail)
        w.bt.copy_(other.w[name].bt)
    after = _search(net, stepper, beam, ids, mask)
    assert after != before
    assert after == _search(net, _stepper(net, batch, beam, longest), beam, ids, mask)
