"""Steps of an SSRU decoder launched before the host has seen the lists of the step in front, against the same searches step by step: tokens and scores are the
same bits, whether hypotheses and sentences end at every step, at some or at none, with one search and with several side by side."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(cuda_device, dim, vocab, eos_bias, seed):
    from marian_dev_b200 import decoder, model
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=8, enc_depth=1, dec_depth=2, vocab=vocab, decoder_autoreg="rnn")
    params = model.random_init(cfg, seed)
    params["decoder_ff_logit_out_b"][0, cfg.eos_id] += eos_bias
    return cfg, decoder.Int8Transformer(cfg, params, cuda_device)


def _batch(cfg, batch, width, seed):
    rng = np.random.default_rng(seed)
    ids = torch.from_numpy(rng.integers(4, cfg.vocab, size=(batch, width)))
    ids[:, -1] = cfg.eos_id
    return ids, torch.ones(batch, width)


def _bits(results):
    return [[(list(t), np.float32(s)) for t, s in r] for r in results]


# one row, and rows that fill the cluster launch's 32 (16 of 512 floats); beams whose first step has fewer rows than the next, and whose second step no longer
# fits the launch (9 x 4); an end-of-sentence bias from none to one that ends almost everything at once; factors that end the search before and at its first step
@pytest.mark.parametrize("dim,batch,beam,vocab,eos_bias,factor", [
    (256, 1, 1, 1003, 0.0, 1.5), (256, 1, 8, 1003, 3.0, 1.5), (256, 32, 1, 130, 3.0, 1.5), (256, 8, 4, 1003, 3.0, 1.5), (256, 8, 4, 257, 6.0, 1.5),
    (256, 9, 4, 1003, 3.0, 1.5), (256, 5, 3, 1003, 30.0, 1.5), (512, 4, 4, 1003, 3.0, 1.5), (512, 16, 1, 1003, 2.0, 1.5), (256, 4, 2, 1003, 0.0, 0.2),
    (256, 4, 2, 1003, 0.0, 0.1)])
def test_same_bits(cuda_device, dim, batch, beam, vocab, eos_bias, factor):
    from marian_dev_b200 import decoder, ops
    cfg, net = _net(cuda_device, dim, vocab, eos_bias, dim + batch)
    width = 11
    batches = [_batch(cfg, batch, width, s) for s in range(3)]
    got = {}
    for ahead in (1, 0):
        stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=width, max_steps=int(1.5 * width) + 2)
        stepper.set_option("step_ahead", ahead)
        search = decoder.BeamSearch(net, beam, factor, 1.0, native=stepper)
        got[ahead] = _bits([search.search(*b) for b in batches])
        assert ops.poll_status() == 0
    assert got[1] == got[0]


@pytest.mark.parametrize("wait", [0, 1, 2])
def test_kinds_of_waiting(cuda_device, wait):
    from marian_dev_b200 import decoder
    cfg, net = _net(cuda_device, 256, 515, 3.0, 1)
    b = _batch(cfg, 6, 9, 1)
    got = []
    for value in (wait, 0):
        stepper = decoder.NativeStepper(net, max_batch=6, beam=2, max_src=9, max_steps=16)
        stepper.set_option("blocking_wait", value)
        got.append(_bits([decoder.BeamSearch(net, 2, 1.5, 1.0, native=stepper).search(*b)]))
    assert got[0] == got[1]


@pytest.mark.parametrize("workers", [2, 4])
def test_searches_side_by_side(cuda_device, workers):
    from marian_dev_b200 import decoder, ops
    cfg, net = _net(cuda_device, 256, 1003, 3.0, 7)
    batches = [_batch(cfg, 6, 12, s) for s in range(3 * workers)]
    pool = decoder.SearchPool(net, workers, beam=4, max_batch=6, max_src=12, max_steps=20)
    got = _bits(pool.run(batches))
    stepper = decoder.NativeStepper(net, max_batch=6, beam=4, max_src=12, max_steps=20)
    stepper.set_option("step_ahead", 0)
    search = decoder.BeamSearch(net, 4, 1.5, 1.0, native=stepper)
    assert got == _bits([search.search(*b) for b in batches]) and ops.poll_status() == 0
