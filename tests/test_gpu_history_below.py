"""The earlier history slabs' keys and values in the launch of the newest slab's projections, against a launch of their own: tokens and scores are the same bits.  Tiles
of every width with whole and ragged ends, searches that pass the limit of the earlier slabs' length, rows beyond the limit; beams change the history's abs-max
(and with it what is recomputed) often, single hypotheses rarely; an end-of-sentence bias lets rows and sentences leave."""
import ctypes

import numpy as np
import pytest
import torch

from tests.kernel_args import arguments

pytestmark = pytest.mark.gpu


def _search(net, cfg, batch, beam, width, side, ids):
    from marian_dev_b200 import decoder
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=width, max_steps=2 * width)
    stepper.set_option("side_stream", side)
    search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
    out = [(list(t), np.float32(s)) for _ in range(2) for t, s in search.search(ids, torch.ones(batch, width))]
    check(lib().mi8_kernel_times_begin())
    search.search(ids, torch.ones(batch, width))
    buf, n = (Mi8KernelTime * 64)(), ctypes.c_int(0)
    check(lib().mi8_kernel_times_end(buf, 64, ctypes.byref(n)))
    return out, sum(r.launches for r in buf[:n.value] if (arguments("mi8_gemm_kernel", r.name.decode()) or {}).get("kBelow"))


@pytest.mark.parametrize("dim,heads,batch,beam,width,eos_bias,launches", [
    (128, 2, 1, 1, 9, 0.0, True), (128, 2, 16, 1, 12, 0.0, True), (256, 4, 17, 1, 9, 2.0, True), (128, 2, 65, 1, 9, 0.0, True), (128, 2, 129, 1, 9, 2.0, True),
    (256, 4, 4, 4, 13, 2.0, True), (256, 4, 7, 3, 13, 2.0, True), (256, 4, 16, 4, 9, 0.0, True), (256, 4, 17, 4, 9, 2.0, True), (384, 6, 64, 4, 9, 2.0, True),
    (256, 4, 128, 4, 16, 0.0, True), (128, 2, 129, 4, 5, 0.0, False)])
def test_same_bits(cuda_device, dim, heads, batch, beam, width, eos_bias, launches):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=heads, enc_depth=1, dec_depth=2, vocab=515)
    params = model.random_init(cfg, dim + batch)
    params["decoder_ff_logit_out_b"][0, cfg.eos_id] += eos_bias
    net = decoder.Int8Transformer(cfg, params, cuda_device)
    ids = torch.from_numpy(np.random.default_rng(batch).integers(4, cfg.vocab, size=(batch, width)))
    ids[:, -1] = cfg.eos_id
    got, n = _search(net, cfg, batch, beam, width, 1, ids)
    want, none = _search(net, cfg, batch, beam, width, 0, ids)
    assert got == want and none == 0 and (n > 0) == launches and ops.poll_status() == 0
    if (batch, beam, width) == (128, 4, 16):     # (the later steps' slabs are too long)
        assert n < 2 * (int(1.5 * width) - 1)
