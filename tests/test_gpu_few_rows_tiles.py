"""Decoder affines of up to 64 rows in 16-row tiles without splits of 2048, against the same searches in tiles of up to 64 rows (the switch for a shared GPU takes the
place of the rule): tokens and scores are the same bits.  Rows around the rule's limits, both schemes, inner dimensions of 2048 and more."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["intgemm8", "packed8avx512"])
@pytest.mark.parametrize("dim,ffn,rnn,batch,beam", [(256, 2048, False, 16, 1), (256, 2048, False, 17, 1), (256, 2304, False, 8, 4), (512, 2048, False, 16, 4),
                                                    (256, 2048, False, 65, 1), (256, 1024, True, 40, 1)])
def test_same_bits(cuda_device, scheme, dim, ffn, rnn, batch, beam):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=ffn, heads=dim // 64, enc_depth=1, dec_depth=2, vocab=544, decoder_autoreg="rnn" if rnn else "self-attention")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, dim + batch), cuda_device, scheme=scheme)
    ids = torch.from_numpy(np.random.default_rng(batch).integers(4, cfg.vocab, size=(batch, 7)))
    ids[:, -1] = cfg.eos_id
    got = []
    for tile in (0, 64):
        stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=7, max_steps=12)
        stepper.set_option("gemm_tile_rows", tile)
        search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
        got.append([(list(t), np.float32(s)) for _ in range(2) for t, s in search.search(ids, torch.ones(batch, 7))])
        assert ops.poll_status() == 0
    assert got[0] == got[1]
