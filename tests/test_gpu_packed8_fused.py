"""packed8avx512 models: the matrices that multiply one activation as one launch against a launch per matrix - the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row, a few, several tiles; an encoder activation large enough for the two-CTA kernel (1024 wide, 2000 rows); both kinds of decoder
@pytest.mark.parametrize("dim,rnn,batch,beam,longest", [(256, False, 1, 1, 7), (256, True, 3, 1, 9), (256, True, 20, 4, 12), (256, False, 9, 3, 21),
                                                        (512, False, 40, 2, 5), (1024, False, 40, 2, 49)])
def test_fused_matrices_give_the_same_bits(cuda_device, dim, rnn, batch, beam, longest):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=dim // 64, enc_depth=1, dec_depth=2, vocab=544,
                                  decoder_autoreg="rnn" if rnn else "self-attention")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, dim + batch), cuda_device, scheme="packed8avx512")
    rng = np.random.default_rng(batch)
    lens = np.sort(rng.integers(max(1, longest - 3), longest + 1, size=batch))[::-1]
    ids = np.full((batch, int(lens[0]) + 1), cfg.eos_id, np.int64)
    mask = np.zeros(ids.shape, np.float32)
    for row, n in enumerate(lens):
        ids[row, :n] = rng.integers(4, cfg.vocab, size=n)
        mask[row, :n + 1] = 1.0
    results = []
    for fuse in (1, 0):
        stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=longest + 1, max_steps=longest + 12)
        stepper.set_option("fuse_weights", fuse)
        search = decoder.BeamSearch(net, beam, 1.1, 1.0, native=stepper)
        results.append([(list(t), np.float32(s)) for t, s in search.search(torch.from_numpy(ids), torch.from_numpy(mask))])
        assert ops.poll_status() == 0
    assert results[0] == results[1]
