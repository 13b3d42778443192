"""A decoder step's merged launches - LayerNorm with the quantisation of its result for few rows, query/key/value projections of the
newest history slab in one GEMM - against the same step with separate launches: the tokens and scores are the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _search(net, batches, beam, options, **room):
    from marian_dev_b200 import decoder
    stepper = decoder.NativeStepper(net, beam=beam, **room)
    for name, value in options.items():
        stepper.set_option(name, value)
    search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
    return [search.search(ids, mask) for ids, mask in batches]


# rows of the merged LayerNorm launch: one or two (one CTA), the ends of what eight CTAs hold (dim 256: 128 rows, 384: 80, 512: 64,
# 1024: 32) and the first counts that take separate launches; 384 is not a multiple of the CTA pair's 256 weight rows
@pytest.mark.parametrize("dim,rnn,batch,beam", [
    (256, True, 1, 1), (256, True, 2, 1), (256, True, 3, 1), (256, True, 17, 1), (256, True, 43, 3), (256, True, 32, 4), (256, True, 26, 5),
    (384, False, 5, 2), (384, False, 27, 3), (384, False, 100, 3), (512, False, 3, 3), (512, False, 16, 4), (512, False, 13, 5),
    (1024, False, 1, 4), (1024, False, 33, 1), (1024, False, 8, 4), (1024, False, 43, 3)])
def test_merged_launches_give_the_same_bits(cuda_device, dim, rnn, batch, beam):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=dim // (32 if dim == 256 else 64), enc_depth=2, dec_depth=2, vocab=1003,
                                  decoder_autoreg="rnn" if rnn else "self-attention")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, dim + batch), cuda_device)
    rng = np.random.default_rng(batch)
    batches = []
    for longest in (3, 9):
        lens = np.sort(rng.integers(max(1, longest - 3), longest + 1, size=batch))[::-1]
        ids = np.full((batch, int(lens[0]) + 1), cfg.eos_id, np.int64)
        mask = np.zeros(ids.shape, np.float32)
        for row, n in enumerate(lens):
            ids[row, :n] = rng.integers(4, cfg.vocab, size=n)
            mask[row, :n + 1] = 1.0
        batches.append((torch.from_numpy(ids), torch.from_numpy(mask)))
    room = {"max_batch": batch, "max_src": 10, "max_steps": 17}
    got = _search(net, batches, beam, {}, **room)
    for options in ({"quant_in_gemm": 1, "fuse_weights": 0}, {"side_stream": 0}, {"side_stream": 1}, {"gemm_tile_rows": 512}):
        want = _search(net, batches, beam, options, **room)
        assert ops.poll_status() == 0
        for a, b in zip(got, want):
            assert [list(t) for t, _ in a] == [list(t) for t, _ in b], options
            assert [np.float32(s) for _, s in a] == [np.float32(s) for _, s in b], options
