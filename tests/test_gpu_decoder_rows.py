"""Few rows of an SSRU decoder: all layers of a step in one cluster launch, and the output layer's write-back that reduces the blocks of the
log-softmax, against the same searches with a launch per operation: tokens and scores are the same bits."""
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


# rows at the edges of the MMA's eight, of a warp's one or two and of what the kernel takes (32 rows of 256 floats, 16 of 512) and one more;
# odd row counts share a head's CTAs unevenly; 1 to 4 layers, 5 (general route); feed-forward widths with an odd number of 16-row tiles per
# CTA and wider than what stays in flight; sources of 1 to 70 positions (attention reads keys 16 or 32 at a time); vocabularies that end
# inside a block of 128; an end-of-sentence bias ends hypotheses and sentences at different steps
@pytest.mark.parametrize("dim,ffn,layers,batch,beam,longest,vocab,eos_bias", [
    (256, 1536, 2, 1, 1, 9, 1003, 0.0), (256, 1536, 2, 1, 4, 22, 513, 2.0), (256, 256, 1, 8, 1, 3, 130, 3.0), (256, 768, 3, 9, 1, 17, 1024, 3.0),
    (256, 1280, 2, 5, 3, 33, 1003, 3.0), (256, 3840, 2, 16, 1, 16, 257, 0.0), (256, 1536, 4, 17, 1, 15, 1003, 3.0), (256, 1536, 2, 31, 1, 7, 999, 3.0),
    (256, 1536, 2, 8, 4, 31, 1003, 3.0), (256, 512, 5, 4, 2, 5, 1003, 0.0), (256, 512, 2, 33, 1, 6, 1003, 3.0), (256, 512, 2, 4, 2, 69, 1003, 0.0),
    (512, 2048, 2, 1, 1, 12, 1003, 0.0), (512, 2048, 2, 3, 5, 20, 1003, 3.0), (512, 1024, 1, 16, 1, 65, 128, 3.0), (512, 2048, 2, 17, 1, 8, 1003, 3.0)])
def test_few_rows_give_the_same_bits(cuda_device, dim, ffn, layers, batch, beam, longest, vocab, eos_bias):
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=ffn, heads=8, enc_depth=1, dec_depth=layers, vocab=vocab, decoder_autoreg="rnn")
    params = model.random_init(cfg, dim + batch)
    params["decoder_ff_logit_out_b"][0, cfg.eos_id] += eos_bias
    net = decoder.Int8Transformer(cfg, params, cuda_device)
    rng = np.random.default_rng(batch + longest)
    batches = []
    for most in (longest, 1):
        lens = np.sort(rng.integers(max(1, most - 4), most + 1, size=batch))[::-1]
        ids = np.full((batch, int(lens[0]) + 1), cfg.eos_id, np.int64)
        mask = np.zeros(ids.shape, np.float32)
        for row, n in enumerate(lens):
            ids[row, :n] = rng.integers(4, cfg.vocab, size=n)
            mask[row, :n + 1] = 1.0
        batches.append((torch.from_numpy(ids), torch.from_numpy(mask)))
    room = {"max_batch": batch, "max_src": longest + 1, "max_steps": int(1.5 * (longest + 1)) + 2}
    got = _search(net, batches, beam, {}, **room)
    # a launch per operation; the same with the output layer's other reduction
    for options in ({"fuse_weights": 0}, {"fuse_weights": 0, "fused_output_max_rows": 4096}):
        want = _search(net, batches, beam, options, **room)
        assert ops.poll_status() == 0
        for a, b in zip(got, want):
            assert [list(t) for t, _ in a] == [list(t) for t, _ in b], options
            assert [np.float32(s) for _, s in a] == [np.float32(s) for _, s in b], options
