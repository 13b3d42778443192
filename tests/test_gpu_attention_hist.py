"""Self-attention over the stored history for all hypotheses of a sentence together (their distinct ancestor rows, each read once), inside whole
searches against the CPU checker's: every sequence and score identical."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# two to eight hypotheses; models narrower than a block's 128 dimensions, with a last block that is not full, and wider; heads of 32 and 64;
# histories of more than one and two stages of sixteen rows; an end-of-sentence bias leaves dummy hypotheses and empties the batch; more than 256
# positions (the rows are listed 256 at a time); six hypotheses of more than 113 positions, which attention1_kernel takes over
@pytest.mark.parametrize("dim,heads,beam,batch,longest,eos_bias", [
    (64, 2, 2, 3, 24, 0.0), (64, 1, 8, 2, 9, 0.0), (192, 3, 5, 4, 13, 3.0), (192, 6, 3, 7, 22, 3.0), (256, 4, 6, 5, 12, 3.0), (256, 8, 4, 1, 44, 0.0),
    (64, 1, 2, 1, 190, -5.0), (64, 2, 6, 1, 90, -5.0)])
def test_beams_share_their_history(cuda_device, dim, heads, beam, batch, longest, eos_bias):
    from marian_dev_b200 import decoder, model, ops
    from oracle.decode_oracle import OracleTransformer, beam_search
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=heads, enc_depth=1, dec_depth=2, vocab=515)
    params = model.random_init(cfg, dim + beam)
    params["decoder_ff_logit_out_b"][0, cfg.eos_id] += eos_bias
    net = decoder.Int8Transformer(cfg, params, cuda_device)
    ref = OracleTransformer(cfg, params, threads=8)
    steps = int(1.5 * (longest + 1)) + 2
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=longest + 1, max_steps=steps)
    search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
    corpus = model.synthetic_corpus(2 * batch, cfg.vocab, beam, "uniform", max(2, longest - 4), longest)
    for _sid, ids, mask in model.make_batches(corpus, batch):
        got = [(list(t), np.float32(x)) for t, x in search.search(ids, mask)]
        assert ops.poll_status() == 0
        assert got == [(list(t), np.float32(x)) for t, x in beam_search(ref, ids, mask, beam=beam)]
