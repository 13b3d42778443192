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


@pytest.mark.parametrize("beam,n_best", [(128, 8), (129, 8), (160, 8), (257, 4)])
@pytest.mark.parametrize("fused_output", [0, 512])
def test_step_of_a_wide_beam(cuda_device, beam, n_best, fused_output):
    """mi8d_step takes as many hypotheses per sentence as the driver has rows: up to 1024 candidates the n-best lists are merged by the
    step's last kernel, beyond by a launch of their own."""
    import ctypes
    from marian_dev_b200 import decoder, model, ops
    cfg = model.CONFIGS["tiny-ssru"]
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, 3), cuda_device)
    stepper = decoder.NativeStepper(net, max_batch=1, beam=beam, max_src=6, max_steps=8)
    stepper.set_option("fused_output_max_rows", fused_output)
    rng = np.random.default_rng(beam)
    ids = torch.from_numpy(rng.integers(4, cfg.vocab, (1, 5))).to(cuda_device)
    stepper.encode(ids, torch.ones(1, 5, device=cuda_device))
    stepper.step(None, None, None, None, 1, 1, n_best)
    words = rng.integers(4, cfg.vocab, beam)
    words[beam // 2:] = words[:beam - beam // 2]                     # equal hypotheses with equal scores: ties across the beam
    prev = rng.integers(-3, 1, beam).astype(np.float32)
    prev[beam // 2:] = prev[:beam - beam // 2]
    prev[0] = -np.inf                                                # a dummy hypothesis
    score, hyp, word, *_ = stepper.step(np.zeros(beam, np.int64), words, np.zeros(1, np.int64), prev, beam, 1, n_best)
    assert ops.poll_status() == 0
    # the same step again on a second driver that keeps its logits; candidates and lists through the separate kernels
    ref = decoder.NativeStepper(net, max_batch=1, beam=beam, max_src=6, max_steps=8)
    ref.check(ref.L.mi8d_keep_logits(ref.h, 1))
    ref.encode(ids, torch.ones(1, 5, device=cuda_device))
    ref.step(None, None, None, None, 1, 1, n_best)
    ref.step(np.zeros(beam, np.int64), words, np.zeros(1, np.int64), prev, beam, 1, 1)
    cs = torch.empty(beam, n_best, device=cuda_device)
    cw = torch.empty(beam, n_best, dtype=torch.int32, device=cuda_device)
    out = [torch.empty(n_best, dtype=t, device=cuda_device) for t in (torch.float32, torch.int32, torch.int32)]
    pd = torch.from_numpy(prev).to(cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    ref.check(ref.L.mi8g_lse_topk(ctypes.c_void_p(ref.L.mi8d_last_logits(ref.h)), beam, cfg.vocab, n_best, pd.data_ptr(), cs.data_ptr(), cw.data_ptr(), stream))
    ref.check(ref.L.mi8g_nbest_merge(cs.data_ptr(), cw.data_ptr(), beam, 1, cfg.vocab, n_best, *[o.data_ptr() for o in out], stream))
    torch.cuda.synchronize()
    assert np.array_equal(score[0], out[0].cpu().numpy())
    assert np.array_equal(hyp[0], out[1].cpu().numpy()) and np.array_equal(word[0], out[2].cpu().numpy())
