"""Decoder affines of up to 64 rows in 16-row tiles without splits of 2048: tokens and scores are the same bits as with the switch for a shared GPU, which takes the
place of the rule in intgemm8's affines, and as the CPU checker's decode, for both schemes; the launches are those tiles where the rule says so and no others.  The
product itself in such tiles, unsplit, against wider tiles and split, and against 64-bit integers.  Rows around the rule's limits, inner dimensions of 2048 and more."""
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


def _items(params):
    from marian_dev_b200.model import is_intgemm_param
    from oracle.oracle import Packed8Oracle
    chk = Packed8Oracle()
    items = {name: chk.prepare_b(np.ascontiguousarray(val, np.float32)) for name, val in params.items() if is_intgemm_param(name)}
    items["Wemb_packed8"] = chk.prepare_b(np.ascontiguousarray(params["Wemb"].T, dtype=np.float32))
    return items


@pytest.mark.parametrize("scheme", ["intgemm8", "packed8avx512"])
@pytest.mark.parametrize("dim,ffn,rnn,batch,beam,tiles", [(256, 2048, False, 17, 1, {16}), (256, 2048, False, 16, 4, {16}), (512, 2048, False, 8, 4, {16}),
                                                          (256, 2048, False, 65, 1, {128}), (256, 1024, True, 40, 1, {16})])
def test_like_the_checker(cuda_device, scheme, dim, ffn, rnn, batch, beam, tiles):
    import ctypes

    from marian_dev_b200 import decoder, model, ops
    from marian_dev_b200.binding import Mi8KernelTime, check, lib
    from oracle.decode_oracle import OracleTransformer, beam_search
    from tests.kernel_args import arguments
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=ffn, heads=dim // 64, enc_depth=1, dec_depth=1, vocab=544, decoder_autoreg="rnn" if rnn else "self-attention")
    params = model.random_init(cfg, dim + batch)
    ids = np.random.default_rng(batch).integers(4, cfg.vocab, size=(batch, 5))
    ids[:, -1] = cfg.eos_id
    mask = np.ones((batch, 5), np.float32)
    ref = OracleTransformer(cfg, params, threads=8, **({"scheme": scheme, "packed_items": _items(params)} if scheme == "packed8avx512" else {}))
    net = decoder.Int8Transformer(cfg, params, cuda_device, scheme=scheme)
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=beam, max_src=5, max_steps=10)
    search = decoder.BeamSearch(net, beam, 1.5, 1.0, native=stepper)
    got = search.search(ids, mask)
    check(lib().mi8_kernel_times_begin())
    try:
        again = search.search(ids, mask)
    finally:
        records, n = (Mi8KernelTime * 64)(), ctypes.c_int(0)
        check(lib().mi8_kernel_times_end(records, 64, ctypes.byref(n)))
    want = beam_search(ref, ids, mask, beam=beam)
    assert [list(t) for t, _ in got] == [list(t) for t, _ in again] == [list(t) for t, _ in want]
    assert [np.float32(s) for _, s in got] == [np.float32(s) for _, s in again] == [np.float32(s) for _, s in want]
    assert ops.poll_status() == 0
    used = [arguments("mi8_gemm_kernel", r.name.decode()) for r in records[:n.value]]
    used = {u["TM"] for u in used if u is not None and not u["kBelow"]}
    assert (16 in used) == (16 in tiles), used


@pytest.mark.parametrize("m", [17, 31, 32, 48, 63, 64])
@pytest.mark.parametrize("k,n", [(2048, 512), (1024, 300), (2048, 129)])
def test_product(cuda_device, m, k, n):
    from marian_dev_b200 import ops, packed8
    g = torch.Generator(device=cuda_device).manual_seed(m + n)
    x, w, b = (torch.randn(*s, generator=g, device=cuda_device) for s in ((m, k), (k, n), (n,)))
    aq, wq = ops.prepareA(x), ops.prepareB(w)
    exact = (aq.data.view(m, k).double() @ wq.data.view(n, k).double().t()).to(torch.int32)
    want = ops.multiply(aq, wq, b, tile_m=64, splits=1)
    for tile, splits in ((16, 1), (32, 2), (64, 2), (0, 0)):
        acc = torch.empty(m, n, dtype=torch.int32, device=cuda_device)
        out = ops.multiply(aq, wq, b, tile_m=tile, splits=splits, acc_out=acc)
        assert torch.equal(acc, exact) and torch.equal(out, want), (tile, splits)
    if k % 256 == 0 and n % 32 == 0:
        p = packed8.quantize_rows(x)
        wp = packed8.prepareB(w)
        exact = (p[0].double() @ wp.bt.view(n, k).double().t()).to(torch.int32)
        want = packed8.multiply(*p, wp, b, tile_m=64, splits=1)
        for tile, splits in ((16, 1), (32, 2), (64, 2), (0, 0)):
            out, acc = packed8.multiply(*p, wp, b, tile_m=tile, splits=splits, want_acc=True)
            assert torch.equal(acc, exact) and torch.equal(out, want), (tile, splits)
    assert ops.poll_status() == 0
