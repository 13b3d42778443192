"""The work that users of this package have it do, as cases that a timing harness can run.

Four kinds of calls, each through the public entry points:

* ``affine``  - one int8 affine on float activations (``ops.affine`` / ``ops.affineWithReluDropout`` / ``ops.dot``)
* ``packed8`` - one affine in the packed8avx512 scheme (``packed8.gemmInt8Packed``)
* ``convert`` - the int8 conversion of one float weight (``ops.prepareB`` / ``packed8.prepareB``)
* ``decode``  - beam search over mini-batches of sentences on the host (``BeamSearch.search`` / ``SearchPool.run``)

Models are the package's own configurations with random-init weights; sentences have uniform token ids and, as after
sorting a corpus by length, lengths that lie close together within a mini-batch.
"""
import math

import numpy as np
import torch

from marian_dev_b200 import decoder, model, ops, packed8

MAX_LENGTH_FACTOR = 1.5


def _affine(name, m, k, n, relu=False, bias=True, half=False):
    return {"name": name, "kind": "affine", "m": m, "k": k, "n": n, "relu": relu, "bias": bias, "half": half}


def _decode(name, net, batch, beam, shortest, longest, workers=1, batches=1, scheme="intgemm8"):
    return {"name": name, "kind": "decode", "net": net, "batch": batch, "beam": beam, "shortest": shortest, "longest": longest,
            "workers": workers, "batches": batches, "scheme": scheme}


def listed():
    return [
        # the first feed-forward affine of the student's decoder at a batch of four: a call of the smallest kind, all latency
        _affine("affine student ffn", 4, 256, 1536, relu=True),
        # the single-affine configuration: 64 sentences x beam 4 through transformer-base's feed-forward layer
        _affine("affine base ffn", 256, 512, 2048, relu=True),
        # the tied output layer of transformer-big in a decoder step with a few finished hypotheses (odd row count)
        _affine("affine output layer", 250, 1024, 32000),
        # transformer-big's encoder feed-forward layer: 127 sentences of 31 tokens
        _affine("affine encoder ffn", 3937, 1024, 4096, relu=True),
        # logits of a whole mini-batch of reference translations (rescoring), half-precision output
        _affine("affine rescoring logits", 4096, 1024, 32000, half=True),
        # a packed8avx512 model's feed-forward layer in a decoder step
        {"name": "packed8 big ffn", "kind": "packed8", "m": 256, "k": 1024, "n": 4096, "bias": True},
        # on-line conversion of a float model: one feed-forward weight of transformer-big
        {"name": "convert big ffn", "kind": "convert", "k": 1024, "n": 4096, "scheme": "intgemm8"},
        # interactive translation: the student, greedy, one sentence
        _decode("decode student x1", "student", 1, 1, 22, 22),
        # a small request batch on the student, greedy
        _decode("decode student x16", "student", 16, 1, 18, 26),
        # transformer-base, beam 4, 64 sentences
        _decode("decode base x64", "base", 64, 4, 32, 38),
        # transformer-big, beam 4, 128 sentences, one search on the GPU
        _decode("decode big x128", "big", 128, 4, 27, 31),
        # throughput serving: four searches side by side on the GPU, fed from one queue of mini-batches
        _decode("decode big pool", "big", 128, 4, 24, 31, workers=4, batches=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["affine", "affine", "affine", "packed8", "convert", "decode", "decode", "decode"])
    if kind == "affine":
        while True:
            # K is a multiple of 16 (the package's condition), M and N are any numbers
            m, k, n = _log_int(rng, 1, 4096), 16 * _log_int(rng, 16, 256), _log_int(rng, 256, 32000)
            if m * n * k <= 4096 * 1024 * 32000:
                break
        bias = rng.random() < 0.8
        c = _affine("", m, k, n, relu=bias and rng.random() < 0.4, bias=bias, half=rng.random() < 0.2)
    elif kind == "packed8":
        # blocks of 256 x 32 weights have no padding in this scheme
        k, n = 256 * rng.choice([1, 2, 3, 4, 6, 8, 16]), 32 * _log_int(rng, 8, 1000)
        c = {"kind": "packed8", "m": _log_int(rng, 1, 2048 if k <= 1024 else 512), "k": k, "n": n, "bias": rng.random() < 0.8}
    elif kind == "convert":
        scheme = rng.choice(["intgemm8", "intgemm8", "packed8avx512"])
        k, n = (16 * _log_int(rng, 16, 256), _log_int(rng, 256, 8192)) if scheme == "intgemm8" else (256 * rng.randint(1, 16), 32 * _log_int(rng, 8, 256))
        c = {"kind": "convert", "k": k, "n": n, "scheme": scheme}
    else:
        net = rng.choice(["student", "base", "big"])
        beam = 1 if net == "student" and rng.random() < 0.5 else rng.choice([1, 2, 4, 4, 6])
        shortest = _log_int(rng, 5, 40)
        longest = shortest + rng.randint(0, 6)
        workers = rng.choice([1, 1, 1, 2, 4])
        batch = _log_int(rng, 1, 128 if beam <= 4 else 64)
        scheme = rng.choice(["intgemm8", "intgemm8", "intgemm8", "packed8avx512"])
        c = _decode("", net, batch, beam, shortest, longest, workers, workers, scheme)
    c.pop("name", None)
    return c


def _matrix(g, rows, cols, std):
    return torch.randn(rows, cols, generator=g, device="cuda") * std


def _params(cfg, g, scheme):
    """Random-init parameters of a model: matrices already converted, the rest in float as a model file holds it."""
    d, f = cfg.dim_emb, cfg.dim_ffn
    p = {}

    def weight(name, k, n):
        a = math.sqrt(6.0 / (k + n))
        w = (torch.rand(k, n, generator=g, device="cuda") * 2 - 1) * a
        p[name] = ops.prepareB(w) if scheme == "intgemm8" else packed8.prepareB(w)

    def bias(name, n):
        p[name] = _matrix(g, 1, n, 0.01).cpu().numpy()

    def norm(prefix):
        p[prefix + "_ln_scale"] = np.ones((1, d), np.float32)
        p[prefix + "_ln_bias"] = np.zeros((1, d), np.float32)

    def attention(prefix):
        for x in "qkvo":
            weight(prefix + "_W" + x, d, d)
            bias(prefix + "_b" + x, d)
        norm(prefix + "_Wo")

    def ffn(prefix):
        weight(prefix + "_W1", d, f)
        bias(prefix + "_b1", f)
        weight(prefix + "_W2", f, d)
        bias(prefix + "_b2", d)
        norm(prefix + "_ffn")

    p["Wemb"] = _matrix(g, cfg.vocab, d, 1.0 / math.sqrt(d)).cpu().numpy()
    for i in range(1, cfg.enc_depth + 1):
        attention("encoder_l%d_self" % i)
        ffn("encoder_l%d_ffn" % i)
    for i in range(1, cfg.dec_depth + 1):
        if cfg.decoder_autoreg == "rnn":
            weight("decoder_l%d_rnn_W" % i, d, d)
            weight("decoder_l%d_rnn_Wf" % i, d, d)
            bias("decoder_l%d_rnn_bf" % i, d)
            norm("decoder_l%d_rnn_ffn" % i)
        else:
            attention("decoder_l%d_self" % i)
        attention("decoder_l%d_context" % i)
        ffn("decoder_l%d_ffn" % i)
    bias("decoder_ff_logit_out_b", cfg.vocab)
    return p


def _mini_batch(rng, cfg, case):
    """Token ids and 0/1 mask [sentences, width] in pinned host memory, longest sentence first, EOS at each end."""
    lens = np.sort(rng.integers(case["shortest"], case["longest"] + 1, size=case["batch"]))[::-1]
    ids = np.full((case["batch"], int(lens[0]) + 1), cfg.eos_id, np.int64)
    mask = np.zeros(ids.shape, np.float32)
    for row, n in enumerate(lens):
        ids[row, :n] = rng.integers(4, cfg.vocab, size=n)
        mask[row, :n + 1] = 1.0
    return torch.from_numpy(ids).pin_memory(), torch.from_numpy(mask).pin_memory()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("affine", "packed8"):
        m, k, n = case["m"], case["k"], case["n"]
        w = _matrix(g, k, n, 0.02)
        return {"case": case, "x": _matrix(g, m, k, 1.0), "w": ops.prepareB(w) if kind == "affine" else packed8.prepareB(w),
                "b": (torch.randn(n, generator=g, device="cuda") * 0.01) if case["bias"] else None}
    if kind == "convert":
        return {"case": case, "w": _matrix(g, case["k"], case["n"], 0.02)}
    cfg = model.CONFIGS[case["net"]]
    net = decoder.Int8Transformer(cfg, _params(cfg, g, case["scheme"]), torch.device("cuda", torch.cuda.current_device()), scheme=case["scheme"])
    rng = np.random.default_rng(seed)
    batches = [_mini_batch(rng, cfg, case) for _ in range(case["batches"])]
    width = case["longest"] + 1
    room = {"max_batch": case["batch"], "beam": case["beam"], "max_src": width, "max_steps": math.ceil(MAX_LENGTH_FACTOR * width) + 2}
    if case["workers"] > 1:
        search = decoder.SearchPool(net, case["workers"], max_length_factor=MAX_LENGTH_FACTOR, normalize=1.0, **room)
    else:
        stepper = decoder.NativeStepper(net, **room)
        search = decoder.BeamSearch(net, case["beam"], MAX_LENGTH_FACTOR, 1.0, native=stepper)
    return {"case": case, "search": search, "batches": batches, "max_tokens": room["max_steps"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "affine":
        dtype = torch.float16 if case["half"] else torch.float32
        if case["relu"]:
            return ops.affineWithReluDropout(state["x"], state["w"], state["b"], out_dtype=dtype)
        if case["bias"]:
            return ops.affine(state["x"], state["w"], state["b"], out_dtype=dtype)
        return ops.dot(state["x"], state["w"], out_dtype=dtype)
    if kind == "packed8":
        return packed8.gemmInt8Packed(state["x"], state["w"], state["b"])
    if kind == "convert":
        if case["scheme"] == "intgemm8":
            w = ops.prepareB(state["w"])
            return {"data": w.data, "quant_mult": w.quant_mult}
        w = packed8.prepareB(state["w"])
        return {"item": w.item, "bt": w.bt}
    if case["workers"] > 1:
        results = state["search"].run(state["batches"])
    else:
        results = [state["search"].search(ids, mask) for ids, mask in state["batches"]]
    # token matrix of all sentences, -1 behind the end of each
    sentences = [s for r in results for s in r]
    tokens = np.full((len(sentences), state["max_tokens"]), -1, np.int32)
    for row, (toks, _) in enumerate(sentences):
        tokens[row, :len(toks)] = toks
    return {"tokens": tokens, "scores": np.array([score for _, score in sentences], np.float32)}


def work(case):
    kind = case["kind"]
    if kind == "convert":
        k, n = case["k"], case["n"]
        # float weight in, int8 weight out; packed8avx512 keeps the item and its row-major copy
        return {"bytes": 4 * k * n + (k * n + 4 if case["scheme"] == "intgemm8" else 2 * k * n + 12 * n), "flops": 0}
    if kind != "decode":
        m, k, n = case["m"], case["k"], case["n"]
        out = 2 if case.get("half") else 4
        return {"bytes": 4 * m * k + k * n + (4 * n if case["bias"] else 0) + (12 * n if kind == "packed8" else 8) + out * m * n, "flops": 2 * m * n * k}
    cfg = model.CONFIGS[case["net"]]
    d, f, v = cfg.dim_emb, cfg.dim_ffn, cfg.vocab
    own = (2 if cfg.decoder_autoreg == "rnn" else 4) * d * d
    width = (case["shortest"] + case["longest"]) // 2 + 1
    steps = math.ceil(MAX_LENGTH_FACTOR * width)
    words = case["batch"] * width
    rows = case["batch"] * (1 + case["beam"] * (steps - 1))          # hypotheses over all steps
    enc = words * cfg.enc_depth * (4 * d * d + 2 * d * f + 2 * d * width)
    kv = words * cfg.dec_depth * 2 * d * d
    history = 0 if cfg.decoder_autoreg == "rnn" else 2 * d * steps / 2
    dec = rows * (cfg.dec_depth * (own + 2 * d * d + 2 * d * f + 2 * d * width + history) + d * v)
    weights = cfg.enc_depth * (4 * d * d + 2 * d * f) + cfg.dec_depth * (own + 4 * d * d + 2 * d * f) + d * v
    moved = 12 * words + 4 * d * (words + rows) + 4 * case["batch"] * steps    # ids and mask, embedding rows, output tokens
    return {"bytes": weights + case["batches"] * moved, "flops": 2 * case["batches"] * (enc + kv + dec)}


def tolerance(case):
    if case["kind"] in ("decode", "convert"):
        return "exact"                                               # token sequences and their scores; int8 weights
    if case["kind"] == "affine" and case["half"]:
        return {"rel": 1e-3, "max": 2e-3}                            # one rounding to half precision
    return {"rel": 1e-6, "max": 1e-5}                                # exact integer sums, two or three float roundings
