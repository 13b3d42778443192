"""Parameters and weights that this library's own kernels write directly in front of the launch that reads them: the launch takes the new values, although
launches overlap and fetch what does not change from call to call before the kernel in front is done.  (A longer kernel of the library goes first, so that the
writer is still at work when the next launch is due.)"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _copy(dst, src):
    """dst = src, by a kernel of the library."""
    from marian_dev_b200.binding import check, lib
    check(lib().mi8_transpose_f32(src.data_ptr(), 1, 1, src.numel(), dst.data_ptr(), _stream()))


def _max_into(multiplier, x, ws):
    """*multiplier = 127 / max|x|, by a kernel of the library."""
    from marian_dev_b200.binding import check, lib
    check(lib().mi8_max_absolute_f32(x.data_ptr(), x.numel(), None, multiplier.data_ptr(), ws.ptr, ws.nbytes, _stream()))


class _Busy:
    def __init__(self, device):
        self.x = torch.randn(2048, 2048, device=device)
        self.y = torch.empty_like(self.x)

    def __call__(self):
        from marian_dev_b200.binding import check, lib
        check(lib().mi8_transpose_f32(self.x.data_ptr(), 1, 2048, 2048, self.y.data_ptr(), _stream()))


@pytest.mark.parametrize("dim,batch", [(256, 1), (256, 8), (512, 4)])
@pytest.mark.parametrize("last", ["ffn_ffn_ln_bias", "rnn_bf", "ffn_b2", "context_Wo_ln_scale", "ffn_W1"])
def test_decoder_step(cuda_device, dim, batch, last):
    """A step of an SSRU decoder whose layers are one launch: the registered vector, or a matrix's multiplier, is written in front of mi8d_step."""
    from marian_dev_b200 import decoder, model, ops
    cfg = model.TransformerConfig(dim_emb=dim, dim_ffn=2 * dim, heads=8, enc_depth=1, dec_depth=2, vocab=515, decoder_autoreg="rnn")
    net = decoder.Int8Transformer(cfg, model.random_init(cfg, dim), cuda_device)
    stepper = decoder.NativeStepper(net, max_batch=batch, beam=1, max_src=5, max_steps=8)
    g = torch.Generator(device=cuda_device).manual_seed(batch)
    ctx, mask = torch.randn(batch, 5, dim, generator=g, device=cuda_device), torch.zeros(batch, 5, device=cuda_device)
    name = "decoder_l2_" + last
    matrix = name in net.w
    assert matrix or name in net.p, sorted(net.p)
    param = net.w[name].quant_mult if matrix else net.p[name].view(-1)
    values = [torch.randn(64 if matrix else param.numel(), generator=g, device=cuda_device) * s + 1.0 for s in (0.3, 0.8)]
    ws, busy = ops.default_workspace(cuda_device), _Busy(cuda_device)

    def step(write):
        stepper.start(ctx, mask)
        write()
        return stepper.step(None, None, None, None, 1, batch, 1)[0].copy()

    def settled(v):
        _max_into(param, v, ws) if matrix else param.copy_(v)
        torch.cuda.synchronize()

    def at_once(v):
        busy()
        _max_into(param, v, ws) if matrix else _copy(param, v)

    want = [step(lambda: settled(v)) for v in values]
    assert not np.array_equal(want[0], want[1])
    for i in range(12):
        assert np.array_equal(step(lambda: at_once(values[i & 1])), want[i & 1])
    assert ops.poll_status() == 0


@pytest.mark.parametrize("m,k,n", [(4, 256, 1536), (1, 1024, 300), (16, 256, 129)])
@pytest.mark.parametrize("entry", ["affine", "slot"])
def test_weight_multiplier(cuda_device, m, k, n, entry):
    """A weight's multiplier written in front of a product that quantises its activation itself."""
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import check, lib
    g = torch.Generator(device=cuda_device).manual_seed(n)
    x = torch.randn(m, k, generator=g, device=cuda_device)
    w = ops.prepareB(torch.randn(k, n, generator=g, device=cuda_device))
    slot = ops.max_absolute(x)
    values = [torch.randn(1 << 18, generator=g, device=cuda_device) * s for s in (0.3, 0.8)]
    ws, busy, scratch = ops.default_workspace(cuda_device), _Busy(cuda_device), torch.empty(m * k + 64, dtype=torch.int8, device=cuda_device)

    def product():
        out = torch.empty(m, n, device=cuda_device)
        if entry == "affine":
            check(lib().mi8_affine_f32(x.data_ptr(), m, k, w.data.data_ptr(), w.quant_mult.data_ptr(), n, None, 1.0, 0, out.data_ptr(), 0, scratch.data_ptr(), ws.ptr,
                                       ws.nbytes, _stream()))
        else:
            check(lib().mi8_multiply_f32_slot(x.data_ptr(), slot.data_ptr(), None, w.data.data_ptr(), m, n, k, w.quant_mult.data_ptr(), 1.0, None, 0, out.data_ptr(), 0,
                                              None, _stream()))
        return out

    want = []
    for v in values:
        _max_into(w.quant_mult, v, ws)
        torch.cuda.synchronize()
        want.append(product())
    assert not torch.equal(want[0], want[1])
    for i in range(12):
        busy()
        _max_into(w.quant_mult, values[i & 1], ws)
        assert torch.equal(product(), want[i & 1])
    assert ops.poll_status() == 0


@pytest.mark.parametrize("writer", ["quantize", "prepare_a", "quantize_slot", "prepare_b", "prepare_b_nk"])
@pytest.mark.parametrize("entry,m,k,n", [(e, *s) for e in ("multiply", "affine", "slot", "cluster") for s in ((4, 256, 1536), (1, 1024, 300), (64, 512, 512), (300, 2048, 1024))
                                         if not (e == "slot" and s[0] == 300 or e == "cluster" and s[2] == 300)])
def test_weight(cuda_device, m, k, n, writer, entry):
    """A weight quantised by any of the entry points that write int8 matrices, directly in front of the product."""
    from marian_dev_b200 import ops
    from marian_dev_b200.binding import check, lib
    g = torch.Generator(device=cuda_device).manual_seed(n)
    x = torch.randn(m, k, generator=g, device=cuda_device)
    aq, own_slot = ops.prepareA(x), ops.max_absolute(x)
    ws, busy, scratch = ops.Workspace(cuda_device), _Busy(cuda_device), torch.empty(m * k + 64, dtype=torch.int8, device=cuda_device)
    own = ops.Workspace(cuda_device)
    values = [torch.randn(n, k, generator=g, device=cuda_device) for _ in range(2)]
    slots = [ops.max_absolute(v) for v in values]
    multipliers = [127.0 / s for s in slots]
    turned = [v.t().contiguous() for v in values]
    bt, qb = torch.zeros(n, k, dtype=torch.int8, device=cuda_device), torch.ones(1, device=cuda_device)

    def write(i):
        v, st = values[i], _stream()
        if writer == "quantize":
            check(lib().mi8_quantize_f32_i8(v.data_ptr(), v.numel(), multipliers[i].data_ptr(), bt.data_ptr(), st))
        elif writer == "prepare_a":
            check(lib().mi8_prepare_a_f32(v.data_ptr(), n, k, bt.data_ptr(), qb.data_ptr(), ws.ptr, ws.nbytes, st))
        elif writer == "quantize_slot":
            check(lib().mi8g_quantize_slot(v.data_ptr(), v.numel(), slots[i].data_ptr(), bt.data_ptr(), qb.data_ptr(), st))
        else:
            nk = writer == "prepare_b_nk"
            check(lib().mi8_prepare_b_f32((v if nk else turned[i]).data_ptr(), k, n, int(nk), bt.data_ptr(), qb.data_ptr(), ws.ptr, ws.nbytes, st))

    def product():
        out = torch.empty(m, n, device=cuda_device)
        if entry == "affine":
            check(lib().mi8_affine_f32(x.data_ptr(), m, k, bt.data_ptr(), qb.data_ptr(), n, None, 1.0, 0, out.data_ptr(), 0, scratch.data_ptr(), own.ptr, own.nbytes,
                                       _stream()))
        elif entry == "slot":
            check(lib().mi8_multiply_f32_slot(x.data_ptr(), own_slot.data_ptr(), None, bt.data_ptr(), m, n, k, qb.data_ptr(), 1.0, None, 0, out.data_ptr(), 0, None,
                                              _stream()))
        elif entry == "cluster":
            check(lib().mi8g_affine_slot(x.data_ptr(), own_slot.data_ptr(), bt.data_ptr(), qb.data_ptr(), m, n, k, 1.0, None, 0, out.data_ptr(), None, 0, 0, _stream()))
        else:
            check(lib().mi8_multiply_i8(aq.data.data_ptr(), bt.data_ptr(), m, n, k, aq.quant_mult.data_ptr(), qb.data_ptr(), 1.0, None, 0, out.data_ptr(), 0, None,
                                        own.ptr, own.nbytes, _stream()))
        return out

    want = []
    for i in range(2):
        write(i)
        torch.cuda.synchronize()
        want.append(product())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    for i in range(8):
        busy()
        write(i & 1)
        assert torch.equal(product(), want[i & 1])
    assert ops.poll_status() == 0
