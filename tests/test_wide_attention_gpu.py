"""Head width 256 on the tensor cores (attn_wide_sm100.cu) against a float64 statement of the same
attention and against the exact fp32 kernels, at the edges of its 128-row tiles and 64-row steps."""
import math

import pytest
import torch

from pluto_b200 import _capi
from pluto_b200.layers import AttentionLayer, DataType, gqa_prefill

pytestmark = pytest.mark.gpu
D = 256
# (batch, tokens, query heads, key/value heads): one row, either side of a step and of a tile, several
# tiles, grouped and ungrouped heads, and a shape whose CTAs walk several heads of a group
SHAPES = [(1, 1, 2, 1), (2, 63, 3, 3), (1, 65, 6, 1), (2, 127, 2, 2), (1, 128, 24, 4), (3, 129, 4, 2),
          (1, 257, 6, 2), (1, 640, 12, 2), (1, 1000, 24, 4), (6, 300, 24, 2)]


def make(shape, seed=0):
    b, t, hq, hkv = shape
    gen = torch.Generator(device="cuda").manual_seed(seed + t)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    return rnd(b, t, hq, D).bfloat16(), rnd(b, t, hkv, D).bfloat16(), rnd(b, t, hkv, D).bfloat16(), rnd(b, t, hq, D)


def reference(q, k, v):
    """(output, maxima, normalizers) in float64."""
    b, t, hq, _ = q.shape
    group = hq // k.shape[2]
    kk, vv = (x.double().repeat_interleave(group, 2) for x in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), kk) / math.sqrt(D)
    s = s.masked_fill(torch.triu(torch.ones(t, t, dtype=torch.bool, device="cuda"), 1), -math.inf)
    m = s.amax(-1)
    e = torch.exp(s - m[..., None])
    l = e.sum(-1)
    return torch.einsum("bhqk,bkhd->bqhd", e / l[..., None], vv), m, l


@pytest.mark.parametrize("shape", SHAPES)
def test_forward(shape):
    q, k, v, _ = make(shape)
    want, m, l = reference(q, k, v)
    got = gqa_prefill(q, k, v, want_core=True, want_stats=True)
    # P enters P V with 24 bits and ex2.approx is good to 2^-22; values are sums of |p| <= 1 weighted
    # N(0, 1) entries: 2^-15 absolute is far above that (test_error_is_that_of_fp32_products is the tight one)
    assert (got["core"].double() - want).abs().max().item() < 3.1e-5
    assert torch.equal(got["out"], got["core"].bfloat16())
    assert (got["maxima"].view_as(m).double() - m).abs().max().item() < 1e-5
    assert ((got["normalizers"].view_as(l).double() - l) / l).abs().max().item() < 1e-4


def test_forward_gate_strided_query_and_growing_maxima():
    b, t, hq, hkv = 2, 300, 6, 2
    q, k, v, g = make((b, t, hq, hkv), 3)
    k = (k.float() * torch.linspace(0.2, 6.0, t, device="cuda")[None, :, None, None]).bfloat16()   # rescales in most steps
    both = torch.stack([q, g.bfloat16()], 3)   # [b, t, hq, 2, D]
    want = gqa_prefill(q, k, v, want_core=True)["core"]
    got = gqa_prefill(both[:, :, :, 0], k, v, gate=both[:, :, :, 1], want_core=True)
    assert (want.double() - reference(q, k, v)[0]).abs().max().item() < 6.2e-5   # |s| up to 100: 2^-24 * 100 in the exponent
    assert torch.equal(got["core"], want)
    sigmoid = torch.sigmoid(both[:, :, :, 1].float()).bfloat16().float()
    expected = want.bfloat16().float() * sigmoid
    assert ((got["out"].float() - expected).abs() <= 2 ** -7 * expected.abs() + 1e-30).all()   # one bf16 ulp: rounding ties of the sigmoid


def backward(q, k, v, d_out, stats, workspace):
    b, t, hq, _ = q.shape
    hkv = k.shape[2]
    L, stream = _capi.lib(), torch.cuda.current_stream().cuda_stream
    dq, dk, dv = torch.empty_like(d_out), torch.empty(b, t, hkv, D, device="cuda"), torch.empty(b, t, hkv, D, device="cuda")
    deltas = (d_out * stats["core"]).sum(-1).permute(0, 2, 1).contiguous()
    size = L.pluto_gqa_prefill_bwd_workspace_bytes(b, t, hq, D, 1) if workspace else 0
    ws = torch.empty(size, dtype=torch.uint8, device="cuda") if workspace else None
    _capi.check(L.pluto_gqa_prefill_bwd(stream, q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, hq * D, D, d_out.data_ptr(),
                                        stats["maxima"].data_ptr(), stats["normalizers"].data_ptr(), deltas.data_ptr(),
                                        dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ws.data_ptr() if workspace else None,
                                        size, b, t, hq, hkv, D))
    torch.cuda.synchronize()
    return dq, dk, dv


@pytest.mark.parametrize("shape", SHAPES)
def test_backward_matches_exact_kernels_and_repeats(shape):
    q, k, v, d_out = make(shape)
    stats = gqa_prefill(q, k, v, want_core=True, want_stats=True)
    exact = backward(q, k, v, d_out, stats, False)
    got = backward(q, k, v, d_out, stats, True)
    again = backward(q, k, v, d_out, stats, True)
    for name, x, y, z in zip(("dq", "dk", "dv"), got, exact, again):
        assert torch.equal(x, z), name
        # Every operand carries 24 bits, products accumulate in fp32.  3e-5 of the largest gradient, and where
        # dP - delta cancels (a single visible key: dS is exactly 0) 4e-5, would do for operands of 16 bits
        # (test_error_is_that_of_fp32_products is the tight one).
        scale = y.abs().max().item()
        assert (x - y).abs().max().item() <= 3e-5 * scale + 4e-5, (name, (x - y).abs().max().item(), scale)
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("tokens", [64, 200, 1000])
@pytest.mark.parametrize("std", [0.5, 1.0])
def test_error_is_that_of_fp32_products(tokens, std):
    """Unrounded core and gradients against float64, 2-norm.  The bounds are what fp32 leaves: a score is 256
    products, rounded to some 2^-23 of |s| <= 5, which is the relative error of its probability; the sums
    behind it add a few 2^-24 apiece.  10 * 2^-24 for the core, 14 for the gradients, which go through two
    more products; operands of 16 bits leave 1.5e-6 and 4e-6."""
    q, k, v, d_out = make((1, tokens, 24, 4), 11)
    q, k, v = ((x.float() * std).bfloat16() for x in (q, k, v))
    relative = lambda x, y: ((x.double() - y).norm() / y.norm()).item()
    qd, kd, vd = (x.double().requires_grad_() for x in (q, k, v))
    core = reference(qd, kd, vd)[0]
    core.backward(d_out.double())
    got = gqa_prefill(q, k, v, round_to_bfloat16=False, want_core=True, want_stats=True)
    assert relative(got["core"], core.detach()) < 10 * 2 ** -24
    stats = dict(got, core=core.detach().float())   # deltas as the caller would have them without an error
    for name, x, y in zip(("dq", "dk", "dv"), backward(q, k, v, d_out, stats, True), (qd.grad, kd.grad, vd.grad)):
        assert relative(x, y) < 14 * 2 ** -24, name
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("batch,tokens,heads", [(1, 1, 1), (2, 63, 3), (1, 129, 2), (3, 200, 5), (1, 640, 6)])
def test_packed_layer(batch, tokens, heads):
    """AttentionLayer of width 256 with the scratch it asks for: packed rows of 3 E, gradients of the same
    layout, row terms from its own bf16 output.  Against float64 with that output, bounds as above, and the
    exact kernels; single rows of a sequence have no gradient through the scores."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(batch * tokens, 3 * heads * D, device="cuda", generator=gen).bfloat16()
    d_out = torch.randn(batch * tokens, heads * D, device="cuda", generator=gen)
    layer = AttentionLayer.Create(tokens, heads, heads * D, DataType.BF16)
    result = layer.fwd([x])
    got = layer.bwd([d_out], result.state)[0]
    layer.tensor_core_backward = False
    exact = layer.bwd([d_out], result.state)[0]
    q, k, v = (x.view(batch, tokens, 3, heads, D)[:, :, i].double() for i in range(3))
    out, g = result.outputs[0].view(batch, tokens, heads, D), d_out.view(batch, tokens, heads, D).double()
    want, _, _ = reference(q, k, v)
    assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()   # half a bf16 ulp of the core
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) / math.sqrt(D)
    p = torch.softmax(s.masked_fill(torch.triu(torch.ones(tokens, tokens, dtype=torch.bool, device="cuda"), 1), -math.inf), -1)
    delta = (g * out.double()).sum(-1).permute(0, 2, 1)[..., None]
    ds = p * (torch.einsum("bqhd,bkhd->bhqk", g, v) - delta) / math.sqrt(D)
    grads = (torch.einsum("bhqk,bkhd->bqhd", ds, k), torch.einsum("bhqk,bqhd->bkhd", ds, q), torch.einsum("bhqk,bqhd->bkhd", p, g))
    scale = max(y.norm().item() for y in grads)
    for i, y in enumerate(grads):
        for gradient in (got, exact):
            z = gradient.view(batch, tokens, 3, heads, D)[:, :, i].double()
            # (dP and delta of one row nearly cancel: what their 256 products leave counts against the largest gradient)
            assert (z - y).norm().item() <= 14 * 2 ** -24 * max(y.norm().item(), scale if i < 2 else 0), i
    assert _capi.kernel_status() == 0
