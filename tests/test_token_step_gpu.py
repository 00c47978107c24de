"""The one-launch token steps (token_step.cu) against the launches they replace, through the C ABI:
contexts of one row, either side of a warp's turn and the longest the single launch takes (then the
first it does not), and every shape rule of the delta-net step."""
import pytest
import torch

from pluto_b200 import _capi
from pluto_b200.layers import (CachedAttentionStep, DeltaNetParameters, DeltaNetState, FullAttentionParameters,
                               KeyValueCache, gqa_decode)

pytestmark = pytest.mark.gpu


def stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("heads,dim,rotary", [((24, 4), 256, 64), ((5, 1), 128, 128), ((3, 3), 64, 32)])
@pytest.mark.parametrize("cache_dtype,io_dtype", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("rounded", [True, False])
def test_cached_step_matches_prepare_and_decode(heads, dim, rotary, cache_dtype, io_dtype, rounded):
    hq, hkv = heads
    p = FullAttentionParameters(query_heads=hq, key_value_heads=hkv, head_dim=dim, rotary_dim=rotary, capacity=1030,
                                round_to_bfloat16=rounded)
    gen = torch.Generator(device="cuda").manual_seed(dim)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    keys, values = rnd(1030, hkv, dim).bfloat16(), rnd(1030, hkv, dim).bfloat16()
    wq, wk = rnd(dim) * 0.1, rnd(dim) * 0.1
    L = _capi.fast()
    for position in (0, 1, 15, 16, 17, 500, 1023, 1024, 1029):
        qg, k, v = rnd(hq, 2, dim).to(io_dtype), rnd(hkv, dim).to(io_dtype), rnd(hkv, dim).to(io_dtype)
        caches = []
        for _ in range(2):
            cache = KeyValueCache.Create(1030, hkv, dim, cache_dtype)
            cache.keys().copy_(keys)
            cache.values().copy_(values)
            cache.position_ = position
            caches.append(cache)
        out = torch.empty(hq, dim, device="cuda", dtype=io_dtype)
        CachedAttentionStep(p, caches[0], qg, k, v, wq, wk, out)
        assert caches[0].position() == position + 1
        # the separate entry points
        queries = torch.empty(1, hq, dim, device="cuda", dtype=torch.bfloat16 if rounded else torch.float32)
        at = torch.tensor([position], dtype=torch.int32, device="cuda")
        code = 1 if io_dtype == torch.bfloat16 else 0
        _capi.check(L.pluto_qk_prepare(stream(), qg.data_ptr(), k.data_ptr(), v.data_ptr(), code, 2 * hq * dim, 2 * dim,
                                       wq.data_ptr(), wk.data_ptr(), at.data_ptr(), queries.data_ptr(),
                                       1 if rounded else 0, caches[1].packed_layout(), 1, 1, hq, hkv, dim, rotary,
                                       p.rms_norm_epsilon, p.rope_theta, int(rounded)))
        want = gqa_decode(queries, caches[1].keys()[None], caches[1].values()[None], at + 1, position + 1,
                          gate=qg[None, :, 1], round_to_bfloat16=rounded,
                          out=torch.empty(1, hq, dim, device="cuda", dtype=io_dtype))[0]
        assert torch.equal(caches[0].values(), caches[1].values())
        if rounded:
            assert torch.equal(caches[0].keys(), caches[1].keys())
        else:   # the unrounded rotation may or may not contract into an fma: one rounding of one product
            assert ((caches[0].keys().float() - caches[1].keys().float()).abs() <= 2 ** -7 * caches[1].keys().float().abs() + 1e-6).all()
        # The decode kernels carry P to 2^-17, so unrounded fp32 results agree to 1e-5 of values of order
        # one; with rounding the core and the product can each fall on either side of a tie, one bf16 ulp
        # (at most 2^-7 of the value) apiece.
        bound = (2 ** -6 if rounded or io_dtype == torch.bfloat16 else 1e-5) * want.float().abs() + 2e-5
        assert ((out.float() - want.float()).abs() <= bound).all(), position
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("key_heads,value_heads,dk,dv,taps", [(2, 6, 128, 128, 4), (3, 3, 128, 128, 1), (1, 8, 128, 128, 3),
                                                              (1, 9, 128, 128, 4), (2, 4, 64, 128, 4), (2, 2, 128, 96, 4),
                                                              (1, 2, 128, 128, 5)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rounded", [True, False])
def test_delta_step_matches_its_four_launches(key_heads, value_heads, dk, dv, taps, dtype, rounded):
    p = DeltaNetParameters(key_heads=key_heads, value_heads=value_heads, key_head_dim=dk, value_head_dim=dv,
                           conv_kernel_dim=taps, round_to_bfloat16=rounded)
    gen = torch.Generator(device="cuda").manual_seed(value_heads * 7 + taps)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    kq = key_heads * dk
    channels = 2 * kq + value_heads * dv
    conv, a_log, dt_bias, norm = rnd(channels, taps), rnd(value_heads), rnd(value_heads), rnd(dv)
    state = DeltaNetState.Create(p)
    window = torch.zeros(channels, taps, device="cuda")
    S = torch.zeros(1, value_heads, dk, dv, device="cuda")
    L, code, rnd_flag = _capi.fast(), 1 if dtype == torch.bfloat16 else 0, int(rounded)
    f32 = dict(device="cuda", dtype=torch.float32)
    for _ in range(6):
        qkv, z, a, b = rnd(channels).to(dtype), rnd(value_heads, dv).to(dtype), rnd(value_heads).to(dtype), rnd(value_heads).to(dtype)
        out = torch.empty(value_heads, dv, device="cuda", dtype=dtype)
        state.Step(qkv, z, a, b, conv, a_log, dt_bias, norm, out)
        post, g, beta = torch.empty(channels, **f32), torch.empty(value_heads, **f32), torch.empty(value_heads, **f32)
        core, want = torch.empty(value_heads, dv, **f32), torch.empty_like(out)
        _capi.check(L.pluto_gdn_conv_silu(stream(), qkv.data_ptr(), conv.data_ptr(), code, 1, 1, channels, taps, rnd_flag,
                                          window.data_ptr(), post.data_ptr(), 0))
        _capi.check(L.pluto_gdn_gates(stream(), a.data_ptr(), b.data_ptr(), a_log.data_ptr(), dt_bias.data_ptr(), code, 1,
                                      value_heads, rnd_flag, g.data_ptr(), beta.data_ptr()))
        _capi.check(L.pluto_gdn_step(stream(), post.data_ptr(), post[kq:].data_ptr(), post[2 * kq:].data_ptr(), 0,
                                     g.data_ptr(), beta.data_ptr(), S.data_ptr(), core.data_ptr(), 0, 1, key_heads,
                                     value_heads, dk, dv, 1, 1.0, rnd_flag))
        _capi.check(L.pluto_gdn_out_norm_gate(stream(), core.data_ptr(), 0, z.data_ptr(), code, norm.data_ptr(), value_heads,
                                              dv, p.rms_norm_epsilon, rnd_flag, 1, want.data_ptr(), code))
        assert torch.equal(state.convolution_state_.view_as(window), window)
        # fp32 sums of 128 terms in another order: 128 * 2^-24 = 8e-6 of the largest entry; outputs one
        # rounding (core, then three products) of their type apart
        assert (state.recurrent_state_ - S).abs().max() <= 1e-5 * S.abs().max()
        bound = (2 ** -6 if rounded or code else 2e-5) * want.float().abs() + 2e-5 * want.float().abs().max()
        assert ((out.float() - want.float()).abs() <= bound).all()
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("heads,dim,rotary,cache_dtype,rounded", [
    (*shape, torch.float32, rounded) for shape in (((24, 4), 256, 64), ((5, 1), 128, 128), ((3, 3), 64, 12))
    for rounded in (True, False)] + [((24, 4), 256, 64, torch.bfloat16, False)])
def test_cached_step_is_the_separate_launches_bit_for_bit(heads, dim, rotary, cache_dtype, rounded):
    """The step forms every sum in the order of prepare + decode + merge, so the number of launches does
    not show in the result: keys, values and output, one row to the longest context, at the edges of the
    64-token chunks.  (fp32 output of calls that the decode entry point gives to its plain kernel.)"""
    hq, hkv = heads
    p = FullAttentionParameters(query_heads=hq, key_value_heads=hkv, head_dim=dim, rotary_dim=rotary, capacity=1024,
                                round_to_bfloat16=rounded)
    gen = torch.Generator(device="cuda").manual_seed(dim)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    keys, values, wq, wk = rnd(1024, hkv, dim).bfloat16(), rnd(1024, hkv, dim).bfloat16(), rnd(dim) * 0.1, rnd(dim) * 0.1
    for position in (0, 1, 3, 4, 31, 63, 64, 65, 127, 128, 255, 256, 300, 511, 512, 1023):
        qg, k, v = rnd(hq, 2, dim), rnd(hkv, dim), rnd(hkv, dim)
        caches = [KeyValueCache.Create(1024, hkv, dim, cache_dtype) for _ in range(2)]
        for cache in caches:
            cache.keys().copy_(keys)
            cache.values().copy_(values)
            cache.position_ = position
        out = torch.empty(hq, dim, device="cuda")
        CachedAttentionStep(p, caches[0], qg, k, v, wq, wk, out)
        queries = torch.empty(1, hq, dim, device="cuda", dtype=torch.bfloat16 if rounded else torch.float32)
        at = torch.tensor([position], dtype=torch.int32, device="cuda")
        _capi.check(_capi.fast().pluto_qk_prepare(
            stream(), qg.data_ptr(), k.data_ptr(), v.data_ptr(), 0, 2 * hq * dim, 2 * dim, wq.data_ptr(), wk.data_ptr(),
            at.data_ptr(), queries.data_ptr(), int(rounded), caches[1].packed_layout(), 1, 1, hq, hkv, dim, rotary,
            p.rms_norm_epsilon, p.rope_theta, int(rounded)))
        want = gqa_decode(queries, caches[1].keys()[None], caches[1].values()[None], at + 1, position + 1,
                          gate=qg[None, :, 1], round_to_bfloat16=rounded, out=torch.empty(1, hq, dim, device="cuda"))[0]
        assert torch.equal(caches[0].keys(), caches[1].keys()) and torch.equal(caches[0].values(), caches[1].values())
        assert torch.equal(out, want), position
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("rounded", [True, False])
def test_delta_step_gates_as_the_sequence_kernels_do(rounded):
    """Convolution SiLU and output gate of the one launch and of the four, bit for bit.  One live channel in q
    and in k leaves every sum behind them a single term, so no order of summation can hide a difference."""
    key_heads, value_heads, taps = 2, 6, 4
    p = DeltaNetParameters(key_heads=key_heads, value_heads=value_heads, conv_kernel_dim=taps, round_to_bfloat16=rounded)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    kq, width = key_heads * 128, value_heads * 128
    channels = 2 * kq + width
    conv, a_log, dt_bias, norm = rnd(channels, taps), rnd(value_heads), rnd(value_heads), rnd(128)
    conv[:2 * kq].view(2 * key_heads, 128, taps)[:, 1:] = 0
    state = DeltaNetState.Create(p)
    window, S = torch.zeros(channels, taps, device="cuda"), torch.zeros(1, value_heads, 128, 128, device="cuda")
    L, f32 = _capi.fast(), dict(device="cuda", dtype=torch.float32)
    for _ in range(4):
        qkv, z, a, b = rnd(channels) * 3, rnd(value_heads, 128) * 4, rnd(value_heads), rnd(value_heads)
        out, want = torch.empty(value_heads, 128, **f32), torch.empty(value_heads, 128, **f32)
        state.Step(qkv, z, a, b, conv, a_log, dt_bias, norm, out)
        post, g, beta, core = (torch.empty(n, **f32) for n in (channels, value_heads, value_heads, width))
        flag = int(rounded)
        _capi.check(L.pluto_gdn_conv_silu(stream(), qkv.data_ptr(), conv.data_ptr(), 0, 1, 1, channels, taps, flag,
                                          window.data_ptr(), post.data_ptr(), 0))
        _capi.check(L.pluto_gdn_gates(stream(), a.data_ptr(), b.data_ptr(), a_log.data_ptr(), dt_bias.data_ptr(), 0, 1,
                                      value_heads, flag, g.data_ptr(), beta.data_ptr()))
        _capi.check(L.pluto_gdn_step(stream(), post.data_ptr(), post[kq:].data_ptr(), post[2 * kq:].data_ptr(), 0,
                                     g.data_ptr(), beta.data_ptr(), S.data_ptr(), core.data_ptr(), 0, 1, key_heads,
                                     value_heads, 128, 128, 1, 1.0, flag))
        _capi.check(L.pluto_gdn_out_norm_gate(stream(), core.data_ptr(), 0, z.data_ptr(), 0, norm.data_ptr(), value_heads,
                                              128, p.rms_norm_epsilon, flag, 1, want.data_ptr(), 0))
        assert torch.equal(state.recurrent_state_, S)
        if rounded:
            assert torch.equal(out, want)
        else:   # the mean square of 128 terms, summed in another order: 2^-23 of its root, and three roundings
            assert ((out - want).abs() <= 2 ** -21 * want.abs()).all()


def test_silu_is_one_quotient_over_its_whole_range():
    """x / (1 + e^-x) with an identity convolution, several tokens and one.  expf is good to 2 ulp, the sum and
    the quotient round once each: 3.5 * 2^-23.  The tail below -87 counts (1 + e^-x is finite down to -88.7)."""
    x = torch.cat([torch.linspace(-88.5, 20, 4096), torch.linspace(-3, 3, 4096)]).cuda()
    channels, tokens = 4, 2048
    weight = torch.zeros(channels, 2, device="cuda")
    weight[:, 1] = 1
    for t in (tokens, 1):
        y = torch.empty(x.numel(), device="cuda")
        c = x.numel() // t
        window = torch.zeros(1, c, 2, device="cuda")
        w = weight[:1].expand(c, 2).contiguous()
        _capi.check(_capi.fast().pluto_gdn_conv_silu(stream(), x.data_ptr(), w.data_ptr(), 0, 1, t, c, 2, 0,
                                                     window.data_ptr(), y.data_ptr(), 0))
        want = x.double() / (1 + torch.exp(-x.double()))
        assert ((y.double() - want).abs() <= 3.5 * 2 ** -23 * want.abs()).all()


@pytest.mark.parametrize("dim,rotary", [(256, 64), (64, 4), (64, 12), (128, 20)])
@pytest.mark.parametrize("rounded", [True, False])
def test_an_inspection_hook_leaves_the_cache_as_it_is(dim, rotary, rounded):
    """The probabilities' query is prepared once more, which rewrites the token's cache row: with the same
    bits, whatever rotary width the prepare kernel's accesses fit, and so the outputs behind it stay too."""
    hq, hkv = 4, 2
    p = FullAttentionParameters(query_heads=hq, key_value_heads=hkv, head_dim=dim, rotary_dim=rotary, capacity=16,
                                round_to_bfloat16=rounded)
    results = []
    for hook in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(dim + rotary)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        cache, wq, wk = KeyValueCache.Create(16, hkv, dim, torch.float32), rnd(dim) * 0.1, rnd(dim) * 0.1
        outs = []
        for t in range(12):
            out, probabilities = torch.empty(hq, dim, device="cuda"), torch.empty(hq, t + 1, device="cuda")
            CachedAttentionStep(p, cache, rnd(hq, 2, dim), rnd(hkv, dim), rnd(hkv, dim), wq, wk, out,
                                probabilities if hook else None)
            outs.append(out)
            if hook:   # fp32 sums of at most 12 terms
                assert (probabilities.sum(1) - 1).abs().max().item() < 12 * 2 ** -23
        results.append((cache.keys().clone(), cache.values().clone(), torch.stack(outs)))
    for x, y in zip(*results):
        assert torch.equal(x, y)


@pytest.mark.parametrize("over", ["k", "v"])
def test_attention_output_over_an_input(over):
    """An output that shares memory with k or v: every head still attends with what the caller passed."""
    hq, hkv, dim = 4, 4, 128
    p = FullAttentionParameters(query_heads=hq, key_value_heads=hkv, head_dim=dim, rotary_dim=dim, capacity=8)
    results = []
    for shared in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(3)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        cache, norm = KeyValueCache.Create(8, hkv, dim, torch.float32), torch.zeros(dim, device="cuda")
        qg, k, v = rnd(hq, 2, dim), rnd(hkv, dim), rnd(hkv, dim)
        out = {"k": k, "v": v}[over] if shared else torch.empty(hq, dim, device="cuda")
        CachedAttentionStep(p, cache, qg, k, v, norm, norm, out)
        results.append((out, cache.keys(), cache.values()))
    for x, y in zip(*results):
        assert torch.equal(x, y)


@pytest.mark.parametrize("over", ["qkv", "z"])
def test_delta_output_over_an_input(over):
    p = DeltaNetParameters(key_heads=2, value_heads=6)
    results = []
    for shared in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(3)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
        channels = 4 * 128 + 6 * 128
        conv, a_log, dt_bias, norm = rnd(channels, 4), rnd(6), rnd(6), rnd(128)
        state, qkv, z, a, b = DeltaNetState.Create(p), rnd(channels), rnd(6, 128), rnd(6), rnd(6)
        out = torch.empty(6, 128, device="cuda")
        if shared:
            out = qkv[:6 * 128].view(6, 128) if over == "qkv" else z
        state.Step(qkv, z, a, b, conv, a_log, dt_bias, norm, out)
        results.append((out, state.recurrent_state_))
    (x, s), (y, t) = results
    # one launch against four: fp32 sums of 128 terms in another order, then bf16 roundings of the output
    assert (s - t).abs().max() <= 1e-5 * s.abs().max()
    assert ((x - y).abs() <= 2 ** -6 * x.abs() + 2e-5 * x.abs().max()).all()
