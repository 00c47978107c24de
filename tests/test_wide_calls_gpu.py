"""Calls of head width 256 that the tensor-core kernels do not take, and caches whose buffers are replaced."""
import math

import pytest
import torch

from pluto_b200 import _capi
from pluto_b200.layers import (CachedAttentionStep, FullAttentionParameters, KeyValueCache, QwenAttentionLayer, gqa_decode,
                               gqa_prefill)

pytestmark = pytest.mark.gpu
D = 256


def rand(seed, *shape):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("workspace,shift", [("none", 0), ("small", 0), ("full", 1)])
def test_backward_without_the_tensor_cores(workspace, shift):
    """A workspace that is too small, and gradients one float off the 16-byte boundary, take the exact kernels."""
    b, t, hq, hkv = 1, 70, 4, 2
    q, k, v, d_out = (rand(i, b, t, h, D) for i, h in enumerate((hq, hkv, hkv, hq)))
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    stats = gqa_prefill(q, k, v, want_core=True, want_stats=True)
    deltas = (d_out * stats["core"]).sum(-1).permute(0, 2, 1).contiguous()
    size = _capi.lib().pluto_gqa_prefill_bwd_workspace_bytes(b, t, hq, D, 1)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    given = {"none": 0, "small": 256, "full": size}[workspace]
    results = []
    for offset, pointer, n in ((0, None, 0), (shift, ws.data_ptr() if given else None, given)):
        grads = [torch.zeros(x.numel() + offset, device="cuda")[offset:] for x in (q, k, v)]
        _capi.check(_capi.lib().pluto_gqa_prefill_bwd(
            torch.cuda.current_stream().cuda_stream, q.data_ptr(), k.data_ptr(), v.data_ptr(), 1, hq * D, D,
            d_out.data_ptr(), stats["maxima"].data_ptr(), stats["normalizers"].data_ptr(), deltas.data_ptr(),
            *(g.data_ptr() for g in grads), pointer, n, b, t, hq, hkv, D))
        results.append(grads)
    for x, y in zip(*results):
        assert torch.equal(x, y)


def test_packed_backward_with_a_small_workspace():
    b, t, h = 1, 40, 2
    qkv = rand(1, b * t, 3 * h * D).bfloat16()
    out, m, l = torch.empty(b * t, h * D, device="cuda", dtype=torch.bfloat16), *(torch.empty(b * h * t, device="cuda") for _ in range(2))
    L, stream = _capi.lib(), torch.cuda.current_stream().cuda_stream
    _capi.check(L.pluto_attn_fwd(stream, qkv.data_ptr(), out.data_ptr(), m.data_ptr(), l.data_ptr(), b, t, h, D, 1))
    d_out, ws, results = rand(2, b * t, h * D), torch.empty(1024, dtype=torch.uint8, device="cuda"), []
    for pointer, n in ((None, 0), (ws.data_ptr(), 1024)):
        d_qkv, deltas = torch.empty(b * t, 3 * h * D, device="cuda"), torch.empty(b * h * t, device="cuda")
        code = L.pluto_attn_bwd(stream, qkv.data_ptr(), out.data_ptr(), d_out.data_ptr(), m.data_ptr(), l.data_ptr(),
                                d_qkv.data_ptr(), deltas.data_ptr(), b, t, h, D, 1, pointer, n)
        _capi.check(code)
        results.append(d_qkv)
    assert torch.equal(*results)


@pytest.mark.parametrize("longest", [1, 100, 3000])
def test_unrounded_decode_keeps_fp32(longest):
    q, k, v = rand(1, 2, 6, D).bfloat16(), rand(2, 2, longest, 2, D).bfloat16(), rand(3, 2, longest, 2, D).bfloat16()
    lens = torch.tensor([longest, max(1, longest // 2)], dtype=torch.int32, device="cuda")
    got = gqa_decode(q, k, v, lens, longest, round_to_bfloat16=False, out=torch.empty(2, 6, D, device="cuda"))
    for b, n in enumerate(lens.tolist()):
        kk, vv = (x[b, :n].double().repeat_interleave(3, 1) for x in (k, v))
        want = torch.einsum("hk,khd->hd", torch.softmax(torch.einsum("hd,khd->hk", q[b].double(), kk) / math.sqrt(D), -1), vv)
        # fp32 throughout: sums of up to 3000 terms of order 1 / n, a few ulps
        assert (got[b].double() - want).abs().max().item() < 3e-6


def test_cache_buffers_may_be_replaced():
    p = FullAttentionParameters(query_heads=2, key_value_heads=1, head_dim=64, rotary_dim=32, capacity=8)
    cache, norm = KeyValueCache.Create(8, 1, 64), torch.zeros(64, device="cuda")
    step = lambda i: CachedAttentionStep(p, cache, rand(i, 2, 2, 64).bfloat16(), rand(i, 1, 64).bfloat16(),
                                         rand(i, 1, 64).bfloat16(), norm, norm, out)
    out = torch.empty(2, 64, device="cuda", dtype=torch.bfloat16)
    step(1)
    old = cache.keys_
    cache.keys_, cache.values_ = old.clone(), cache.values_.clone()
    step(2)
    assert old[1].abs().sum().item() == 0 and cache.keys_[1].abs().sum().item() > 0


@pytest.mark.parametrize("change", ["cache heads", "cache capacity", "parameters"])
def test_a_layer_whose_cache_no_longer_fits_is_refused(change):
    make = lambda **k: FullAttentionParameters(**{**dict(query_heads=2, key_value_heads=1, head_dim=64, rotary_dim=32, capacity=8), **k})
    norm = torch.zeros(64, device="cuda")
    layer = QwenAttentionLayer.Create(make(), norm, norm, 1, KeyValueCache.Create(8, 1, 64))
    token = [rand(1, 1, 256).bfloat16(), rand(2, 1, 64).bfloat16(), rand(3, 1, 64).bfloat16()]
    layer.fwd(token)
    if change == "cache heads":
        layer.cache_ = KeyValueCache.Create(8, 2, 64)
    elif change == "cache capacity":
        layer.cache_ = KeyValueCache.Create(16, 1, 64)
    else:
        layer.parameters_ = make(capacity=4)
    with pytest.raises(_capi.PlutoStatusError, match="does not match parameters"):
        layer.fwd(token)


@pytest.mark.parametrize("dim", [64, 128, 256])
def test_cache_buffers_off_the_16_byte_boundary(dim):
    """One element further on, the one-launch step does not apply, and the same call takes the separate launches."""
    p = FullAttentionParameters(query_heads=4, key_value_heads=2, head_dim=dim, rotary_dim=32, capacity=8)
    norm, outs = torch.zeros(dim, device="cuda"), []
    for shift in (0, 1):
        cache = KeyValueCache.Create(8, 2, dim)
        cache.keys_, cache.values_ = (torch.zeros(x.numel() + 8, device="cuda", dtype=x.dtype)[shift:shift + x.numel()].view_as(x)
                                      for x in (cache.keys_, cache.values_))
        out = torch.empty(4, dim, device="cuda", dtype=torch.bfloat16)
        for i in range(3):
            CachedAttentionStep(p, cache, rand(i, 4, 2, dim).bfloat16(), rand(i + 9, 2, dim).bfloat16(),
                                rand(i + 99, 2, dim).bfloat16(), norm, norm, out)
        outs.append((out.float(), cache.keys_.clone()))
    assert torch.equal(outs[0][1], outs[1][1])
    # the core and its product with the gate can each fall on either side of a tie: one bf16 ulp apiece
    assert ((outs[0][0] - outs[1][0]).abs() <= 2 ** -6 * outs[1][0].abs() + 1e-6).all()
