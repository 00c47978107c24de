"""Decode in its two forms (parts of a cluster; chunks + merge kernel) and at all three head widths
against float64, with lengths at the edges of the tiles (64 tokens, at width 256 32) and of the parts: one
token, fewer tokens than parts, and part boundaries.  Unrounded fp32 results run on the tensor cores at
widths 64 and 128 and on the plain kernel at 256, whose tensor-core form has a test of its own."""
import math

import pytest
import torch

from pluto_b200 import _capi
from pluto_b200.layers import gqa_decode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,hq,hkv,dim,longest", [
    # 256 MB of cache at most: one launch, 1 to 16 parts; more: chunks and the merge kernel
    (1, 24, 4, 256, 1), (5, 24, 4, 256, 130), (2, 24, 4, 256, 4096), (40, 8, 4, 256, 300), (17, 24, 4, 256, 4000),
    (1, 40, 8, 128, 64), (4, 40, 8, 128, 65), (7, 5, 1, 128, 2000), (40, 8, 8, 128, 500), (9, 40, 8, 128, 8200),
    (1, 12, 12, 64, 63), (30, 12, 12, 64, 129), (6, 12, 12, 64, 1025), (1, 16, 1, 64, 8200), (12, 12, 12, 64, 8200)])
@pytest.mark.parametrize("page", [0, 16, 64])
def test_decode_matches_float64(batch, hq, hkv, dim, longest, page):
    gen = torch.Generator(device="cuda").manual_seed(longest + dim)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    capacity = (longest + 63) // 64 * 64
    k, v = rnd(batch, capacity, hkv, dim).bfloat16(), rnd(batch, capacity, hkv, dim).bfloat16()
    q, gate = rnd(batch, hq, dim).bfloat16(), rnd(batch, hq, dim).bfloat16()
    lens = torch.randint(1, longest + 1, (batch,), device="cuda", generator=gen, dtype=torch.int32)
    lens[0] = longest
    edges = [x for x in (1, 63, 64, 65, longest // 2, longest - 1) if 1 <= x <= longest]
    for i, x in enumerate(edges[:batch - 1]):
        lens[1 + i] = x
    # rows past a sequence's end must not matter, whatever they hold
    dead = torch.arange(capacity, device="cuda")[None, :] >= lens[:, None]
    k[dead] = float("nan")
    v[dead] = float("inf")
    group = hq // hkv
    kk = k.double().repeat_interleave(group, 2).masked_fill(dead[:, :, None, None], 0)
    vv = v.double().repeat_interleave(group, 2).masked_fill(dead[:, :, None, None], 0)
    s = torch.einsum("bhd,bthd->bht", q.double(), kk) / math.sqrt(dim)
    s = s.masked_fill(dead[:, None, :], -math.inf)
    want = torch.einsum("bht,bthd->bhd", torch.softmax(s, -1), vv)
    table, pool_k, pool_v = None, k, v
    if page:
        blocks = capacity // page
        table = torch.randperm(batch * blocks, device="cuda", generator=gen).to(torch.int32).view(batch, blocks)
        pool_k, pool_v = (torch.empty(batch * blocks, page, hkv, dim, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        pool_k[table.reshape(-1).long()] = k.view(-1, page, hkv, dim)
        pool_v[table.reshape(-1).long()] = v.view(-1, page, hkv, dim)
    out = torch.empty(batch, hq, dim, device="cuda")
    got, lse = gqa_decode(q, pool_k, pool_v, lens, longest, block_table=table, round_to_bfloat16=False, out=out, want_lse=True)
    # P carries 2^-17 relative error into a weighted mean of N(0, 1) values; fp32 sums of up to 8200 terms
    assert (got.double() - want).abs().max().item() < 4e-5
    assert (lse.double() - torch.logsumexp(s, -1)).abs().max().item() < 2e-5
    gated = gqa_decode(q, pool_k, pool_v, lens, longest, block_table=table, gate=gate)
    expected = want.bfloat16().double() * torch.sigmoid(gate.double()).bfloat16().double()
    # the core and the product can each fall on either side of a tie: one bf16 ulp (at most 2^-7) apiece
    assert ((gated.double() - expected).abs() <= 2 ** -6 * expected.abs() + 4e-5).all()
    assert torch.equal(gated, gqa_decode(q, pool_k, pool_v, lens, longest, block_table=table, gate=gate))
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("rounded", [True, False])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_width_256_keeps_fp32_queries(rounded, out_dtype):
    """fp32 queries that bf16 cannot hold are attended with as given: the log of the softmax sum is an fp32
    result of the scores, and a query rounded to bf16 moves it by 1e-3 and more."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    k, v, q = rnd(2, 200, 2, 256).bfloat16(), rnd(2, 200, 2, 256).bfloat16(), rnd(2, 6, 256)
    lens = torch.tensor([200, 77], dtype=torch.int32, device="cuda")
    _, lse = gqa_decode(q, k, v, lens, 200, round_to_bfloat16=rounded, out=torch.empty(2, 6, 256, device="cuda", dtype=out_dtype),
                        want_lse=True)
    for b, n in enumerate(lens.tolist()):
        s = torch.einsum("hd,thd->ht", q[b].double(), k[b, :n].double().repeat_interleave(3, 1)) / 16
        assert (lse[b].double() - torch.logsumexp(s, -1)).abs().max().item() < 5e-6   # fp32 sums of 256 products


# One, two and a dozen units (sequence x KV head), either side of the lines between the two forms: long
# parts go to chunks, and 12, 20, 32, 64 and 148 units are the most that are cut into 16, 12, 8, 4 and 2 parts.
@pytest.mark.parametrize("batch,hq,hkv,dim,longest", [
    (1, 5, 1, 128, 14400), (1, 5, 1, 128, 14500), (2, 1, 1, 64, 33000), (1, 6, 1, 256, 6400), (1, 6, 1, 256, 6401),
    (2, 6, 1, 256, 20000), (12, 1, 1, 64, 700), (13, 1, 1, 64, 380), (20, 2, 1, 128, 500), (21, 2, 1, 128, 500), (32, 2, 1, 128, 300), (33, 2, 1, 128, 300),
    (64, 1, 1, 64, 200), (65, 1, 1, 64, 200), (149, 1, 1, 64, 100)])
def test_few_units_and_the_lines_between_the_forms(batch, hq, hkv, dim, longest):
    test_decode_matches_float64(batch, hq, hkv, dim, longest, 0)


@pytest.mark.parametrize("batch,hq,hkv,longest", [
    (1, 6, 1, 1), (1, 24, 4, 33), (5, 24, 4, 130), (2, 24, 4, 3000), (40, 8, 4, 300),        # one launch
    (1, 6, 1, 9000), (3, 24, 4, 6500), (17, 24, 4, 4000)])                                   # chunks and the merge
@pytest.mark.parametrize("page", [0, 16, 64])
def test_width_256_on_the_tensor_cores(batch, hq, hkv, longest, page):
    """bf16 queries, rounded result in fp32: the log of the softmax sum and the ungated output.  The core is
    good to a few 2^-24 of values of order one, so its rounding to bf16 is the nearest value or, within 2e-6
    of a tie, the other neighbour; P in two parts instead of three would leave 1e-5."""
    gen = torch.Generator(device="cuda").manual_seed(longest)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    capacity = (longest + 63) // 64 * 64
    k, v, q = rnd(batch, capacity, hkv, 256).bfloat16(), rnd(batch, capacity, hkv, 256).bfloat16(), rnd(batch, hq, 256).bfloat16()
    lens = torch.randint(1, longest + 1, (batch,), device="cuda", generator=gen, dtype=torch.int32)
    lens[0] = longest
    for i, x in enumerate([x for x in (31, 32, 33, longest - 1) if 1 <= x <= longest][:batch - 1]):
        lens[1 + i] = x
    table, pool_k, pool_v = None, k, v
    if page:
        blocks = capacity // page
        table = torch.randperm(batch * blocks, device="cuda", generator=gen).to(torch.int32).view(batch, blocks)
        pool_k, pool_v = (torch.empty(batch * blocks, page, hkv, 256, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        pool_k[table.reshape(-1).long()] = k.view(-1, page, hkv, 256)
        pool_v[table.reshape(-1).long()] = v.view(-1, page, hkv, 256)
    got, lse = gqa_decode(q, pool_k, pool_v, lens, longest, block_table=table, out=torch.empty(batch, hq, 256, device="cuda"),
                          want_lse=True)
    for b, n in enumerate(lens.tolist()):
        kk, vv = (x[b, :n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        s = torch.einsum("hd,thd->ht", q[b].double(), kk) / 16
        want = torch.einsum("ht,thd->hd", torch.softmax(s, -1), vv)
        assert (lse[b].double() - torch.logsumexp(s, -1)).abs().max().item() < 5e-6
        half_ulp = 2.0 ** (torch.floor(torch.log2(want.abs().clamp(min=1e-30))) - 8)
        assert ((got[b].double() - want).abs() <= half_ulp + 2e-6).all()
        assert torch.equal(got[b], got[b].bfloat16().float())
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("dim,hq,hkv", [(64, 12, 12), (128, 10, 2)])
@pytest.mark.parametrize("batch,capacity", [(3, 1), (5, 182), (2, 1455), (1, 20003)])
def test_contiguous_caches_off_16_tokens_keep_24_bits(dim, hq, hkv, batch, capacity):
    """Without a block table the cache may have any length.  Where 16 does not divide it, P keeps 24 bits: the
    rounded result is the nearest bf16 value or, within 2e-6 of a tie, the other neighbour (two bf16 parts
    leave 1e-5); an unrounded fp32 result and fp32 queries run in fp32 throughout."""
    gen = torch.Generator(device="cuda").manual_seed(capacity)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    k, v = rnd(batch, capacity, hkv, dim).bfloat16(), rnd(batch, capacity, hkv, dim).bfloat16()
    lens = torch.randint(1, capacity + 1, (batch,), device="cuda", generator=gen, dtype=torch.int32)
    lens[0] = capacity
    for q in (rnd(batch, hq, dim).bfloat16(), rnd(batch, hq, dim)):
        new = lambda: torch.empty(batch, hq, dim, device="cuda")
        rounded, lse = gqa_decode(q, k, v, lens, capacity, out=new(), want_lse=True)
        plain = gqa_decode(q, k, v, lens, capacity, round_to_bfloat16=False, out=new())
        for b, n in enumerate(lens.tolist()):
            kk, vv = (x[b, :n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
            s = torch.einsum("hd,thd->ht", q[b].double(), kk) / math.sqrt(dim)
            want = torch.einsum("ht,thd->hd", torch.softmax(s, -1), vv)
            assert (plain[b].double() - want).abs().max().item() < 3e-6
            assert (lse[b].double() - torch.logsumexp(s, -1)).abs().max().item() < 5e-6
            half_ulp = 2.0 ** (torch.floor(torch.log2(want.abs().clamp(min=1e-30))) - 8)
            assert ((rounded[b].double() - want).abs() <= half_ulp + 2e-6).all()
    assert _capi.kernel_status() == 0
