"""The streaming kernels around the delta-net recurrence (gdn.cu, gdn_bwd.cu) against float64, where
their tiles end: 16-token segments of the convolution, 32 token ranges of its backward, 128-channel
groups and strips of rows of the output norm, and the calls their wide accesses do not fit."""
import pytest
import torch

from pluto_b200 import _capi

pytestmark = pytest.mark.gpu
F32, BF16 = 0, 1


def stream():
    return torch.cuda.current_stream().cuda_stream


def code(t):
    return BF16 if t.dtype == torch.bfloat16 else F32


def rand(seed, *shape):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def causal(x, w, history):
    """[b, t, c] in float64: sum over the taps, the history first."""
    width = w.shape[1]
    long = torch.cat([history.transpose(1, 2), x], 1)   # `width` old inputs, then the new ones
    return sum(long[:, 1 + tap:1 + tap + x.shape[1]] * w[:, tap] for tap in range(width))


@pytest.mark.parametrize("width", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("tokens", [1, 2, 15, 16, 17, 50])
@pytest.mark.parametrize("channels,shift", [(36, 0), (516, 0), (35, 0), (36, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_convolution(width, tokens, channels, shift, dtype):
    """Unrounded, with a history, apart and in place; `shift` elements off the 16-byte boundary."""
    batch = 2
    x = rand(1, batch, tokens, channels).to(dtype)
    w, history = rand(2, channels, width), rand(3, batch, channels, width)
    s = causal(x.double(), w.double(), history.double())
    want = s * torch.sigmoid(s)
    store = torch.empty(x.numel() + shift, device="cuda", dtype=dtype)[shift:]
    store.copy_(x.flatten())
    new_state = torch.cat([history.transpose(1, 2), x.float()], 1)[:, -width:].transpose(1, 2)
    for in_place in (False, True):
        state = history.clone()
        out = store if in_place else torch.empty_like(store)
        _capi.check(_capi.fast().pluto_gdn_conv_silu(stream(), store.data_ptr(), w.data_ptr(), code(x), batch, tokens,
                                                     channels, width, 0, state.data_ptr(), out.data_ptr(), code(x)))
        got = out.view_as(x).double()
        # five fp32 products and sums of N(0, 1) pairs and a SiLU (slope <= 1.1): 1e-5; stored in bf16, half an ulp
        assert ((got - want).abs() <= 1e-5 + (2 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)).all(), in_place
        assert torch.equal(state, new_state)


@pytest.mark.parametrize("width", [1, 3, 4, 5])
@pytest.mark.parametrize("tokens", [1, 2, 31, 32, 33, 100])
@pytest.mark.parametrize("channels", [34, 35, 130])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_convolution_backward(width, tokens, channels, dtype):
    batch = 2
    x, w, up = rand(1, batch, tokens, channels).to(dtype), rand(2, channels, width), rand(3, batch, tokens, channels)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    s = causal(xd, wd, torch.zeros(batch, channels, width, device="cuda", dtype=torch.float64))
    want_dx, want_dw = torch.autograd.grad((s * torch.sigmoid(s) * up.double()).sum(), (xd, wd))
    dx, dw = torch.empty_like(up), torch.ones_like(w)
    _capi.check(_capi.fast().pluto_gdn_conv_silu_bwd(stream(), x.data_ptr(), code(x), w.data_ptr(), up.data_ptr(),
                                                     dx.data_ptr(), dw.data_ptr(), batch, tokens, channels, width, 0))
    # dx: five products of values up to 4; dw: a sum of 200 such in fp32, 2^-24 * sqrt(200) * 4 * 10
    assert (dx.double() - want_dx).abs().max().item() < 2e-5
    assert (dw.double() - 1 - want_dw).abs().max().item() < 5e-5


@pytest.mark.parametrize("dim", [1, 4, 100, 128, 130, 132, 256])
@pytest.mark.parametrize("rows", [1, 8, 9, 5000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_output_norm_and_its_backward(dim, rows, dtype):
    core, z, norm, dy = rand(1, rows, dim).to(dtype), rand(2, rows, dim).to(dtype), 1 + 0.1 * rand(3, dim), rand(4, rows, dim)
    cd, zd, nd = (t.double().requires_grad_() for t in (core, z, norm))
    want = cd * (cd.square().mean(-1, keepdim=True) + 1e-2).rsqrt() * nd * zd * torch.sigmoid(zd)
    grads = torch.autograd.grad((want * dy.double()).sum(), (cd, zd, nd))
    L = _capi.fast()
    out = torch.empty(rows, dim, device="cuda")
    _capi.check(L.pluto_gdn_out_norm_gate(stream(), core.data_ptr(), code(core), z.data_ptr(), code(z), norm.data_ptr(),
                                          rows, dim, 1e-2, 0, 0, out.data_ptr(), F32))
    # a handful of fp32 products of values up to 5 x 5, rsqrtf good to two ulps
    assert (out.double() - want).abs().max().item() < 2e-5
    dcore, dz, dnorm = torch.empty(rows, dim, device="cuda"), torch.empty(rows, dim, device="cuda"), torch.ones(dim, device="cuda")
    size = L.pluto_gdn_out_norm_gate_bwd_workspace_bytes(rows, dim)
    ws = torch.empty(size, device="cuda", dtype=torch.uint8)
    _capi.check(L.pluto_gdn_out_norm_gate_bwd(stream(), core.data_ptr(), code(core), z.data_ptr(), code(z), norm.data_ptr(),
                                              dy.data_ptr(), dcore.data_ptr(), dz.data_ptr(), dnorm.data_ptr(),
                                              ws.data_ptr(), size, rows, dim, 1e-2, 0))
    # 1 / rms is at most 10 at width 1, where a gradient is a difference of terms up to 10 * 25: 250 * 2^-23
    assert (dcore.double() - grads[0]).abs().max().item() < (3e-4 if dim == 1 else 5e-5)
    assert (dz.double() - grads[1]).abs().max().item() < 5e-5
    # up to 5000 products of order one summed in fp32, in runs of at most a few dozen
    assert (dnorm.double() - 1 - grads[2]).abs().max().item() < 1e-5 * rows ** 0.5 + 1e-5


@pytest.mark.parametrize("dim", [128, 256, 66])
@pytest.mark.parametrize("over", ["core", "z"])
def test_output_norm_in_place(dim, over):
    rows = 77
    core, z, weight = rand(1, rows, dim), rand(2, rows, dim), rand(3, dim)
    run = lambda c, g, out: _capi.check(_capi.fast().pluto_gdn_out_norm_gate(
        stream(), c.data_ptr(), F32, g.data_ptr(), F32, weight.data_ptr(), rows, dim, 1e-6, 1, 0, out.data_ptr(), F32))
    want = torch.empty_like(core)
    run(core, z, want)
    got = (core if over == "core" else z).clone()
    run(got if over == "core" else core, got if over == "z" else z, got)
    assert torch.equal(got, want)


@pytest.mark.parametrize("dim", [128, 256, 66])
@pytest.mark.parametrize("which", ["dcore", "dz"])
def test_output_norm_backward_over_its_upstream(dim, which):
    rows = 1203
    core, z, weight, dy = rand(1, rows, dim), rand(2, rows, dim), rand(3, dim), rand(4, rows, dim)
    size = _capi.fast().pluto_gdn_out_norm_gate_bwd_workspace_bytes(rows, dim)
    results = []
    for shared in (False, True):
        upstream, dw = dy.clone(), torch.zeros(dim, device="cuda")
        grads = {name: torch.empty_like(dy) for name in ("dcore", "dz")}
        if shared:
            grads[which] = upstream
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        _capi.check(_capi.fast().pluto_gdn_out_norm_gate_bwd(
            stream(), core.data_ptr(), F32, z.data_ptr(), F32, weight.data_ptr(), upstream.data_ptr(), grads["dcore"].data_ptr(),
            grads["dz"].data_ptr(), dw.data_ptr(), ws.data_ptr(), size, rows, dim, 1e-6, 1))
        results.append((grads["dcore"], grads["dz"], dw))
    for x, y in zip(*results):
        assert torch.equal(x, y)


@pytest.mark.parametrize("heads,dim,rotary", [(24, 256, 64), (3, 128, 128), (1, 66, 12)])
def test_norm_backward_over_its_upstream(heads, dim, rotary):
    tokens = 45
    x, weight, grad = rand(1, tokens, heads, dim).bfloat16(), rand(2, dim) * 0.1, rand(3, tokens, heads, dim)
    size = _capi.fast().pluto_qk_prepare_bwd_workspace_bytes(1, tokens, heads, dim)
    results = []
    for shared in (False, True):
        upstream, dw = grad.clone(), torch.zeros(dim, device="cuda")
        dx, ws = upstream if shared else torch.empty_like(grad), torch.empty(size, dtype=torch.uint8, device="cuda")
        _capi.check(_capi.fast().pluto_qk_prepare_bwd(
            stream(), x.data_ptr(), heads * dim, dim, weight.data_ptr(), upstream.data_ptr(), None, dx.data_ptr(), heads * dim,
            dim, dw.data_ptr(), ws.data_ptr(), size, 1, tokens, heads, dim, rotary, 1e-6, 1e7, 1))
        results.append((dx, dw))
    for x, y in zip(*results):
        assert torch.equal(x, y)
