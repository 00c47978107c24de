"""Dense and block-linear products that are cut along K (few tiles, long K), ragged and with the least
workspace, against float64 over the same 2-byte operands."""
import pytest
import torch

from pluto_b200 import _capi

pytestmark = pytest.mark.gpu


def rand(seed, *shape):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def close(got, want, size, name):
    # products are exact and accumulate in fp32 in the tensor core and over the parts: 2^-18 of the sum
    # of magnitudes leaves room for truncation over 128 K steps
    assert ((got.double() - want).abs() <= 2 ** -18 * size + 1e-12).all(), name


# the forward is cut at (64, 4096, 260), dX at (100, 260, 4096), dW at 4096 rows; 259 columns are never cut
@pytest.mark.parametrize("rows,width,out", [(64, 4096, 260), (100, 260, 4096), (4096, 136, 520), (4100, 136, 259),
                                            (1, 2048, 4), (129, 640, 384), (8192, 768, 256)])
@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("least", [False, True])
def test_dense(rows, width, out, bf16, least):
    dtype = torch.bfloat16 if bf16 else torch.float16
    x, w, bias, dy = rand(1, rows, width), rand(2, width, out) * 0.05, rand(3, out), rand(4, rows, out)
    xin = x.bfloat16() if bf16 else x
    L, stream = _capi.fast(), torch.cuda.current_stream().cuda_stream
    r, i, o = ((v + 127) // 128 * 128 for v in (rows, width, out))
    size = 2 * (r * i + i * o + r * o) + 4 * 16 * o if least else L.pluto_dense_workspace_bytes(rows, width, out)
    ws = torch.empty(size + 4096, dtype=torch.uint8, device="cuda").fill_(0xff)
    assert ws.data_ptr() % 256 == 0
    y = torch.empty(rows, out, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
    _capi.check(L.pluto_dense_fwd(stream, xin.data_ptr(), int(bf16), w.data_ptr(), bias.data_ptr(), y.data_ptr(), rows,
                                  width, out, ws.data_ptr(), size))
    xd, wd, gd = (t.to(dtype).double() for t in (xin, w, dy))
    want, magnitude = xd @ wd + bias.double(), xd.abs() @ wd.abs() + bias.double().abs()
    if bf16:   # and half an ulp of the stored bf16
        assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -18 * magnitude).all()
    else:
        close(y, want, magnitude, "y")
    dx, dw, db = (torch.empty(s, device="cuda") for s in ((rows, width), (width, out), (out,)))
    _capi.check(L.pluto_dense_bwd(stream, xin.data_ptr(), int(bf16), w.data_ptr(), dy.data_ptr(), dx.data_ptr(),
                                  dw.data_ptr(), db.data_ptr(), rows, width, out, ws.data_ptr(), size))
    close(dx, gd @ wd.T, gd.abs() @ wd.abs().T, "dx")
    close(dw, xd.T @ gd, xd.abs().T @ gd.abs(), "dw")
    close(db, dy.double().sum(0), dy.double().abs().sum(0), "db")
    assert (ws[size:] == 0xff).all()
    assert _capi.kernel_status() == 0


@pytest.mark.parametrize("tokens,width,out", [(64, 4096, 260), (100, 260, 2048), (2048, 136, 520), (7, 384, 384)])
def test_block_linear(tokens, width, out):
    x, w, dy = rand(1, tokens, width).bfloat16(), rand(2, out, width).bfloat16(), rand(3, tokens, out)
    L, stream = _capi.fast(), torch.cuda.current_stream().cuda_stream
    size = L.pluto_block_linear_workspace_bytes(tokens, width, out)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda").fill_(0xff)
    y, dx, dw = (torch.empty(s, device="cuda") for s in ((tokens, out), (tokens, width), (out, width)))
    _capi.check(L.pluto_block_linear_fwd(stream, w.data_ptr(), x.data_ptr(), y.data_ptr(), 0, tokens, width, out,
                                         ws.data_ptr(), size))
    dw.fill_(2.0)   # the gradient accumulates
    _capi.check(L.pluto_block_linear_bwd(stream, w.data_ptr(), x.data_ptr(), dy.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                         tokens, width, out, ws.data_ptr(), size))
    xd, wd, gd = x.double(), w.double(), dy.double()
    close(y, xd @ wd.T, xd.abs() @ wd.abs().T, "y")
    # dY enters as two bf16 parts: 2^-17 of every term, and the accumulation as above
    for got, want, magnitude in ((dx, gd @ wd, gd.abs() @ wd.abs()), (dw - 2, gd.T @ xd, gd.abs().T @ xd.abs())):
        assert ((got.double() - want).abs() <= 2 ** -16 * magnitude + 1e-6).all()
    assert _capi.kernel_status() == 0
