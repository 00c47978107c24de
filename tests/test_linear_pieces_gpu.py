"""FP8 projections on the weight ring (linear_gemv_stream_e4m3) against float64 over the same quantised
operands: two, four and eight pieces per row, ragged last slabs, one to nine tokens (passes of up to
eight), and the shapes either side of each rule."""
import pytest
import torch

from pluto_b200.layers import FullyConnectedLayer, MatrixStorage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,rows", [
    (256, 2368), (256, 2367), (512, 1187), (1024, 592), (1024, 591), (3072, 2370), (4096, 2371), (5120, 1187),
    (5120, 2371), (8192, 1185), (10240, 1187), (11776, 1186), (12288, 593), (640, 1200), (768, 5121)])
@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 8, 9])
def test_pieces(cols, rows, tokens):
    gen = torch.Generator(device="cuda").manual_seed(cols + rows)
    codes = torch.randn(rows, cols, device="cuda", generator=gen).to(torch.float8_e4m3fn)
    scales = 0.5 + torch.rand((rows + 127) // 128, (cols + 127) // 128, device="cuda", generator=gen)
    x = torch.randn(tokens, cols, device="cuda", generator=gen).bfloat16()
    layer = FullyConnectedLayer.Create(codes.view(torch.uint8), MatrixStorage.kFp8E4M3, cols, rows, scales)
    got = layer.fwd([x]).outputs[0].double()
    groups = x.float().view(tokens, -1, 128)
    step = torch.div(groups.abs().amax(-1, keepdim=True), torch.full((1,), 448.0, device="cuda"))   # (by a scalar: * 1 / 448)
    quantised = ((groups / step.clamp_min(1e-12)).to(torch.float8_e4m3fn).double() * step.double()).view(tokens, cols)
    w = codes.double() * scales.double().repeat_interleave(128, 0)[:rows].repeat_interleave(128, 1)[:, :cols]
    want, size = quantised @ w.T, quantised.abs() @ w.abs().T
    # one rounding to bf16, and sums whose error stays below 2^-16 of the sum of magnitudes
    assert ((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -16 * size).all()
    assert torch.equal(layer.fwd([x]).outputs[0].double(), got)
