"""The CTA-pair prefill kernel around its 256-token tile and its channel tiles (64 to 256 in steps of 64): rows that leave the
second CTA of a pair without any, fewer channels than a tile or a slab, ragged last tiles, one and several tiles per pair, with
and without the finishing chain and its residual, against the weight-streaming kernel on the same operands: identical bits for
INT8 (exact sums, the same finishing arithmetic), FP8 within its tolerance."""
import pytest
import torch

from tests.oracle_binding import FP8, I8

pytestmark = pytest.mark.gpu
TCGEN05 = 5
SHAPES = [(1, 16, 256), (65, 48, 128), (128, 80, 512), (256, 144, 384), (257, 208, 256), (1, 512, 128), (129, 256, 128), (160, 2048, 512), (161, 768, 2048), (192, 4096, 1024), (225, 4112, 384), (301, 12288, 256),
          (750, 4096, 1024), (1021, 2048, 640), (1500, 2048, 512), (2048, 2064, 256)]


def operands(ctx, m, n, k, fmt, seed):
    from breeze_tts_cpp_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    return ctx.quantize_rows(x, ops.RowScaledView.empty(m, k, fmt)), ctx.quantize_rows(w, ops.RowScaledView.empty(n, k, fmt)), g


@pytest.mark.parametrize("mode,fmt", [("int8", I8), ("fp8", FP8)])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("dtype,chain", [(torch.bfloat16, None), (torch.float16, None), (torch.bfloat16, 0), (torch.float16, 4),
                                         (torch.bfloat16, 5), (torch.float16, 3), (torch.bfloat16, "bias"),
                                         (torch.float16, "residual_f32")])
def test_pair_kernel_matches_weight_streaming_kernel(ctx_factory, mode, fmt, m, n, k, dtype, chain):
    ctx = ctx_factory(mode)
    xv, wv, g = operands(ctx, m, n, k, fmt, m + n + k)
    kw = {}
    if chain == "bias":
        kw = dict(bias=torch.randn(1, n, generator=g, device="cuda").to(dtype))
    elif chain == "residual_f32":
        kw = dict(residual_f32=torch.randn(m, n, generator=g, device="cuda"))
    elif chain is not None:
        kw = dict(bias=torch.randn(1, n, generator=g, device="cuda").to(dtype), activation=chain, value_scale=0.7,
                  residual=torch.randn(m, n, generator=g, device="cuda").to(dtype), residual_scale=1.3, output_scale=0.9)
    out, other = (torch.full((m, n), float("nan"), dtype=dtype, device="cuda") for _ in range(2))
    ctx.quant_linear((TCGEN05, 256, 128, 1), xv, wv, out, **kw)
    ctx.quant_linear((TCGEN05, 64, 128, 1), xv, wv, other, **kw)
    assert ctx.status() == 0
    if fmt == I8:
        assert torch.equal(out.view(torch.int16), other.view(torch.int16))
    else:
        assert float((out.double() - other.double()).norm() / other.double().norm()) < 2e-3
