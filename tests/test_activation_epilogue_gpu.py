"""SiLU and sigmoid in the GEMM's own epilogue over every value of the storage type, against the finishing pass: identical bits
(any NaN for a NaN)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["int8", "group_fp8"])
@pytest.mark.parametrize("m,tokens", [(32, 0), (512, 0), (512, 256)])  # as planned: streaming tiles; 256 or 128: the persistent kernels
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("activation", [3, 8])
def test_activation_of_every_value(ctx_factory, mode, m, tokens, dtype, activation):
    from breeze_tts_cpp_b200 import ops
    ctx, n, k = ctx_factory(mode), 65536 // m, 128
    group, _, rotation = ops.groups_of(mode)
    every = torch.arange(65536, device="cuda").to(torch.int16).view(dtype).view(m, n)
    zeros = lambda *shape: torch.zeros(*shape, dtype=dtype, device="cuda")
    w = ctx.quantize_rows(zeros(n, k), ops.RowScaledView.empty(n, k, ops.format_of(mode), group, rotation))
    scratch = ops.RowScaledView.empty(m, k, ops.format_of(mode), group, rotation)
    ctx.prepare_quantized(m, n, k, out_dtype=dtype)
    fused, two = torch.empty(m, n, dtype=dtype, device="cuda"), torch.empty(m, n, dtype=dtype, device="cuda")
    if tokens:
        path = (5, 128 if group else tokens, 128, 1)
        ctx.quant_linear(path, ctx.quantize_rows(zeros(m, k), scratch), w, fused, residual=every, activation=activation)
    else:
        ctx.linear(zeros(m, k), w, scratch, fused, residual=every, activation=activation)
    ctx.pointwise(zeros(m, n), two, residual=every, activation=activation)
    assert ctx.status() == 0
    assert bool(((fused.view(torch.int16) == two.view(torch.int16)) | (fused.isnan() & two.isnan())).all())
