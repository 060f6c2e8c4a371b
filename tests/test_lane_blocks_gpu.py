"""Long lists of rotated K blocks take one lane per block: the bytes and scales of the four-lane kernel on the same rows, at the list length
where the kernels change, for rows that are no multiple of a warp, strides, both types and infinities and NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["group_int8", "group_fp8"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols,pad", [(10657, 2048, 0), (10624, 2048, 32), (10655, 2048, 0), (3553, 6144, 0), (2670, 8192, 16), (170497, 128, 0)])
def test_same_bytes_as_short_lists(ctx_factory, mode, dtype, rows, cols, pad):
    from breeze_tts_cpp_b200 import ops
    ctx, fmt = ctx_factory(mode), ops.format_of(mode)
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols + pad, generator=g, device="cuda").to(dtype)
    for i, value in enumerate((float("inf"), float("nan"), -float("inf"), 0.0, 1e-7, 6e4)):
        x[rows // 7 * (i + 1), (97 * i) % cols] = value
    x[rows - 1] = 0.0
    x = x[:, :cols]
    whole = ctx.quantize_rows(x, ops.RowScaledView.empty(rows, cols, fmt, 128, 128))
    step = 333  # short lists
    for first in [*range(0, rows, max(step, rows // 12)), rows - step]:
        part = ctx.quantize_rows(x[first:first + step], ops.RowScaledView.empty(min(step, rows - first), cols, fmt, 128, 128))
        assert torch.equal(part.values, whole.values[first:first + step])
        assert torch.equal(part.scales.view(torch.int32), whole.scales[:, first:first + step].contiguous().view(torch.int32))
