"""Aligned rows take packed 16-bit kernels, all others the general ones. Both see the same values here (the general kernels because
every operand starts two bytes off), with infinities, NaN, signed zeros and subnormals among them: every output has the same bits,
over every combination of operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
MODES = ["int8", "fp8", "group_int8", "group_fp8"]


def off_alignment(t):
    """The same values, dense rows, two bytes past an aligned address."""
    if t is None:
        return None
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


class Source:
    def __init__(self, seed, dtype):
        self.g, self.dtype = torch.Generator(device="cuda").manual_seed(seed), dtype

    def rows(self, rows, cols, std=1.0, mean=0.0, special=False):
        x = torch.randn(rows, cols, generator=self.g, device="cuda") * std + mean
        if special:  # two rows with values that are not ordinary numbers, one of tiny ones
            x[0, :cols // 2] *= -0.0
            x[rows // 2] *= 1e-39 if self.dtype == torch.bfloat16 else 1e-6
            x[rows - 1, 3], x[rows - 1, cols - 2] = float("inf"), float("nan")
        return x.to(self.dtype)


def same_bits(a, b):
    if a.dtype == torch.float32:
        return torch.equal(a.view(torch.int32), b.view(torch.int32))
    return torch.equal(a.view(torch.int16 if a.dtype.itemsize == 2 else torch.uint8), b.view(torch.int16 if b.dtype.itemsize == 2 else torch.uint8))


def view(ops, ctx_mode, rows, cols):
    group, _, rotation = ops.groups_of(ctx_mode)
    return ops.RowScaledView.empty(rows, cols, ops.format_of(ctx_mode), group, rotation)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(5, 128), (700, 384), (40, 1024), (12, 2048)])
@pytest.mark.parametrize("operands", ["", "projection_bias", "residual", "gate residual", "projection_bias gate", "scale shift",
                                      "projection_bias gate residual scale shift"])
def test_layer_norm(ctx_factory, mode, dtype, rows, cols, operands):
    from breeze_tts_cpp_b200 import ops
    ctx, source = ctx_factory(mode), Source(rows + cols, dtype)
    x = source.rows(rows, cols, 1.5, 0.25, special=True)
    weight, bias = source.rows(1, cols, 0.2, 1.0), source.rows(1, cols, 0.3)
    fusion = {name: source.rows(rows if name == "residual" else 1, cols, 0.7) for name in operands.split()}
    if "projection_bias" in fusion:
        fusion["projection_bias"][0, :cols // 4] = -0.0
    results = []
    for place in (lambda t: t, off_alignment):
        out, kept, raw = view(ops, mode, rows, cols), place(torch.zeros_like(x)), place(torch.zeros_like(x))
        ctx.layer_norm_quantize(place(x), out, place(weight), place(bias), 1e-5, retained=kept, raw=raw,
                                **{name: place(t) for name, t in fusion.items()})
        results.append((raw, kept, out.scales, out.values))
    for packed, general in zip(*results):
        assert same_bits(packed, general)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(3, 128), (301, 2048), (600, 1152)])
@pytest.mark.parametrize("update,scaled", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("gemma", [False, True])
def test_rms_norm(ctx_factory, mode, dtype, rows, cols, update, scaled, gemma):
    from breeze_tts_cpp_b200 import ops
    ctx, source = ctx_factory(mode), Source(rows + cols, dtype)
    x, weight = source.rows(rows, cols, special=True), source.rows(1, cols, 0.1, 1.0)
    add, scale = source.rows(rows, cols, 0.7) if update else None, source.rows(1, cols, 0.5) if scaled else None
    results = []
    for place in (torch.Tensor.clone, off_alignment):
        out, residual = view(ops, mode, rows, cols), place(x)
        ctx.quantized_norm(residual, None if add is None else place(add), place(weight), out, 1e-6, gemma,
                           None if scale is None else place(scale))
        results.append((residual, out.scales, out.values))
    for packed, general in zip(*results):
        assert same_bits(packed, general)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(3, 128), (64, 6144), (301, 2048), (1300, 1152)])
def test_gate_and_rows(ctx_factory, mode, dtype, rows, cols):
    from breeze_tts_cpp_b200 import ops
    ctx, source = ctx_factory(mode), Source(rows + cols, dtype)
    x = source.rows(rows, 2 * cols, 2.0, special=True)
    results = []
    for place in (lambda t: t, off_alignment):
        gated, plain = view(ops, mode, rows, cols), view(ops, mode, rows, cols)
        ctx.quantized_gated(place(x), gated)
        ctx.quantize_rows(place(x[:, :cols].contiguous()), plain)
        results.append((gated.scales, gated.values, plain.scales, plain.values))
    for packed, general in zip(*results):
        assert same_bits(packed, general)
