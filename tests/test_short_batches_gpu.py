"""The producers with one scale per row around the row counts where their launches change: CTA widths of the gate, the rehearsal of
short batches (a kernel walks its code once before its input exists), against the oracle-checked general form on single rows. Each
producer follows a kernel that overwrites its input, so that a read ahead of that kernel shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["int8", "fp8"])
@pytest.mark.parametrize("cols", [2048, 2056, 4096, 6144, 8192])
@pytest.mark.parametrize("rows", [1, 148, 149, 296, 297, 740, 741])
def test_gate_by_row_count(ctx_factory, mode, cols, rows):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, 2 * cols, generator=g, device="cuda").to(torch.bfloat16)
    whole = ctx.quantized_gated(x, ops.RowScaledView.empty(rows, cols, ops.format_of(mode)))
    for row in sorted({0, rows // 2, rows - 1}):
        one = ctx.quantized_gated(x[row:row + 1].clone(), ops.RowScaledView.empty(1, cols, ops.format_of(mode)))
        assert torch.equal(one.values[0], whole.values[row]) and float(one.scales[0]) == float(whole.scales[row])


@pytest.mark.parametrize("mode", ["int8", "fp8"])
@pytest.mark.parametrize("rows", [3, 64, 148])
def test_inputs_written_by_the_kernel_before(ctx_factory, mode, rows):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    fmt, k, n = ops.format_of(mode), 2048, 4096
    g = torch.Generator(device="cuda").manual_seed(rows)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    w = ctx.quantize_rows(draw(n, k), ops.RowScaledView.empty(n, k, fmt))
    ctx.prepare_quantized(rows, n, k, weight=w)
    gamma, update = draw(1, k), torch.zeros(rows, k, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    y = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
    q = lambda c: ops.RowScaledView.empty(rows, c, fmt)
    for _ in range(8):
        x = ctx.quantize_rows(draw(rows, k), q(k))
        y.fill_(7.0)
        torch.cuda.synchronize()
        ctx.matmul(x, w, y)
        rows_q, gate_q = q(n), q(n // 2)
        ctx.quantize_rows(y, rows_q)
        ctx.matmul(x, w, y)
        ctx.quantized_gated(y, gate_q)
        torch.cuda.synchronize()
        again = ctx.quantize_rows(y, q(n)), ctx.quantized_gated(y, q(n // 2))
        for one, two in zip((rows_q, gate_q), again):
            assert torch.equal(one.values, two.values) and torch.equal(one.scales, two.scales)
        residual = draw(rows, n)[:, :k].contiguous()
        norm_q, norm_again, kept = q(k), q(k), residual.clone()
        ctx.quantized_norm(residual, update, gamma, norm_q, 1e-6)  # writes the residual back ...
        ctx.quantized_norm(residual, update, gamma, norm_again, 1e-6)  # ... in front of this one
        assert torch.equal(residual, kept) and torch.equal(norm_q.values, norm_again.values)


@pytest.mark.parametrize("mode", ["int8", "fp8"])
@pytest.mark.parametrize("rows", [1, 5, 64, 148])
def test_norm_repeats_itself(ctx_factory, mode, rows):
    """The rehearsal and the pass behind it share memory: a short batch, over and over, against the same rows in a batch too long for one."""
    from breeze_tts_cpp_b200 import ops
    ctx, fmt, k = ctx_factory(mode), ops.format_of(mode), 2048
    g = torch.Generator(device="cuda").manual_seed(rows)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    x, update, gamma = draw(600, k), draw(600, k), draw(1, k)
    torch.cuda.synchronize()  # gamma is a parameter
    whole = ctx.quantized_norm(x.clone(), update, gamma, ops.RowScaledView.empty(600, k, fmt), 1e-6)
    outs = [ops.RowScaledView.empty(rows, k, fmt) for _ in range(200)]
    inputs = [x[:rows].clone() for _ in outs]
    for kept, out in zip(inputs, outs):
        ctx.quantized_norm(kept, update[:rows], gamma, out, 1e-6)
    assert torch.equal(torch.stack([o.values for o in outs]), whole.values[:rows].expand(len(outs), -1, -1))
    assert torch.equal(torch.stack([o.scales for o in outs]), whole.scales[:rows].expand(len(outs), -1, -1))
