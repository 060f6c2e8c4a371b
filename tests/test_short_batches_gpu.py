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


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("rows", [3, 64, 65, 148])
@pytest.mark.parametrize("aligned", [True, False])
def test_inputs_written_by_the_kernel_before(ctx_factory, mode, rows, aligned):
    """Stale values are settled in a producer's input, then the GEMM that writes it and the producer are queued behind a long kernel, so that the
    producer starts while the GEMM runs. Unaligned rows take the producers' general forms."""
    from breeze_tts_cpp_b200 import ops
    ctx, k, n = ctx_factory(mode), 2048, 4096
    fmt, (group, _, rotation) = ops.format_of(mode), ops.groups_of(mode)
    g = torch.Generator(device="cuda").manual_seed(rows)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    q = lambda r, c: ops.RowScaledView.empty(r, c, fmt, group, rotation)
    place = lambda c: torch.empty(rows * c + 1, dtype=torch.bfloat16, device="cuda")[0 if aligned else 1:][:rows * c].view(rows, c)
    wide, square = (ctx.quantize_rows(draw(c, k), q(c, k)) for c in (n, k))
    for w, c in ((wide, n), (square, k)):
        ctx.prepare_quantized(rows, c, k, weight=w)
    gamma, beta, residual, busy = draw(1, k), draw(1, k), draw(rows, k), draw(4096, 4096)
    producers = [  # weight of the GEMM in front, its output's columns, the producer on that output -> tensors
        (wide, n, lambda y: ctx.quantize_rows(y, q(rows, n))),
        (wide, n, lambda y: ctx.quantized_gated(y, q(rows, n // 2))),
        (square, k, lambda y: ctx.quantized_norm(kept[-1], y, gamma, q(rows, k), 1e-6)),
        (square, k, lambda y: ctx.quantized_norm(y, residual, gamma, q(rows, k), 1e-6)),
        (square, k, lambda y: ctx.layer_norm_quantize(y, q(rows, k), gamma, beta)),
        (square, k, lambda y: ctx.layer_norm_quantize(residual, q(rows, k), gamma, beta, residual=y)),
    ]
    x = ctx.quantize_rows(draw(rows, k), q(rows, k))
    for w, columns, produce in producers:
        y, kept, got = place(columns), [], []
        for settled in (False, True, False, False):
            y.fill_(7.0)
            kept.append(residual.clone())
            torch.cuda.synchronize()
            torch.mm(busy, busy)
            ctx.matmul(x, w, y)
            if settled:
                torch.cuda.synchronize()
            out = produce(y)
            torch.cuda.synchronize()
            got.append((out.values, out.scales, y.clone(), kept[-1]))
        for other in got:
            assert all(torch.equal(a, b) for a, b in zip(other, got[1]))


@pytest.mark.parametrize("mode", ["int8", "fp8"])
@pytest.mark.parametrize("rows", [1, 5, 64, 65, 148])
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


@pytest.mark.parametrize("mode", ["int8", "group_fp8"])
@pytest.mark.parametrize("cols,rows", [(256, 1), (512, 1184), (512, 1185), (768, 148), (768, 149), (2048, 148), (2048, 149)])
def test_layer_norm_by_row_count(ctx_factory, mode, cols, rows):
    """On both sides of the rehearsal's limits, the rows of a batch too long for one."""
    from breeze_tts_cpp_b200 import ops
    ctx, fmt, (group, _, rotation) = ctx_factory(mode), ops.format_of(mode), ops.groups_of(mode)
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    x, residual, gamma, beta = draw(1300, cols), draw(1300, cols), draw(1, cols), draw(1, cols)
    whole = ctx.layer_norm_quantize(x, ops.RowScaledView.empty(1300, cols, fmt, group, rotation), gamma, beta, residual=residual)
    for _ in range(20):
        part = ctx.layer_norm_quantize(x[:rows], ops.RowScaledView.empty(rows, cols, fmt, group, rotation), gamma, beta, residual=residual[:rows])
        assert torch.equal(part.values, whole.values[:rows])
        assert torch.equal(part.scales, whole.scales[:, :rows] if group else whole.scales[:rows])
