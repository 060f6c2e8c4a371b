"""Plans of one 128-token tile per slab take the CTA-pair kernel when a finishing chain follows: the same rows as GEMM and finishing pass one
after the other, on both sides of the rule (one token tile, several; with and without a chain; outputs that kernel cannot store)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["int8", "fp8"])
@pytest.mark.parametrize("rows,n,k", [(128, 4096, 1024), (129, 4096, 1024), (420, 2064, 512), (301, 144, 2048), (257, 2048, 144)])
@pytest.mark.parametrize("activation", [0, 1, 2, 3])
def test_one_plan_with_and_without_a_chain(ctx_factory, mode, rows, n, k, activation):
    from breeze_tts_cpp_b200 import ops
    ctx, fmt = ctx_factory(mode), ops.format_of(mode)
    g = torch.Generator(device="cuda").manual_seed(rows + n + k)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
    x, w = (ctx.quantize_rows(draw(r, k), ops.RowScaledView.empty(r, k, fmt)) for r in (rows, n))
    bias, residual = draw(1, n), draw(rows, n)
    values = lambda q: q.values.view(torch.float8_e4m3fn).float().abs() * q.scales
    plain, want, got = (torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    unaligned = torch.empty(rows * n + 1, dtype=torch.bfloat16, device="cuda")[1:].view(rows, n)  # rows that no vector store reaches
    path = (5, 128, 128, 1)
    if mode == "fp8":
        magnitudes = (values(x) @ values(w).T).double()
    ctx.quant_linear(path, x, w, plain)
    ctx.pointwise(plain, want, bias=bias, residual=residual, activation=activation)
    ctx.quant_linear(path, x, w, got, bias=bias, residual=residual, activation=activation)
    ctx.quant_linear(path, x, w, unaligned, bias=bias, residual=residual, activation=activation)
    assert ctx.status() == 0
    for result in (got, unaligned):
        if mode == "int8":
            assert torch.equal(result.view(torch.int16), want.view(torch.int16))
        else:
            # Each kernel's fp32 sum of k products is within k * 2^-24 of the sum of their magnitudes; after that every rounding to bf16 (the
            # plain row, bias, residual, activation) may fall to the neighbouring value, 2^-7 of it at most, and the activations steepen an error by less than 1.13.
            step = lambda v: v.abs() / 128
            mid = plain.double() + bias.double()
            before = mid + residual.double()
            bound = step(plain.double()) + 2 * k * 2.0 ** -24 * magnitudes + step(mid) + step(before)
            assert bool(((result.double() - want.double()).abs() <= 1.13 * bound + step(want.double())).all())
