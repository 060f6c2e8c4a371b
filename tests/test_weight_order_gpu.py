"""A GEMM enqueued behind the kernel that writes its weight reads the finished weight, whichever kernel it takes, also when that
kernel is still running two launches back: not announced, announced after the writing call, and announced before and overwritten."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("rows", [4, 96, 640])  # streaming, streaming or persistent, persistent
@pytest.mark.parametrize("announced", ["no", "after", "before"])
def test_weight_written_in_stream_order(mode, rows, announced):
    from breeze_tts_cpp_b200 import ops
    n, k = 12288, 2048
    group, _, rotation = ops.groups_of(mode)
    view = lambda r: ops.RowScaledView.empty(r, k, ops.format_of(mode), group, rotation)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, xv, wv = torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16), view(rows), view(n)
    old, new = ((torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16) for _ in range(2))
    want, got = (torch.empty(rows, n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ctx = ops.Context(mode)
    ctx.prepare_quantized(rows, n, k)
    for matrix, out in ((old, got), (new, want), (old, got)):  # loads every kernel; leaves the old weight behind
        ctx.quantize_rows(matrix, wv)
        torch.cuda.synchronize()
        ctx.quantize_rows(x, xv)
        ctx.matmul(xv, wv, out)
        torch.cuda.synchronize()
    if announced == "before":
        ctx.prepare_quantized(rows, n, k, weight=wv)
        torch.cuda.synchronize()
    ctx.quantize_rows(new, wv)
    if announced == "after":
        ctx.prepare_quantized(rows, n, k, weight=wv)
    ctx.quantize_rows(x, xv)
    ctx.matmul(xv, wv, got)
    assert ctx.status() == 0 and torch.equal(got, want)
    # and when only part of an announced weight is written
    if announced == "before" and not group:
        ctx.quantize_rows(old[: n // 2], wv.rows(0, n // 2))
        ctx.quantize_rows(x, xv)
        ctx.matmul(xv, wv, got)
        torch.cuda.synchronize()
        ctx.matmul(xv, wv, want)
        assert torch.equal(got, want)
    ctx.close()
