"""The persistent K-group kernel at the edges of its tiles (128 tokens, 64 or 128 channels): any number of rows, ragged
channels, one and many K blocks, one and several tiles per CTA, both output types, with and without the finishing chain,
against the weight-streaming K-group kernel on the same operands. INT8 adds the same products in the same order, so an
unsplit launch gives the same bits. And that kernel at every token tile, unsplit with more K blocks than its ring and its
accumulators hold, against the oracle."""
import numpy as np
import pytest
import torch

from tests import synth
from tests.oracle_binding import FP8, I8

pytestmark = pytest.mark.gpu
TCGEN05 = 5
SHAPES = [(65, 64, 128), (129, 144, 256), (127, 2048, 640), (301, 4096, 512), (443, 2064, 384), (1021, 2048, 1024), (1302, 1152, 256),
          (2500, 4096, 128), (640, 4096, 2176)]


@pytest.mark.parametrize("mode,fmt", [("group_int8", I8), ("group_fp8", FP8)])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("dtype,chain", [(torch.bfloat16, None), (torch.float16, None), (torch.bfloat16, 0), (torch.float16, 4),
                                         (torch.bfloat16, 3)])
def test_persistent_group_kernel_matches_weight_streaming_kernel(ctx_factory, mode, fmt, m, n, k, dtype, chain):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    xv = ctx.quantize_rows(x, ops.RowScaledView.empty(m, k, fmt, 128, 128))
    wv = ctx.quantize_rows(w, ops.RowScaledView.empty(n, k, fmt, 128, 128))
    kw = {}
    if chain is not None:
        kw = dict(bias=torch.randn(1, n, generator=g, device="cuda").to(dtype), activation=chain, value_scale=0.7,
                  residual=torch.randn(m, n, generator=g, device="cuda").to(dtype), residual_scale=1.3, output_scale=0.9)
    out, other = (torch.full((m, n), float("nan"), dtype=dtype, device="cuda") for _ in range(2))
    ctx.quant_linear((TCGEN05, 128, 128, 1), xv, wv, out, **kw)
    ctx.quant_linear((TCGEN05, 64, 128, 1), xv, wv, other, **kw)
    assert ctx.status() == 0
    if fmt == I8:
        assert torch.equal(out.view(torch.int16), other.view(torch.int16))
    else:
        assert float((out.double() - other.double()).norm() / other.double().norm()) < 2e-3


# Rounds of K blocks that are not full, over several tiles per CTA and over one; an fp32 residual, rows and channels past the end.
@pytest.mark.parametrize("m,n,k", [(1302, 4096, 384), (1150, 2064, 640), (301, 4096, 128), (300, 144, 640), (97, 1024, 896)])
def test_persistent_group_kernel_with_fp32_residual(ctx_factory, m, n, k):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory("group_int8")
    g = torch.Generator(device="cuda").manual_seed(m * n + k)
    xv = ctx.quantize_rows(torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16), ops.RowScaledView.empty(m, k, I8, 128, 128))
    wv = ctx.quantize_rows(torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16), ops.RowScaledView.empty(n, k, I8, 128, 128))
    residual = torch.randn(m, n, generator=g, device="cuda")
    out, other = (torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ctx.quant_linear((TCGEN05, 128, 128, 1), xv, wv, out, residual_f32=residual)
    ctx.quant_linear((TCGEN05, 64, 128, 1), xv, wv, other, residual_f32=residual)
    assert ctx.status() == 0
    assert torch.equal(out.view(torch.int16), other.view(torch.int16))  # the same products added in the same order


@pytest.mark.parametrize("late", [0, 100_000])  # nanoseconds the refill waiter starts late: by then stages may have been filled twice
@pytest.mark.parametrize("group,m,tokens,splits,k", [(128, 3, 16, 1, 6144), (128, 20, 32, 1, 4096), (128, 64, 64, 1, 2560), (128, 100, 128, 2, 2304),
                                                     (32, 9, 16, 1, 3072), (64, 33, 64, 1, 2048), (0, 16, 16, 1, 6144), (0, 64, 64, 1, 3072)])
def test_weight_streaming_kernel_refills_ring_and_accumulators(oracle, ctx_factory, group, m, tokens, splits, k, late):
    from breeze_tts_cpp_b200 import _lib, ops
    ctx = ctx_factory("group_int8" if group else "int8")
    n = 144
    xq, sx = oracle.row_quantize(oracle.to_bf16(synth.activations(m, k, m + k, student_t=3.0)), I8, group, 0)
    wq, sw = oracle.row_quantize(oracle.to_bf16(synth.weights(n, k, m + k + 1)), I8, group, 0)
    scales = lambda s, rows: torch.from_numpy(s).cuda().reshape((-1, rows) if group else (rows, 1))
    xv = ops.RowScaledView(torch.from_numpy(xq).cuda(), scales(sx, m), I8, group, 0)
    wv = ops.RowScaledView(torch.from_numpy(wq).cuda(), scales(sw, n), I8, group, 0)
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    _lib.call("b200q_inject_refill_delay", late)
    ctx.quant_linear((TCGEN05, tokens, 128, splits), xv, wv, out)
    want, exact = oracle.quant_linear(xq, sx, wq, sw, I8, group, group)
    assert ctx.status() == 0
    if splits == 1:
        assert np.array_equal(out.view(torch.int16).cpu().numpy().view(np.uint16), want)
    else:
        assert float(np.linalg.norm(out.float().cpu().numpy() - exact) / np.linalg.norm(exact)) < 1e-2
