"""A per-sequence gate in the GEMM's own epilogue, against the projection followed by the finishing pass: identical bits, in
every kernel (streaming with and without split K, CTA pairs, K groups), for one gate row and one per sequence."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("sequences,length,k,n", [(1, 1, 256, 128), (3, 1, 512, 144), (4, 16, 2048, 512), (4, 93, 2048, 512),
                                                  (5, 300, 512, 2064), (2, 513, 128, 256)])
@pytest.mark.parametrize("dtype,shared,scales", [(torch.bfloat16, False, False), (torch.float16, True, True), (torch.bfloat16, True, True)])
def test_gate_equals_finishing_pass(ctx_factory, mode, sequences, length, k, n, dtype, shared, scales):
    from breeze_tts_cpp_b200 import ops
    ctx, m = ctx_factory(mode), sequences * length
    group, _, rotation = ops.groups_of(mode)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)
    w = ctx.quantize_rows(draw(n, k), ops.RowScaledView.empty(n, k, ops.format_of(mode), group, rotation))
    scratch = ops.RowScaledView.empty(m, k, ops.format_of(mode), group, rotation)
    ctx.prepare_quantized(m, n, k, out_dtype=dtype)
    x, bias = draw(m, k), draw(1, n)
    finish = dict(gate=draw(1 if shared else sequences, n), rows_per_sequence=length, residual=draw(m, n), activation=1 if scales else 0)
    if scales:
        finish.update(value_scale=0.7, residual_scale=1.3, output_scale=0.9)
    fused, raw, two = (torch.full((m, n), float("nan"), dtype=dtype, device="cuda") for _ in range(3))
    ctx.linear(x, w, scratch, fused, bias=bias, **finish)
    ctx.linear(x, w, scratch, raw)
    ctx.pointwise(raw, two, bias=bias, **finish)
    assert ctx.status() == 0
    assert torch.equal(fused.view(torch.int16), two.view(torch.int16))


def test_gate_is_refused_where_only_a_fused_finish_is_taken(ctx_factory):
    """matmul and the path-level entry points take what the GEMM alone has always taken; a gate goes through linear()."""
    import ctypes as C

    from breeze_tts_cpp_b200 import B200QError, _lib, ops
    ctx, m, n, k = ctx_factory("int8"), 4, 128, 256
    make = lambda *shape: torch.ones(*shape, dtype=torch.bfloat16, device="cuda")
    x, w = (ctx.quantize_rows(make(r, k), ops.RowScaledView.empty(r, k, ops.I8)) for r in (m, n))
    out, gate = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda"), make(1, n)
    ctx.prepare_quantized(m, n, k)
    with pytest.raises(B200QError, match="epilogue cannot be fused"):
        ctx.matmul(x, w, out, gate=gate)
    with pytest.raises(B200QError, match="unsupported quantized native Finish path"):
        ctx.quant_linear((5, 16, 128, 1), x, w, out, gate=gate)
    with pytest.raises(B200QError, match="unsupported quantized native Finish path"):
        _lib.call("b200q_quant_linear_static", 0, None, None, C.byref(x.c()), C.byref(w.c()), C.byref(ops._tensor(out)),
                  C.byref(ops._epilogue(gate=gate)))
    torch.cuda.synchronize()
    assert bool((out == 0).all())
