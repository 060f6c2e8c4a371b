"""A layer on a few rows quantizes them inside the GEMM's launch: the same bits as the quantizer and the GEMM one after the other, at
the edges of what the launch takes (rows per warp, K blocks per split, alignment, strides), for every finishing chain, for
infinities and NaN, and where it declines."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pair(ctx_factory, mode, rows, k, n, dtype, bias=False, seed=0):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    g = torch.Generator(device="cuda").manual_seed(seed + rows * k + n)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(dtype)
    w = draw(n, k)
    b = draw(1, n) if bias else None
    layer = ops.Linear(ctx, [w], bias=b, max_rows=rows)
    group, _, rotation = ops.groups_of(mode)
    wv = ctx.quantize_rows(w, ops.RowScaledView.empty(n, k, ops.format_of(mode), group, rotation))
    scratch = ops.RowScaledView.empty(rows, k, ops.format_of(mode), group, rotation)
    ctx.prepare_quantized(rows, n, k, out_dtype=dtype, weight=wv)

    def compare(x, residual=None, out=None, **epilogue):
        if residual is not None:
            epilogue["residual"] = residual
        if b is not None:
            epilogue_two = dict(epilogue, bias=b)
        else:
            epilogue_two = epilogue
        one = torch.full((rows, n), float("nan"), dtype=dtype, device="cuda") if out is None else out
        two = torch.full((rows, n), float("nan"), dtype=dtype, device="cuda")
        ctx.linear(x, wv, scratch, two, **epilogue_two)  # its scratch is the caller's: two launches
        layer.forward(x, one, **epilogue)
        assert ctx.status() == 0
        assert torch.equal(one.view(torch.int16), two.view(torch.int16))
    return draw, compare


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("rows,k,n", [(1, 128, 16), (1, 2048, 2048), (2, 6144, 2048), (3, 2048, 4096), (4, 1408, 144), (5, 2048, 2048),
                                      (8, 2048, 2064), (9, 2048, 2048), (16, 1024, 256), (1, 16384, 256), (2, 16384, 256), (1, 144, 64),
                                      (17, 384, 512), (1, 2048, 12288)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_same_bits_as_two_launches(ctx_factory, mode, rows, k, n, dtype):
    if mode.startswith("group") and k % 128:
        pytest.skip("K groups need whole blocks")
    draw, compare = _pair(ctx_factory, mode, rows, k, n, dtype)
    compare(draw(rows, k))
    compare(torch.zeros(rows, k, dtype=dtype, device="cuda"))
    wide = draw(rows, k + 32)
    compare(wide[:, :k])  # a stride
    compare(wide[:, 1:k + 1])  # rows that cannot be read in 16-byte pieces


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("activation", [0, 1, 3, 4])
def test_finishing_chain(ctx_factory, mode, activation):
    draw, compare = _pair(ctx_factory, mode, 6, 1024, 528, torch.bfloat16, bias=True)
    compare(draw(6, 1024), residual=draw(6, 528), activation=activation, value_scale=0.7, residual_scale=1.3, output_scale=0.9)
    compare(draw(6, 1024), activation=activation, gate=draw(2, 528), rows_per_sequence=3, residual=draw(6, 528))
    compare(draw(6, 1024), residual_f32=torch.randn(6, 528, device="cuda"))


@pytest.mark.parametrize("mode", ["int8", "fp8", "group_int8", "group_fp8"])
@pytest.mark.parametrize("rows", [1, 3, 7])
def test_infinities_nan_and_tiny_values(ctx_factory, mode, rows):
    draw, compare = _pair(ctx_factory, mode, rows, 512, 128, torch.bfloat16)
    for value in (float("inf"), float("-inf"), float("nan"), 1e-38, 3e38):
        x = draw(rows, 512)
        x[rows // 2, 77] = value
        x[0, 300] = value
        compare(x)
    compare(torch.full((rows, 512), float("nan"), dtype=torch.bfloat16, device="cuda"))


@pytest.mark.parametrize("mode", ["int8", "group_int8"])
def test_output_over_its_input(ctx_factory, mode):
    """Every CTA reads whole rows, so a result in their place has to wait for all of them: two launches."""
    draw, compare = _pair(ctx_factory, mode, 4, 512, 512, torch.bfloat16)
    for _ in range(5):
        x = draw(4, 512)
        compare(x, out=x)


def _kernels(run):
    """Names of the library's kernels that `run` launches."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as trace:
        run()
        torch.cuda.synchronize()
    names = (e.name for e in trace.events())
    return ["gemm" if "w8a8_tcgen05_gemm" in n else "quantize" for n in names if "w8a8_tcgen05" in n or "row_quantize" in n]


@pytest.mark.parametrize("mode,rows,k,n,one", [
    ("int8", 1, 2048, 2048, True), ("int8", 8, 2048, 2048, True), ("int8", 9, 2048, 2048, False), ("fp8", 2, 6144, 2048, True),
    ("fp8", 4, 6144, 2048, False), ("int8", 3, 2048, 12288, True), ("int8", 4, 2048, 12288, False), ("int8", 1, 144, 64, False),
    ("group_int8", 1, 2048, 4096, True), ("group_int8", 8, 6144, 2048, True), ("group_fp8", 21, 384, 512, True), ("group_fp8", 33, 384, 512, False)])
def test_which_calls_are_one_launch(ctx_factory, mode, rows, k, n, one):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    layer = ops.Linear(ctx, [torch.randn(n, k, device="cuda").to(torch.bfloat16)], max_rows=rows)
    x, out = torch.randn(rows, k, device="cuda").to(torch.bfloat16), torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")
    layer.forward(x, out)
    assert _kernels(lambda: layer.forward(x, out)) == (["gemm"] if one else ["quantize", "gemm"])


@pytest.mark.parametrize("mode,rows,one", [("int8", 1, False), ("int8", 3, False), ("group_fp8", 4, True), ("group_fp8", 5, False)])
def test_captured_calls(mode, rows, one):
    from breeze_tts_cpp_b200 import ops
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = ops.Context(mode, stream=stream)
        layer = ops.Linear(ctx, [torch.randn(512, 1024, device="cuda").to(torch.bfloat16)], max_rows=rows)
        x, eager, replayed = torch.randn(rows, 1024, device="cuda").to(torch.bfloat16), *(torch.zeros(rows, 512, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        layer.forward(x, eager)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            layer.forward(x, replayed)
        assert _kernels(graph.replay) == (["gemm"] if one else ["quantize", "gemm"])
    torch.cuda.synchronize()
    assert torch.equal(eager.view(torch.int16), replayed.view(torch.int16))
    del graph
    ctx.close()
