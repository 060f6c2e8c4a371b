"""The block-wise rotation quantizers (four lanes per 128-column block) and the packed per-row ones at the sizes where
they can go wrong: one block, rows that are no multiple of eight, columns past the sign table, every stretch count of
the packed LayerNorm, infinities and NaN. Bytes and scales against the CPU oracle."""
import numpy as np
import pytest
import torch

from tests import synth
from tests.oracle_binding import BF16, F16, FP8, I8

pytestmark = pytest.mark.gpu
DTYPES = {BF16: torch.bfloat16, F16: torch.float16}


def device(x16, dtype):
    return torch.from_numpy(np.ascontiguousarray(x16).view(np.int16)).cuda().view(dtype)


def assert_bytes(got, want, fmt):
    got = got.cpu().numpy()
    differs = got != want
    if fmt == FP8:
        differs &= ((got | want) & 0x7F) != 0  # the sign of a zero
    assert not differs.any()


@pytest.mark.parametrize("fmt", [I8, FP8])
@pytest.mark.parametrize("rows,cols", [(1, 128), (7, 256), (9, 2048), (130, 384), (3, 8320), (1300, 640), (2, 16384)])
def test_rotated_blocks_match_oracle(oracle, ctx_factory, fmt, rows, cols):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory("group_fp8" if fmt == FP8 else "group_int8")
    x16 = oracle.to_bf16(synth.activations(rows, cols, rows + cols, student_t=3.0))
    out = ctx.quantize_rows(device(x16, torch.bfloat16), ops.RowScaledView.empty(rows, cols, fmt, 128, 128))
    values, scales = oracle.row_quantize(x16, fmt, 128, 128)
    assert np.array_equal(out.scales.cpu().numpy().reshape(scales.shape).view(np.uint32), scales.view(np.uint32))
    assert_bytes(out.values, values, fmt)


@pytest.mark.parametrize("mode,fmt,group", [("int8", I8, 0), ("fp8", FP8, 0), ("group_int8", I8, 128)])
@pytest.mark.parametrize("rows,cols", [(4, 256), (1300, 1024)])
def test_rows_with_infinities_and_nan_stay_to_themselves(ctx_factory, mode, fmt, group, rows, cols):
    """A row (or block) with an infinity or a NaN takes the clamping encoder; every other one keeps its bytes and scales."""
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory(mode)
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    clean = torch.randn(rows, cols, generator=g, device="cuda").to(torch.bfloat16)
    dirty = clean.clone()
    dirty[1, 5], dirty[2, cols - 1] = float("nan"), float("inf")
    want, got = (ctx.quantize_rows(x, ops.RowScaledView.empty(rows, cols, fmt, group, group)) for x in (clean, dirty))
    torch.cuda.synchronize()
    untouched = [0, *range(3, rows)]
    assert torch.equal(got.values[untouched], want.values[untouched])
    scales = (got.scales[:, untouched], want.scales[:, untouched]) if group else (got.scales[untouched], want.scales[untouched])
    assert torch.equal(*scales)
    if not group:
        assert bool(torch.isinf(got.scales[2]).all()) and bool(torch.isfinite(got.scales[1]).all())  # NaN does not count
        if fmt == I8:
            assert int(got.values[1, 5].view(torch.int8)) == -127  # a NaN encodes as the lower clamp


@pytest.mark.parametrize("type_code", [BF16, F16])
@pytest.mark.parametrize("rows,cols,group", [(3, 128, 0), (700, 256, 0), (5, 512, 128), (2, 776, 0), (33, 1024, 128), (9, 1536, 128),
                                             (600, 2048, 0), (4, 2048, 64)])
def test_packed_layer_norm_matches_oracle(oracle, ctx_factory, type_code, rows, cols, group):
    from breeze_tts_cpp_b200 import ops
    ctx = ctx_factory("group_int8" if group else "int8")
    rotation = 128 if group == 128 else 0
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    make = lambda r, s, m=0.0: (torch.randn(r, cols, generator=g, device="cuda") * s + m).to(DTYPES[type_code])
    x, weight, bias = make(rows, 1.5, 0.25), make(1, 0.2, 1.0), make(1, 0.3)
    fusion = dict(residual=make(rows, 1.0), scale=make(1, 0.5), shift=make(1, 0.5))
    kept, raw = torch.zeros_like(x), torch.zeros_like(x)
    out = ctx.layer_norm_quantize(x, ops.RowScaledView.empty(rows, cols, I8, group, rotation), weight, bias, 1e-5, retained=kept,
                                  raw=raw, **fusion)
    torch.cuda.synchronize()
    host = lambda t: t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)
    normalized, want_raw, _, _ = oracle.layer_norm_quantize(host(x), host(weight), host(bias), 1e-5, I8, group, rotation, type_code,
                                                            **{k: host(v) for k, v in fusion.items()})
    assert np.array_equal(host(raw), want_raw)
    a, b = kept.double().cpu(), torch.from_numpy(normalized.view(np.int16)).view(DTYPES[type_code]).double()
    # one storage step of the normalized value, carried through the scale and shift that follow it
    assert bool(((a - b).abs() <= (2.0 ** -6 if type_code == BF16 else 2.0 ** -9) * b.abs().clamp_min(1.0)).all())
    values, scales = oracle.row_quantize(host(kept), I8, group, rotation) if type_code == BF16 else (None, None)
    if values is not None:  # the kept rows quantize to exactly the bytes the kernel wrote
        assert np.array_equal(out.values.cpu().numpy(), values)
        assert np.array_equal(out.scales.cpu().numpy().reshape(scales.shape).view(np.uint32), scales.view(np.uint32))
