"""Planned segmented Scan and Reduce where the windows' form changes: the longest
vectors of a window of 8-byte elements, and how many vectors of which lengths
share a record of the Reduce.  Whole numbers, so every result is exact."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def segments(pattern, total, seed):
    rng = np.random.default_rng(seed)
    lens = []
    while sum(lens) < total:
        lens += list(rng.permutation(pattern))
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)


@pytest.mark.parametrize("dtype", [np.float64, np.int64])
@pytest.mark.parametrize("pattern", [[1023, 1024, 1025, 0], [2047, 2048, 2049, 1, 0], [7, 8, 9, 255, 256, 257], [2048]])
@pytest.mark.parametrize("shift,items", [(0, 0), (1, 0), (1, 16)])
def test_wide_scan_windows(scl, dtype, pattern, shift, items):
    off = segments(pattern, 50_000, 5)
    n, o = int(off[-1]), off.astype(np.int64)
    x = np.random.default_rng(6).integers(0, 9, n + shift).astype(dtype)
    v, lens = x[shift:].astype(np.int64), np.diff(o)
    c = np.concatenate([[0], np.cumsum(v)])
    forward = c[1:] - np.repeat(c[o[:-1]], lens)
    backward = np.repeat(c[o[1:]], lens) - c[:-1]
    t = S.CL_TYPE[np.dtype(dtype)]
    scan = S.Program(S.KIND_SCAN, f"{t} func({t} x, {t} y){{ return x + y; }}", [t], identity="0")
    base, out = S.DeviceArray.from_numpy(x), S.DeviceArray(n + shift, dtype)
    plan = S.SegPlan(S.DeviceArray.from_numpy(off), n)
    for flags in (0, S.SHAPE_INCLUSIVE, S.SHAPE_REVERSE, S.SHAPE_INCLUSIVE | S.SHAPE_REVERSE):
        want = backward if flags & S.SHAPE_REVERSE else forward
        if not flags & S.SHAPE_INCLUSIVE:
            want = want - v
        scan.launch([base.view(shift, n), out.view(shift, n)], n=n, flags=flags, segments=plan,
                    tuning=S.Tuning(items=items))
        assert np.array_equal(out.to_numpy()[shift:], want.astype(dtype)), flags
    plan.release()


@pytest.mark.parametrize("dtype", [np.float32, np.uint8, np.int16, np.float64])
@pytest.mark.parametrize("pattern", [[4096, 0, 4095], [512] * 8, [455] * 9, [500] * 7 + [0, 33],  # a warp each
                                     [4000] + [3] * 20, [900] + [31, 32, 33] * 6,                 # uneven
                                     [300] * 15, [128] * 31 + [130], [4000] + [1] * 31])          # groups
@pytest.mark.parametrize("shift", [0, 1])
def test_reduce_records(scl, dtype, pattern, shift):
    off = segments(pattern, 60_000, 7)
    n, o = int(off[-1]), off.astype(np.int64)
    x = np.random.default_rng(8).integers(0, 9, n + shift).astype(dtype)
    c = np.concatenate([[0], np.cumsum(x[shift:].astype(np.int64))])
    want = (c[o[1:]] - c[o[:-1]]).astype(dtype)
    t = S.CL_TYPE[np.dtype(dtype)]
    red = S.Program(S.KIND_REDUCE, f"{t} func({t} x, {t} y){{ return x + y; }}", [t], identity="0")
    base, out = S.DeviceArray.from_numpy(x), S.DeviceArray(len(want), dtype)
    plan = S.SegPlan(S.DeviceArray.from_numpy(off), n)
    red.launch([base.view(shift, n), out], n=n, segments=plan)
    assert np.array_equal(out.to_numpy(), want)
    plan.release()


@pytest.mark.parametrize("dtype,code", [(np.float32, S.DTYPE_F32), (np.float64, S.DTYPE_F64)])
@pytest.mark.parametrize("mean", [47, 48, 199, 200])
@pytest.mark.parametrize("shift", [0, 1])
def test_broadcast_forms(scl, dtype, code, mean, shift):
    lens = np.random.default_rng(9).permutation(np.tile([0, 1, mean - 1, mean, mean + 1, 2 * mean - 1, 2 * mean], 300))
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    n = int(off[-1])
    assert n // len(lens) == mean
    rng = np.random.default_rng(10)
    g, x = rng.integers(-99, 100, len(lens)).astype(dtype), rng.integers(-99, 100, n + shift).astype(dtype)
    dg, doff = S.DeviceArray.from_numpy(g), S.DeviceArray.from_numpy(off)
    for acc in (0, 1):
        gx = S.DeviceArray.from_numpy(x)
        S.check(S.lib().scl_adjoint_broadcast_segments(dg.ptr, gx.view(shift, n).ptr, doff.ptr, len(lens), n, code, acc))
        assert np.array_equal(gx.to_numpy()[shift:], np.repeat(g, lens) + (x[shift:] if acc else 0)), acc
        assert np.array_equal(gx.to_numpy()[:shift], x[:shift])
