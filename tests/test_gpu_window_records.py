"""Planned segmented Scan and Reduce over window records: whole-number data,
so that every result is exact whatever the order of the folds."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu

# lengths at the edges of a lane's chunk, a row, a vector of the window, the
# longest one of a scan's and of a reduce's window (32-bit elements), and how
# many vectors share a record: one thread or many, several warps, one each
PATTERNS = {
    "edges": [1, 7, 8, 9, 0, 15, 16, 17, 255, 256, 257, 2047, 2048, 2049, 0, 0, 4095, 4096, 4097],
    "ones": [1],
    "tiny": [0, 1, 2, 3],
    "forty": [150, 3, 90, 199],
    "few": [1500, 1999],
    "pairs": [3000, 3001],
    "one": [4096, 4000],
    "empty": [0],
}


def expect(x, off, inclusive, reverse):
    out, sums = np.empty_like(x), np.zeros(len(off) - 1, x.dtype)
    for s in range(len(off) - 1):
        v = x[off[s]:off[s + 1]]
        w = v[::-1] if reverse else v
        c = np.cumsum(w, dtype=x.dtype)
        if not inclusive:
            c = c - w
        out[off[s]:off[s + 1]] = c[::-1] if reverse else c
        sums[s] = v.sum(dtype=x.dtype)
    return out, sums


@pytest.mark.parametrize("dtype", [np.int32, np.uint8, np.float64])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_window_records(scl, pattern, shift, dtype):
    rng = np.random.default_rng(3)
    total = 0 if pattern == "empty" else 40_000
    lens = []
    while sum(lens) < total or len(lens) < 300:
        lens += list(rng.permutation(PATTERNS[pattern]))
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    n = int(off[-1])
    x = rng.integers(0, 5, n + shift).astype(dtype)
    t = S.CL_TYPE[np.dtype(dtype)]
    add = f"{t} func({t} x, {t} y){{ return x + y; }}"
    base = S.DeviceArray.from_numpy(x if len(x) else np.zeros(1, dtype))
    dx, dy = base.view(shift, n), S.DeviceArray(n + shift, dtype).view(shift, n)
    dr, doff = S.DeviceArray(len(lens), dtype), S.DeviceArray.from_numpy(off)
    plan = S.SegPlan(doff, n)
    scan, red = (S.Program(k, add, [t], identity="0") for k in (S.KIND_SCAN, S.KIND_REDUCE))
    io = off.astype(np.int64)
    for flags in (0, S.SHAPE_INCLUSIVE, S.SHAPE_REVERSE, S.SHAPE_INCLUSIVE | S.SHAPE_REVERSE):
        want, sums = expect(x[shift:], io, flags & S.SHAPE_INCLUSIVE, flags & S.SHAPE_REVERSE)
        if n:
            scan.launch([dx, dy], n=n, flags=flags, segments=plan)
            assert np.array_equal(dy.to_numpy(), want), (pattern, flags)
    red.launch([dx, dr], n=n, segments=plan)
    assert np.array_equal(dr.to_numpy(), sums)
    plan.release()
