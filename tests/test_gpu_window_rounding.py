"""Planned segmented Reduce: a long vector among many short ones is folded in
chains no longer than a warp's, one of up to 256 elements in four or more."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long,ones,bits", [(3072, 300, 20), (3072, 40, 20), (512, 40, 21), (256, 200, 19),
                                            (256, 4, 19), (256, 2, 19), (256, 0, 19)])
def test_long_among_short(scl, long, ones, bits):
    """Whole numbers whose second half undoes the first: with chains of at most
    long / 128 elements (long / 4 up to 256) single precision holds every
    partial sum."""
    rng = np.random.default_rng(long + ones)
    lens = np.tile([long] + [1] * ones, 60)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    n = int(off[-1])
    x = rng.integers(1 << (bits - 1), 1 << bits, n).astype(np.float32)
    for s in np.flatnonzero(lens == long):
        lo = int(off[s])
        x[lo + long // 2:lo + long] = -x[lo:lo + long // 2]
        x[lo + long - 1] += s
    add = "float func(float x, float y){ return x + y; }"
    dx, doff, out = S.DeviceArray.from_numpy(x), S.DeviceArray.from_numpy(off), S.DeviceArray(len(lens), np.float32)
    plan = S.SegPlan(doff, n)
    S.Program(S.KIND_REDUCE, add, ["float"], identity="0").launch([dx, out], n=n, segments=plan)
    assert np.array_equal(out.to_numpy(), np.add.reduceat(x.astype(np.float64), off[:-1].astype(np.int64)))
    plan.release()
