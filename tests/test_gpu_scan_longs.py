"""Scan of 64-bit whole numbers around the size at which its tile changes."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, S.SHAPE_INCLUSIVE, S.SHAPE_INCLUSIVE | S.SHAPE_REVERSE, S.SHAPE_REVERSE])
def test_scan_longs(scl, flags):
    scan = S.Program(S.KIND_SCAN, "long func(long x, long y){ return x + y; }", ["long"], identity="0")
    rng = np.random.default_rng(3)
    tile = 4096
    for n in (1, tile + 1, 38 * tile - 1, 38 * tile, 38 * tile + 1, 76 * tile + 1):
        for shift in (0, 1):
            x = rng.integers(-(1 << 40), 1 << 40, n + shift).astype(np.int64)
            base, out = S.DeviceArray.from_numpy(x), S.DeviceArray(n, np.int64)
            v = x[shift:][::-1] if flags & S.SHAPE_REVERSE else x[shift:]
            s = np.cumsum(v) - (0 if flags & S.SHAPE_INCLUSIVE else v)
            for _ in range(2):
                scan.launch([base.view(shift, n), out], n=n, flags=flags)
                assert np.array_equal(out.to_numpy(), s[::-1] if flags & S.SHAPE_REVERSE else s), (n, shift)
