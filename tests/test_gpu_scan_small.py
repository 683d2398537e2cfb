"""Scan and the fused Scan-Map around the sizes at which the tile changes: half
tiles while the whole ones leave SMs idle.  Whole numbers, so results are
exact; a second launch finds the first's state put back."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.uint8, np.int16])
@pytest.mark.parametrize("flags", [0, S.SHAPE_INCLUSIVE, S.SHAPE_INCLUSIVE | S.SHAPE_REVERSE, S.SHAPE_REVERSE])
def test_scan_sizes(scl, dtype, flags):
    t = S.CL_TYPE[np.dtype(dtype)]
    add = f"{t} func({t} x, {t} y){{ return x + y; }}"
    scan = S.Program(S.KIND_SCAN, add, [t], identity="0")
    fused = S.Program(S.KIND_SCAN_MAP, add, [t] * 2, source2=f"{t} m({t} x){{ return x + x; }}", func2="m",
                      identity="0")
    tile = 2048 * (16 // np.dtype(dtype).itemsize)
    rng = np.random.default_rng(3)
    sizes = {1, 31, tile // 2 - 1, tile // 2, tile // 2 + 1, tile, 5 * tile + 3, 76 * tile - 1, 76 * tile,
             76 * tile + 1, 80 * tile}
    for n in sorted(sizes):
        for shift in (0, 1):
            x = rng.integers(0, 2, n + shift).astype(dtype)
            base, out = S.DeviceArray.from_numpy(x), S.DeviceArray(n, dtype)
            v = x[shift:][::-1] if flags & S.SHAPE_REVERSE else x[shift:]
            s = np.cumsum(v, dtype=np.int64)
            s = s if flags & S.SHAPE_INCLUSIVE else s - v.astype(np.int64)
            want = (s[::-1] if flags & S.SHAPE_REVERSE else s).astype(dtype)
            for _ in range(2):
                scan.launch([base.view(shift, n), out], n=n, flags=flags)
                assert np.array_equal(out.to_numpy(), want), (n, shift)
                fused.launch([base.view(shift, n), out], n=n, flags=flags)
                assert np.array_equal(out.to_numpy(), (want + want).astype(dtype)), (n, shift)
