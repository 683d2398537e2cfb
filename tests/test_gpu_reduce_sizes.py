"""Reduce and the fused Zip-Reduce where their grid changes: one block, a
block per SM, full rounds of loads; whole numbers, so every result is exact."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.uint8])
@pytest.mark.parametrize("shift", [0, 1])
def test_reduce_sizes(scl, dtype, shift):
    t = S.CL_TYPE[np.dtype(dtype)]
    add = f"{t} func({t} x, {t} y){{ return x + y; }}"
    red = S.Program(S.KIND_REDUCE, add, [t], identity="0")
    dot = S.Program(S.KIND_ZIP_REDUCE, add, [t] * 3, source2=f"{t} m({t} x, {t} y){{ return x * y; }}", func2="m",
                    identity="0")
    rng = np.random.default_rng(8)
    V = 16 // np.dtype(dtype).itemsize
    edges = [1, 255, 512, 2048, 4096, 152 * 256, 152 * 256 * 4, 152 * 256 * 8]
    for n in sorted({1, 2, 31, 33} | {max(1, e * V + d) for e in edges for d in (-1, 0, 1)}):
        if n > 3_000_000:
            continue
        x = rng.integers(0, 4, n + shift).astype(dtype)
        base, out = S.DeviceArray.from_numpy(x), S.DeviceArray(1, dtype)
        v = base.view(shift, n)
        for _ in range(2):  # (the second finds the first's ticket put back)
            red.launch([v, out], n=n)
            assert out.to_numpy()[0] == x[shift:].sum(dtype=dtype), n
            dot.launch([v, v, out], n=n)
            assert out.to_numpy()[0] == (x[shift:] * x[shift:]).sum(dtype=dtype), n
