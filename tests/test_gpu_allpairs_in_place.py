"""AllPairs whose output takes an operand's place: X := X W by a small square W,
W := X W, X := X X."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,dtype", [("float", np.float32), ("int", np.int32), ("double", np.float64),
                                     ("unsigned char", np.uint8)])
@pytest.mark.parametrize("m,k", [(20, 20), (100, 100), (500, 100), (128, 128), (2000, 64), (2000, 200), (300, 256)])
def test_in_place(scl, t, dtype, m, k):
    p = S.Program(S.KIND_ALLPAIRS, f"{t} func({t} x, {t} y){{ return x+y; }}", [t] * 3,
                  source2=f"{t} func({t} x, {t} y){{ return x*y; }}", identity="0")
    rng = np.random.default_rng(m)
    x, w = rng.integers(0, 8, (m, k)).astype(dtype), rng.integers(0, 8, (k, k)).astype(dtype)

    def matmul(a, b):  # (whole numbers; bytes wrap around)
        return (a.astype(np.int64) @ b.astype(np.int64)).astype(dtype)

    def launch(a, b, out, rows, cols):
        p.launch([a, b, out], rows=rows, cols=cols, dim=k)
        return out.to_numpy().reshape(rows, cols)

    for _ in range(3):
        dx, dw = S.DeviceArray.from_numpy(x), S.DeviceArray.from_numpy(w)
        assert np.array_equal(launch(dx, dw, dx, m, k), matmul(x, w))
        dx, dw = S.DeviceArray.from_numpy(np.ascontiguousarray(x.T)), S.DeviceArray.from_numpy(w)
        assert np.array_equal(launch(dw, dx, dx, k, m), matmul(w, x.T))
        assert np.array_equal(launch(dw, dw, dw, k, k), matmul(w, w))
