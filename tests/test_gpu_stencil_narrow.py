"""MapOverlap of matrices narrower or shorter than a window, whose rows no tile
copy takes: most of a window lies outside.  Whole numbers, so sums are exact."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.uint8])
@pytest.mark.parametrize("nearest", [True, False])
@pytest.mark.parametrize("R", [1, 3])
def test_narrow(scl, R, nearest, dtype):
    t = S.CL_TYPE[np.dtype(dtype)]
    src = (f"int func(input_matrix_t m) {{ int s = 0; for (int dy = -{R}; dy <= {R}; ++dy)"
           f" for (int dx = -{R}; dx <= {R}; ++dx) s += (1 + (dy + {R}) * 11 + dx + {R}) * (int)getData(m, dx, dy);"
           " return s; }")
    p = S.Program(S.KIND_MAPOVERLAP, src, [t, "int"], overlap_range=R,
                  padding=S.PAD_NEAREST if nearest else S.PAD_NEUTRAL, neutral="7")
    rng = np.random.default_rng(R)
    for h, w in ((1, 1), (2, 3), (70, 1), (70, 7), (200, 33), (1, 333), (3, 129), (67, 131)):
        img = rng.integers(0, 100, (h, w)).astype(dtype)
        pad = np.pad(img.astype(np.int64), R, **({"mode": "edge"} if nearest else {"constant_values": 7}))
        want = sum((1 + dy * 11 + dx) * pad[dy:dy + h, dx:dx + w] for dy in range(2 * R + 1) for dx in range(2 * R + 1))
        for shift in (0, 1):
            base = S.DeviceArray.from_numpy(np.concatenate([np.zeros(shift, dtype), img.ravel()]))
            out = S.DeviceArray(h * w, np.int32)
            p.launch([base.view(shift, h * w), out], rows=h, cols=w, tuning=S.Tuning(variant=S.VARIANT_LDST))
            assert np.array_equal(out.to_numpy().reshape(h, w), want), (h, w, shift)
