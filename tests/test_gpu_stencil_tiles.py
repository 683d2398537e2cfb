"""MapOverlap at the edges of its tiles: whole-number data and weights, so the
sums are exact; both stagings, both paddings, aligned and odd rows."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def expect(img, R, nearest, neutral):
    h, w = img.shape
    p = np.pad(img.astype(np.int64), R, mode="edge") if nearest else \
        np.pad(img.astype(np.int64), R, constant_values=neutral)
    out = np.zeros((h, w), np.int64)
    for dy in range(2 * R + 1):
        for dx in range(2 * R + 1):
            out += (1 + (dy * 3 + dx) % 4) * p[dy:dy + h, dx:dx + w]
    return out


@pytest.mark.parametrize("types", [(np.float32, np.float32), (np.uint8, np.int32), (np.int16, np.float64)])
@pytest.mark.parametrize("nearest,neutral", [(True, 0), (False, 0), (False, 3)])
@pytest.mark.parametrize("R", [1, 4])
def test_stencil_tiles(scl, R, nearest, neutral, types):
    tin, tout = (S.CL_TYPE[np.dtype(t)] for t in types)
    W = 2 * R + 1
    src = (f"{tout} func(input_matrix_t m) {{ {tout} s = 0; for (int dy = -{R}; dy <= {R}; ++dy)"
           f" for (int dx = -{R}; dx <= {R}; ++dx)"
           f" s += ({tout})(1 + ((dy + {R}) * 3 + dx + {R}) % 4) * ({tout})getData(m, dx, dy); return s; }}")
    p = S.Program(S.KIND_MAPOVERLAP, src, [tin, tout], overlap_range=R,
                  padding=S.PAD_NEAREST if nearest else S.PAD_NEUTRAL, neutral=str(neutral))
    rng = np.random.default_rng(R)
    for h, w in ((1, 1), (3, 200), (31, 127), (32, 128), (33, 129), (64, 256), (65, 131), (97, 384), (300, 5)):
        img = rng.integers(0, 9, (h, w)).astype(types[0])
        want = expect(img, R, nearest, neutral)
        # (and one element off 16 bytes: the window by plain loads, no wide store)
        for variant, shift in ((S.VARIANT_AUTO, 0), (S.VARIANT_LDST, 0), (S.VARIANT_AUTO, 1)):
            base = S.DeviceArray.from_numpy(np.concatenate([np.zeros(shift, types[0]), img.ravel()]))
            out = S.DeviceArray(h * w + shift, types[1])
            p.launch([base.view(shift, h * w), out.view(shift, h * w)], rows=h, cols=w,
                     tuning=S.Tuning(variant=variant))
            got = out.to_numpy()[shift:].reshape(h, w)
            assert np.array_equal(got.astype(np.int64), want), (h, w, variant, shift)
