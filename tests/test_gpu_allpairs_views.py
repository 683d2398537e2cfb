"""AllPairs zip(x*y)/reduce(x+y) on the tensor cores into and out of views that
start at any element, in every form of the kernel."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def program():
    return S.Program(S.KIND_ALLPAIRS, "float func(float x, float y){ return x+y; }", ["float"] * 3,
                     source2="float func(float x, float y){ return x*y; }", identity="0")


# M x N and K by which form takes them with no tuning: the fused split, split-K,
# 128-column tiles, CTA pairs for two waves of those, 256-column tiles
SHAPES = [(2100, 64, 8), (2100, 64, 36), (300, 64, 260), (600, 1000, 260), (4096, 600, 8), (12800, 300, 36),
          (6600, 300, 260), (20000, 64, 260), (20000, 40, 260)]


@pytest.mark.parametrize("tuning", [{}, {"tile_h": 128}, {"tile_h": 256}, {"tile_h": 256, "items": 3},
                                    {"tile_h": 256, "items": 2}])
@pytest.mark.parametrize("shape", SHAPES)
def test_unaligned_outputs(scl, orc, shape, tuning):
    """Whole numbers: every product and sum is exact."""
    M, K, N = shape
    rng = np.random.default_rng(5)
    a, b = (rng.integers(-8, 9, n + 1).astype(np.float32) for n in (M * K, K * N))
    want = a[1:].reshape(M, K) @ b[1:].reshape(K, N)
    dA, dB = S.DeviceArray.from_numpy(a), S.DeviceArray.from_numpy(b)
    p = program()
    for shift in (0, 1, 2, 3):
        out = S.DeviceArray.from_numpy(np.full(M * N + 4, 7, np.float32))
        p.launch([dA.view(1, M * K), dB.view(1, K * N), out.view(shift, M * N)], rows=M, cols=N, dim=K,
                 tuning=S.Tuning(variant=S.VARIANT_TC3XBF16, **tuning))
        got = out.to_numpy()
        assert np.array_equal(got[shift:shift + M * N].reshape(M, N), want), shift
        assert np.all(got[:shift] == 7) and np.all(got[shift + M * N:] == 7), shift
