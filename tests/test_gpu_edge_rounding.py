"""The NEAREST stencil adjoint's edge part: sums of many taps that round about
as often as their result does."""
import numpy as np
import pytest

import skelcl_gb300 as S
from test_gpu_adjoint_edges import edge_part

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [5, 9, 20])
@pytest.mark.parametrize("shape", [(400, 300), (12, 2000), (2000, 12)])
def test_edge_rounding(scl, shape, R):
    """Positive taps: the root mean square of the relative error stays below
    2^-24, the largest error of a single rounding."""
    rng = np.random.default_rng(R)
    W = 2 * R + 1
    g, w = rng.uniform(0, 1, shape).astype(np.float32), rng.uniform(0, 1, (W, W)).astype(np.float32)
    dg, dw, out = (S.DeviceArray.from_numpy(a.ravel()) for a in (g, w, np.zeros(shape, np.float32)))
    S.check(S.lib().scl_mapoverlap_adjoint_edges(dg.ptr, dw.ptr, out.ptr, shape[0], shape[1], R))
    want = edge_part(g.astype(np.float64), w, R)
    got = out.to_numpy().reshape(shape).astype(np.float64)
    inner = np.zeros(shape, bool)  # (the four corners are a warp's)
    inner[1:-1, 0] = inner[1:-1, -1] = inner[0, 1:-1] = inner[-1, 1:-1] = True
    assert np.sqrt(np.mean((got[inner] / want[inner] - 1) ** 2)) < 2.0 ** -24
