"""The NEAREST stencil adjoint's edge part and the segmented broadcast, at the
sizes where their launches change shape."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def edge_part(g, w, R):
    """What the clamped reads send to the edge pixels: the transposed stencil
    on the extended matrix, outside positions folded onto their edge pixels."""
    rows, cols = g.shape
    ext = np.zeros((rows + 2 * R, cols + 2 * R))
    for dy in range(-R, R + 1):
        for dx in range(-R, R + 1):
            # position p' takes w(dy, dx) g[p' + (dy, dx)]
            ext[R - dy:R - dy + rows, R - dx:R - dx + cols] += float(w[dy + R, dx + R]) * g
    inside = ext[R:R + rows, R:R + cols].copy()
    iy = np.clip(np.arange(-R, rows + R), 0, rows - 1)
    ix = np.clip(np.arange(-R, cols + R), 0, cols - 1)
    out = np.zeros((rows, cols))
    np.add.at(out, (iy[:, None], ix[None, :]), ext)
    return out - inside


@pytest.mark.parametrize("R", [1, 5, 9, 64])
@pytest.mark.parametrize("shape", [(1, 1), (1, 40), (40, 1), (2, 2), (2, 300), (300, 2), (4, 129), (128, 130), (257, 7)])
def test_stencil_edges(scl, shape, R):
    rng = np.random.default_rng(R)
    W = 2 * R + 1
    g = rng.uniform(-1, 1, shape).astype(np.float32)
    w = rng.uniform(-1, 1, (W, W)).astype(np.float32)
    start = rng.uniform(-1, 1, shape).astype(np.float32)
    dg, dw, out = (S.DeviceArray.from_numpy(a.ravel()) for a in (g, w, start))
    S.check(S.lib().scl_mapoverlap_adjoint_edges(dg.ptr, dw.ptr, out.ptr, shape[0], shape[1], R))
    want = edge_part(g.astype(np.float64), w, R) + start
    # every product and every addition, of at most (R + 1)^2 outside positions
    # times W^2 taps, rounds once
    size = edge_part(np.abs(g).astype(np.float64), np.abs(w), R) + np.abs(start)
    assert np.all(np.abs(out.to_numpy().reshape(shape) - want) <= (2 * W * W + 2 * R) * 2.0 ** -24 * size)


@pytest.mark.parametrize("dtype,code", [(np.float32, S.DTYPE_F32), (np.float64, S.DTYPE_F64)])
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("lens", ["ones", "mixed", "long", "chunk", "one_long"])
def test_broadcast_segments(scl, lens, shift, dtype, code):
    """Elements before the first and past the last segment stay as they are."""
    rng = np.random.default_rng(4)
    ls = {"ones": np.ones(20_000, int), "mixed": rng.integers(0, 9, 20_000), "long": np.array([0, 50_000, 0, 3, 0]),
          "chunk": np.array([8160, 4064, 1, 8159, 8161, 4063, 0, 0, 0, 4065]),
          "one_long": np.concatenate([[30_000], rng.integers(0, 3, 3000), [8160 * 3], np.ones(900, int)])}[lens]
    off = (np.concatenate([[0], np.cumsum(ls)]) + 5).astype(np.uint64)
    n = int(off[-1]) + 7
    g = rng.uniform(-1, 1, len(ls)).astype(dtype)
    old = rng.uniform(-1, 1, n + shift).astype(dtype)
    dg, doff = S.DeviceArray.from_numpy(g), S.DeviceArray.from_numpy(off)
    for acc in (0, 1):
        buf = S.DeviceArray.from_numpy(old)
        gx = buf.view(shift, n)
        S.check(S.lib().scl_adjoint_broadcast_segments(dg.ptr, gx.ptr, doff.ptr, len(ls), n, code, acc))
        want = old.copy()
        lo, hi = shift + 5, shift + n - 7
        want[lo:hi] = np.repeat(g, ls) + (want[lo:hi] if acc else 0)
        assert np.array_equal(buf.to_numpy(), want), acc
