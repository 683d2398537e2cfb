"""AllPairs on the CUDA cores: the four output tiles, at their edges and at
remainders of their k-tiles.  The fold runs along k in order, so results equal
the same fold on the CPU bit for bit."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu

NP = {"float": np.float32, "double": np.float64, "int": np.int32, "long": np.int64, "unsigned char": np.uint8,
      "short": np.int16}


def check(orc, left, right, out, zip_expr, M, K, N, extra=None, locals_=""):
    seed = M * 7 + K * 3 + N
    make = lambda n, t, s: (orc.normal_f32(n, s) * np.float32(40)).astype(np.int32).astype(NP[t]) \
        if np.issubdtype(NP[t], np.integer) else orc.normal_f32(n, s).astype(NP[t])
    A, B = make(M * K, left, seed).reshape(M, K), make(K * N, right, seed + 1).reshape(K, N)
    p = S.Program(S.KIND_ALLPAIRS, f"{out} func({out} x, {out} y{locals_}){{ return x+y; }}", [left, right, out],
                  source2=f"{out} func({left} x, {right} y){{ return {zip_expr}; }}", identity="0")
    dA, dB, dP = S.DeviceArray.from_numpy(A), S.DeviceArray.from_numpy(B), S.DeviceArray(M * N, NP[out])
    kw = {} if extra is None else {"extra": extra}
    p.launch([dA, dB, dP], rows=M, cols=N, dim=K, tuning=S.Tuning(variant=S.VARIANT_SIMT), **kw)
    ref = np.zeros((M, N), NP[out])
    for k in range(K):
        x, y = A[:, k:k + 1].astype(NP[out]), B[k:k + 1, :].astype(NP[out])
        ref = ref + (np.abs(x - y) if "fabs" in zip_expr else x * y)
    assert np.array_equal(dP.to_numpy().reshape(M, N), ref)


# 16, 32, 64 and 64 x 128 outputs per block, in this order, on 152 SMs
SHAPES = [(1, 1, 1), (1, 300, 5), (17, 15, 31), (16, 64, 16), (200, 65, 190), (15, 130, 1000),
          (300, 31, 310), (305, 33, 304), (64, 97, 1500),
          (700, 32, 716), (701, 66, 719), (1300, 17, 1301),
          (3776, 16, 3776), (3777, 21, 3713)]


@pytest.mark.parametrize("shape", SHAPES)
def test_float_tiles(scl, orc, shape):
    M, K, N = shape
    check(orc, "float", "float", "float", "fabs(x - y)", M, K, N)


@pytest.mark.parametrize("types", [("double", "double", "double", "fabs(x - y)"), ("long", "long", "long", "x * y"),
                                   ("int", "int", "int", "x * y"), ("unsigned char", "unsigned char", "int", "x * y"),
                                   ("short", "float", "float", "fabs(x - y)"),
                                   ("float", "double", "double", "fabs(x - y)")])
@pytest.mark.parametrize("shape", [(17, 66, 31), (300, 33, 312), (701, 35, 719), (1500, 18, 1490), (2600, 17, 2604)])
def test_other_types(scl, orc, types, shape):
    M, K, N = shape
    check(orc, *types, M, K, N)


@pytest.mark.parametrize("kib", [12, 13, 16, 100, 195])
def test_room_for_local_arguments(scl, orc, kib):
    """Local memory as large as a launch accepts beside any tile."""
    for M, K, N in [(20, 9, 20), (300, 9, 310), (701, 9, 719)]:
        check(orc, "float", "float", "float", "fabs(x - y)", M, K, N, extra=S.local(kib * 1024),
              locals_=", __local float* s")
