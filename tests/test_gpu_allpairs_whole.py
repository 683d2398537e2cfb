"""CUDA-core AllPairs of whole numbers where the large tile takes half as many
waves as the one before it (wrapping products and sums are exact)."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left,right,out", [(np.int32, np.int32, np.int32), (np.int32, np.uint8, np.int32)])
@pytest.mark.parametrize("M,N", [(1217, 1216), (1345, 1409), (1536, 1537), (1800, 1793), (705, 2881)])
def test_whole_numbers(scl, M, N, left, right, out):
    tl, tr, to = (S.CL_TYPE[np.dtype(d)] for d in (left, right, out))
    K, rng = 19, np.random.default_rng(M)
    A = rng.integers(0, 200, (M, K)).astype(left) * left(12345)
    B = rng.integers(0, 200, (K, N)).astype(right)
    p = S.Program(S.KIND_ALLPAIRS, f"{to} func({to} x, {to} y){{ return x + y; }}", [tl, tr, to],
                  source2=f"{to} func({tl} x, {tr} y){{ return x * y; }}", identity="0")
    P = S.DeviceArray(M * N, out)
    p.launch([S.DeviceArray.from_numpy(A.ravel()), S.DeviceArray.from_numpy(B.ravel()), P], rows=M, cols=N, dim=K)
    want = (A.astype(np.int64) @ B.astype(np.int64)).astype(out)
    assert np.array_equal(P.to_numpy().reshape(M, N), want)
