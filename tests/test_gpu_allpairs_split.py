"""The split of FP32 operands into bf16 parts ahead of the tensor-core AllPairs:
every part of every row against the same roundings in numpy, at the edges of
its tiles, for operands that take either depth of tile, in every orientation."""
import ctypes

import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def bf16(x):
    """x rounded to bfloat16 (to nearest even), as its upper 16 bits."""
    u = x.view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def parts_of(x, n):
    out = []
    for _ in range(n):
        h = bf16(x)
        out.append(h)
        x = x - (h.astype(np.uint32) << 16).view(np.float32)
    return out


@pytest.mark.parametrize("M,K,N", [(5, 16, 70), (64, 64, 65), (63, 65, 130), (130, 127, 63), (65, 129, 200),
                                   (70, 320, 64), (260, 384, 4), (33000, 1030, 64), (64, 190, 180000)])
@pytest.mark.parametrize("trans", [0, 1, 2, 3])
@pytest.mark.parametrize("parts", [2, 3])
def test_parts(scl, M, K, N, trans, parts):
    if trans == 2 and M * K > 1 << 24:
        pytest.skip("large operands: three orientations")
    rng = np.random.default_rng(M + K)
    A, B = (rng.standard_normal(s, dtype=np.float32) for s in ((M, K), (K, N)))
    dA = S.DeviceArray.from_numpy(np.ascontiguousarray(A.T if trans & 1 else A).ravel())
    dB = S.DeviceArray.from_numpy(np.ascontiguousarray(B.T if trans & 2 else B).ravel())
    need = ctypes.c_size_t(0)
    split = S.lib().scl_debug_allpairs_split
    S.check(split(dA.ptr, dB.ptr, M, N, K, parts, trans, None, 0, ctypes.byref(need)))
    scratch = S.DeviceArray(need.value // 2, np.uint16)
    S.check(split(dA.ptr, dB.ptr, M, N, K, parts, trans, scratch.ptr, need.value, None))
    got = scratch.to_numpy()[(-scratch.ptr % 1024) // 2:]
    Mp, Np, Kp = -(-M // 256) * 256, -(-N // 256) * 256, -(-K // 64) * 64
    a = got[:parts * Mp * Kp].reshape(parts, Mp, Kp)
    b = got[parts * Mp * Kp:parts * (Mp + Np) * Kp].reshape(parts, Np, Kp)
    for planes, x in ((a, A), (b, np.ascontiguousarray(B.T))):
        for p, want in enumerate(parts_of(x, parts)):
            assert np.array_equal(planes[p, :len(x), :K], want), p
            assert not planes[p, :len(x), K:].any(), p
