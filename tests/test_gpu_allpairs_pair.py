"""AllPairs zip(x*y)/reduce(x+y) on the tensor cores: 256-column tiles on CTA
pairs with FP16 parts and the bf16 parts the device falls back to, and
128-column tiles shared by the blocks of a cluster."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu

# |error| <= C * (|A| |B|), per output: 2^-21 for the split (23 bits of either
# operand, the lo*lo product dropped), and the four full-size accumulations
# of a 64-wide drain at up to two units of 2^-23 each
C = 2.0 ** -21 + 8 * 2.0 ** -23


def program():
    return S.Program(S.KIND_ALLPAIRS, "float func(float x, float y){ return x+y; }", ["float"] * 3,
                     source2="float func(float x, float y){ return x*y; }", identity="0")


def run(p, A, B, items=0, flags=0, cols=256):
    M, K = A.shape
    N = B.shape[1]
    a = np.ascontiguousarray(A.T if flags & S.SHAPE_TRANS_LEFT else A)
    b = np.ascontiguousarray(B.T if flags & S.SHAPE_TRANS_RIGHT else B)
    dA, dB, dP = S.DeviceArray.from_numpy(a), S.DeviceArray.from_numpy(b), S.DeviceArray(M * N, np.float32)
    p.launch([dA, dB, dP], rows=M, cols=N, dim=K, flags=flags,
             tuning=S.Tuning(variant=S.VARIANT_TC3XBF16, items=items, tile_h=cols))
    return dP.to_numpy().reshape(M, N)


@pytest.mark.parametrize("flags", [0, S.SHAPE_TRANS_LEFT, S.SHAPE_TRANS_RIGHT])
@pytest.mark.parametrize("shape", [(255, 47, 257), (128, 48, 256), (256, 64, 512), (257, 65, 129), (129, 127, 255),
                                   (384, 128, 300), (130, 129, 1027), (1000, 520, 513)])
def test_pair_against_fp64(scl, orc, shape, flags):
    M, K, N = shape
    A = orc.normal_f32(M * K, 41).reshape(M, K)
    B = orc.normal_f32(K * N, 42).reshape(K, N)
    P = run(program(), A, B, flags=flags).astype(np.float64)
    bound = C * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64))
    assert np.all(np.abs(P - A.astype(np.float64) @ B.astype(np.float64)) <= bound)


# more tiles than a GPU holds pairs: each pair walks over several
@pytest.mark.parametrize("shape", [(2300, 48, 2600), (2500, 130, 2305), (2561, 500, 2048), (4600, 1000, 4370),
                                   (4100, 1100, 1300)])
def test_pair_walk_against_fp64(scl, orc, shape):
    M, K, N = shape
    A = orc.normal_f32(M * K, 81).reshape(M, K)
    B = orc.normal_f32(K * N, 82).reshape(K, N)
    p = program()
    P = run(p, A, B)
    bound = C * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64))
    assert np.all(np.abs(P - A.astype(np.float64) @ B.astype(np.float64)) <= bound)
    A[M - 1, 3] = np.inf  # bf16 parts
    assert np.array_equal(run(p, A, B), run(p, A, B, items=3), equal_nan=True)


# 128-column tiles in two waves, CTA pairs in one
@pytest.mark.parametrize("flags", [0, S.SHAPE_TRANS_LEFT, S.SHAPE_TRANS_RIGHT])
@pytest.mark.parametrize("shape", [(2000, 16, 2000), (2050, 64, 2047), (1665, 130, 1700), (2431, 65, 1537),
                                   (257, 500, 9000), (2000, 1001, 1930)])
def test_bf16_pairs_same_bits_as_small_tiles(scl, orc, shape, flags):
    M, K, N = shape
    A = orc.normal_f32(M * K, 91).reshape(M, K)
    A[M - 1, 0] = np.inf
    A[M // 2, K // 2] = 2.0 ** -100
    B = orc.normal_f32(K * N, 92).reshape(K, N)
    p = program()
    assert np.array_equal(run(p, A, B, flags=flags, cols=0), run(p, A, B, flags=flags, cols=128), equal_nan=True)


# one wave, few k-blocks: the operands split in the contraction itself
@pytest.mark.parametrize("flags", [0, S.SHAPE_TRANS_LEFT, S.SHAPE_TRANS_RIGHT,
                                   S.SHAPE_TRANS_LEFT | S.SHAPE_TRANS_RIGHT])
@pytest.mark.parametrize("shape", [(128, 16, 128), (129, 63, 131), (300, 64, 301), (130, 65, 1029), (1400, 128, 1401),
                                   (500, 190, 600), (1, 17, 16400), (257, 256, 384), (1000, 500, 1100),
                                   (512, 1000, 640)])
def test_fused_split_same_bits(scl, orc, shape, flags):
    M, K, N = shape
    A = orc.normal_f32(M * K, 95).reshape(M, K)
    A[M - 1, 0] = np.inf
    A[M // 2, K // 2] = 2.0 ** -100
    B = orc.normal_f32(K * N, 96).reshape(K, N)
    B[K - 1, N - 1] = np.nan
    p = program()
    assert np.array_equal(run(p, A, B, flags=flags, cols=0), run(p, A, B, flags=flags, cols=128), equal_nan=True)


def test_fused_split_unaligned_operands(scl, orc):
    M, K, N = 200, 64, 260
    a, b = orc.normal_f32(M * K + 1, 97), orc.normal_f32(K * N + 1, 98)
    p, out = program(), []
    for cols in (0, 128):
        dA, dB, dP = S.DeviceArray.from_numpy(a), S.DeviceArray.from_numpy(b), S.DeviceArray(M * N, np.float32)
        p.launch([dA.view(1, M * K), dB.view(1, K * N), dP], rows=M, cols=N, dim=K, flags=S.SHAPE_TRANS_RIGHT,
                 tuning=S.Tuning(variant=S.VARIANT_TC3XBF16, tile_h=cols))
        out.append(dP.to_numpy())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("exp", [-10, -26, -27, -30, -45, -70])
def test_pair_small_elements(scl, exp):
    """A small element of A that meets the only non-zero element of B's column
    keeps its own precision: FP16 parts while they hold it, bf16 parts below."""
    M, K, N = 256, 128, 256
    small = np.float32((1 + 0x2a5a5b / 2.0 ** 23) * 2.0 ** exp)
    A = np.full((M, K), 1.75, np.float32)
    A[:, 77] = small
    B = np.zeros((K, N), np.float32)
    B[77] = 1.5
    P = run(program(), A, B).astype(np.float64)
    assert np.all(np.abs(P / (np.float64(small) * 1.5) - 1) <= C)


@pytest.mark.parametrize("what", ["inf", "nan", "huge", "tiny", "small_times_zero"])
def test_pair_falls_back_to_bf16_parts(scl, orc, what):
    """Operands that FP16 parts do not hold give what the six bf16 products
    give, bit for bit; a call after them on other operands is not affected."""
    M, K, N = 300, 200, 520
    A0 = orc.normal_f32(M * K, 51).reshape(M, K)
    B = orc.normal_f32(K * N, 52).reshape(K, N)
    p = program()
    clean = run(p, A0, B)
    A = A0.copy()
    if what == "inf":
        A[17, 5] = np.inf
    elif what == "nan":
        A[299, 199] = np.nan
    elif what == "huge":
        A[3, :] *= np.float32(2.0 ** 60)
    elif what == "tiny":
        A[4, 128:] *= np.float32(2.0 ** -60)
    else:
        A[8, 130] = np.float32(2.0 ** -40)
        B = B.copy()
        B[129:, 9] = 0.0
    P = run(p, A, B)
    assert np.array_equal(P, run(p, A, B, items=3), equal_nan=True)
    if what != "small_times_zero":
        assert np.array_equal(run(p, A0, B), clean)


@pytest.mark.parametrize("shape", [(300, 200, 520), (300, 137, 520), (130, 53, 300)])
@pytest.mark.parametrize("zeros", [1, 10, 80, 100])
def test_pair_tiny_elements_beside_zeros(scl, orc, zeros, shape):
    """Tiny elements on one side, zeros (`zeros` of 128 per column) on the
    other: as exact as without them, whichever parts the launch takes."""
    M, K, N = shape
    A = orc.normal_f32(M * K, 55).reshape(M, K)
    B = orc.normal_f32(K * N, 56).reshape(K, N)
    rng = np.random.default_rng(zeros)
    A[rng.integers(0, M, 40), rng.integers(0, K, 40)] = 2.0 ** -40
    A[:, 7] *= np.float32(2.0 ** -33)
    B[rng.permuted(np.tile(np.arange(K)[:, None], (1, N)), axis=0) % 128 < zeros] = 0.0
    for a, b in ((A, B), (np.ascontiguousarray(B.T), np.ascontiguousarray(A.T))):
        P = run(program(), a, b).astype(np.float64)
        bound = C * (np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64))
        assert np.all(np.abs(P - a.astype(np.float64) @ b.astype(np.float64)) <= bound)


def test_pair_in_a_graph(scl, orc):
    """A recorded launch decides for each replay's operands by itself."""
    import ctypes

    M, K, N = 256, 96, 512
    A = orc.normal_f32(M * K, 61).reshape(M, K)
    B = orc.normal_f32(K * N, 62).reshape(K, N)
    odd = A.copy()
    odd[0, 0] = np.inf
    p = program()
    dA, dB, dP = S.DeviceArray.from_numpy(A), S.DeviceArray.from_numpy(B), S.DeviceArray(M * N, np.float32)

    def launch():
        p.launch([dA, dB, dP], rows=M, cols=N, dim=K, tuning=S.Tuning(variant=S.VARIANT_TC3XBF16, tile_h=256))
        return dP

    want = launch().to_numpy()
    dA.upload(odd)
    want_odd = launch().to_numpy()
    L, g = S.lib(), ctypes.c_void_p()
    S.check(L.scl_graph_begin())
    launch()
    S.check(L.scl_graph_end(ctypes.byref(g)))
    for a, ref in ((A, want), (odd, want_odd), (A, want)):
        dA.upload(a)
        S.check(L.scl_graph_launch(g))
        assert np.array_equal(dP.to_numpy(), ref, equal_nan=True)
    S.check(L.scl_graph_destroy(g))


@pytest.mark.parametrize("flags", [0, S.SHAPE_TRANS_LEFT, S.SHAPE_TRANS_RIGHT])
@pytest.mark.parametrize("shape", [(128, 448, 128), (128, 512, 128), (127, 640, 131), (130, 1024, 129), (257, 1000, 72),
                                   (300, 2100, 258), (1000, 500, 1100), (640, 2100, 500)])
def test_split_k_against_fp64(scl, orc, shape, flags):
    """One, two, four and eight blocks to a tile; their k-blocks shared out
    evenly and unevenly."""
    M, K, N = shape
    A = orc.normal_f32(M * K, 71).reshape(M, K)
    B = orc.normal_f32(K * N, 72).reshape(K, N)
    p = program()
    P = run(p, A, B, flags=flags, cols=128)
    bound = C * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64))
    assert np.all(np.abs(P - A.astype(np.float64) @ B.astype(np.float64)) <= bound)
    assert np.array_equal(P, run(p, A, B, flags=flags, cols=128))  # summed in one order
