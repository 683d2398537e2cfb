"""AllPairs zip(x*y)/reduce(x+y) on the tensor cores where the sequential FP32
fold is exact: three bf16 parts hold every bit of an operand, so these products
come out bit for bit in every form; and CTA pairs give what the tiles whose
place they take give."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


def program():
    return S.Program(S.KIND_ALLPAIRS, "float func(float x, float y){ return x+y; }", ["float"] * 3,
                     source2="float func(float x, float y){ return x*y; }", identity="0")


def run(p, A, B, **tuning):
    M, K = A.shape
    N = B.shape[1]
    dA, dB, dP = S.DeviceArray.from_numpy(A), S.DeviceArray.from_numpy(B), S.DeviceArray(M * N, np.float32)
    p.launch([dA, dB, dP], rows=M, cols=N, dim=K, tuning=S.Tuning(variant=S.VARIANT_TC3XBF16, **tuning))
    return dP.to_numpy().reshape(M, N)


# by the form that takes them: the fused split, split-K, 128-column tiles, CTA
# pairs for two waves of them, CTA pairs for 256-column tiles (one tile to a
# pair, several to a pair), 256-column tiles
SHAPES = [(300, 100, 400), (600, 700, 500), (1500, 300, 1500), (2000, 200, 2000), (2560, 2600, 2048),
          (2560, 200, 2560), (1, 300, 40000)]


@pytest.mark.parametrize("shape", SHAPES)
def test_one_hot_operand(scl, orc, shape):
    """A row or column of B selected by a one-hot operand: its own bits."""
    M, K, N = shape
    rng = np.random.default_rng(M)
    pick = rng.integers(0, K, max(M, N))
    x = orc.normal_f32(K * max(M, N), 3)
    B = x[:K * N].reshape(K, N)
    A = np.zeros((M, K), np.float32)
    A[np.arange(M), pick[:M]] = 1.0
    p = program()
    assert np.array_equal(run(p, A, B), B[pick[:M]])
    A = x[:M * K].reshape(M, K)
    B = np.zeros((K, N), np.float32)
    B[pick[:N], np.arange(N)] = 1.0
    assert np.array_equal(run(p, A, B), A[:, pick[:N]])


@pytest.mark.parametrize("shape", SHAPES)
def test_whole_numbers(scl, shape):
    """Products of 12-bit whole numbers, one to an output: below 2^24."""
    M, K, N = shape
    rng = np.random.default_rng(N)
    A = np.zeros((M, K), np.float32)
    A[np.arange(M), rng.integers(0, K, M)] = rng.choice([4095, 4093, 4091, 2047], M)
    B = rng.integers(3000, 4096, (K, N)).astype(np.float32)
    assert np.array_equal(run(program(), A, B), (A.astype(np.float64) @ B.astype(np.float64)).astype(np.float32))


# sizes on both sides of the rules that choose between the two
@pytest.mark.parametrize("shape", [(2560, 16, 2048), (2560, 48, 2560), (8200, 130, 1281), (300, 256, 20000),
                                   (300, 257, 20000), (100, 128, 39000), (99, 128, 39000), (128, 129, 39000),
                                   (1100, 512, 20000), (640, 300, 7936), (2600, 2560, 2600), (2600, 2561, 2600),
                                   (20000, 70, 40)])
def test_pairs_same_bits_as_wide_tiles(scl, orc, shape):
    M, K, N = shape
    A = orc.normal_f32(M * K, 61).reshape(M, K)
    B = orc.normal_f32(K * N, 62).reshape(K, N)
    A[M - 1, 0] = np.inf
    A[M // 2, K // 2] = 2.0 ** -100
    B[K - 1, N - 1] = np.nan
    p = program()
    assert np.array_equal(run(p, A, B, tile_h=256), run(p, A, B, tile_h=256, items=3), equal_nan=True)
