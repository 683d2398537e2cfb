"""The flat Reduce and the fused Zip-Reduce of floats: FP64 carries from the
first few elements of a thread's fold on."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 2048, 2049, 4096, 8192, 16384, 16390, 65536, 300_001, 1 << 20])
@pytest.mark.parametrize("shift", [0, 1])
def test_reduce_rounds_once(scl, n, shift):
    """21-bit whole numbers: single precision holds the sum of any 8 of them,
    and a thread folds at most 8 of one sign, so nothing rounds before the
    result."""
    t = "float"
    add = "float func(float x, float y){ return x + y; }"
    red = S.Program(S.KIND_REDUCE, add, [t], identity="0")
    dot = S.Program(S.KIND_ZIP_REDUCE, add, [t] * 3, source2="float m(float x, float y){ return x * y; }", func2="m",
                    identity="0")
    out = S.DeviceArray(1, np.float32)
    for seed in range(4):
        rng = np.random.default_rng(seed)
        x = rng.integers(1 << 20, 1 << 21, n + shift).astype(np.float32)
        # a sum near zero shows what the folds lost
        x[shift + n // 2:] *= -1
        v = S.DeviceArray.from_numpy(x).view(shift, n)
        one = S.DeviceArray.from_numpy(np.ones(n + shift, np.float32)).view(shift, n)
        want = np.float32(x[shift:].astype(np.float64).sum())
        red.launch([v, out], n=n)
        assert out.to_numpy()[0] == want
        dot.launch([v, one, out], n=n)
        assert out.to_numpy()[0] == want
