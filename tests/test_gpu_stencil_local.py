"""MapOverlap whose Local arguments leave the tile's outputs no room in shared
memory."""
import numpy as np
import pytest

import skelcl_gb300 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("local_kb", [4, 190, 200, 215])
def test_wide_outputs_beside_local(scl, local_kb):
    """Bytes to doubles: a window of 34 x 160 bytes, outputs of 32 x 128 x 8 (an
    odd row length: not by TMA)."""
    rows, cols = 100, 301
    img = (np.arange(rows * cols) % 251).astype(np.uint8).reshape(rows, cols)
    src = ("double func(input_matrix_t m, __local int* t) {"
           " t[get_local_id(1) * 32 + get_local_id(0)] = 1;"
           " return getData(m, 1, -1) + 0.5 * getData(m, -1, 1); }")
    p = S.Program(S.KIND_MAPOVERLAP, src, ["unsigned char", "double"], overlap_range=1, padding=S.PAD_NEAREST)
    din, dout = S.DeviceArray.from_numpy(img), S.DeviceArray(rows * cols, np.float64)
    p.launch([din, dout], rows=rows, cols=cols, extra=S.local(local_kb * 1024))

    def at(dx, dy):
        return img[np.clip(np.arange(rows) + dy, 0, rows - 1)][:, np.clip(np.arange(cols) + dx, 0, cols - 1)]
    assert np.array_equal(dout.to_numpy().reshape(rows, cols), at(1, -1) + 0.5 * at(-1, 1))
