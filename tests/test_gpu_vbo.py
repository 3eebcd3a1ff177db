"""The drop-in frame driver's one-pass VBO against the oracle, every slot equal:
frames of one cell to a few blocks of cells with remainders on either side of a
block, images of few colours (cells cut on all sides, polygons of up to sixteen
vertices, cells at the image's edge that read through the linear addressing),
padded rows, with and without subdivision, and with either device buffer left
out."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
CELL = 45
SIZES = [(1, 1), (2, 1), (1, 3), (9, 7), (8, 8), (13, 5), (127, 1), (129, 3), (67, 50)]


@pytest.mark.parametrize("subdivide", [0, 1])
@pytest.mark.parametrize("pad", [0, 5])
@pytest.mark.parametrize("colours", [2, 3, 12])
def test_vbo_matches_oracle(cuda, colours, pad, subdivide):
    import depix
    torch = cuda
    for k, (w, h) in enumerate(SIZES):
        rng = np.random.default_rng(1000 * colours + 100 * pad + 10 * k + subdivide)
        palette = rng.integers(0, 256, size=(colours, 3)).astype(np.uint8)
        ws = 3 * w + pad
        bgr = rng.integers(0, 256, size=(h, ws)).astype(np.uint8)
        bgr[:, :3 * w] = palette[rng.integers(0, colours, size=(h, w))].reshape(h, 3 * w)
        f = O.frame(bgr, w, h, ws, subdivide, (5, 7, 6))
        for with_pos, with_col in ((True, True), (k % 2 == 0, k % 2 == 1)):
            pos = torch.full((w * h * CELL * 2,), 7.0, dtype=torch.float32, device="cuda") if with_pos else None
            col = torch.full((w * h * CELL * 4,), 7, dtype=torch.uint8, device="cuda") if with_col else None
            ec, graph = np.zeros(w * h, np.int32), np.zeros(w * h, np.uint8)
            r = depix.launch_kernel_compat(pos, col, bgr, w, h, ws, ec, graph, subdivide)
            diag = np.ctypeslib.as_array(ctypes.cast(r, ctypes.POINTER(ctypes.c_float)), (w * h * CELL * 2,)).copy()
            ctypes.CDLL(None).free(ctypes.c_void_p(r))
            assert np.array_equal(graph, f.graph), (w, h)
            assert np.array_equal(ec, f.ec), (w, h)
            assert np.array_equal(diag, f.pos), (w, h)
            if with_pos:
                assert np.array_equal(pos.cpu().numpy(), f.pos), (w, h)
            if with_col:
                assert np.array_equal(col.cpu().numpy(), f.col), (w, h)
