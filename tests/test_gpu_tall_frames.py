"""Frames of one or two columns and so many rows that a stage's tiles are about
as many as a grid takes (65,535 rows of tiles): against the oracle, through the
graph stage call, the frame path and a refiner that resolves its own graph."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 262140), (1, 262141), (1, 262144), (2, 131072), (1, 262145), (1, 1048560)])
@pytest.mark.parametrize("layout", ["rgba", "bgr"])
def test_tall_frame(cuda, w, h, layout):
    import depix
    torch = cuda
    rng = np.random.default_rng([w, h])
    img = rng.integers(0, 4, size=(h, w, 1)).astype(np.uint8) * np.uint8(60) + np.zeros((1, 1, 4), np.uint8)
    img[..., 3] = 255
    ws = (3 * w + 3) & ~3
    bgr = np.zeros((h, ws), np.uint8)
    bgr[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
    raw, triv, res = O.graph(bgr.reshape(-1), w, h, ws)[:3]
    p = depix.params(scale=1)
    if layout == "rgba":
        d_img, s, lay = torch.from_numpy(img.reshape(-1).copy()).cuda(), 4 * w, depix.LAYOUT_RGBA
    else:
        d_img, s, lay = torch.from_numpy(bgr.reshape(-1).copy()).cuda(), ws, depix.LAYOUT_BGR
    out = torch.full((w * h,), 255, dtype=torch.uint8, device="cuda")
    for fuse, want in ((False, raw), (True, triv)):
        depix.graph(d_img, w, h, s, lay, p, out, fuse_trivial=fuse)
        assert np.array_equal(out.cpu().numpy(), want)
    ctx = depix.Context(w * h, 1)
    labels = torch.empty(w * h, dtype=torch.int32, device="cuda")
    ctx.frame(d_img, w, h, s, lay, p, None, out, labels)
    assert np.array_equal(out.cpu().numpy(), res)
    assert np.array_equal(labels.cpu().numpy(), O.label_cc(res, w, h))
    ctx.close()


def test_refiner_of_a_tall_frame(cuda):
    import depix
    w, h = 1, 262144
    img = np.full((h, 4), 255, np.uint8)
    img[1000::5000, :3] = 0
    r = depix.Refiner(w * h)
    r.setup(cuda.from_numpy(img.reshape(-1).copy()).cuda(), w, h, 4, depix.LAYOUT_RGBA, None, depix.params(scale=1),
            depix.refine_params())
    assert r.counts()["edges"] > 0
    r.close()
