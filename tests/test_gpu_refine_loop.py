"""The captured Adam loop of a refiner that goes from frame to frame: one
capture serves frames whose counts move to and fro, whichever loop runs gives
the bits that a refiner of the frame's own gives, and a call with other steps
or weights does not run the old loop."""
import numpy as np
import pytest

import oracle as O
from depix import synth

pytestmark = pytest.mark.gpu

W, H = 160, 120


def frames(shares):
    """One picture, flat beyond a share of its rows."""
    full = synth.frame(3, w=W, h=H)
    out = []
    for s in shares:
        img = full.copy()
        img[int(H * s):] = img[0, 0]
        out.append(img)
    return out


def refine(torch, rf, img, rp):
    import depix
    bgr, ws = synth.rgba_to_bgr(img)
    graph = torch.from_numpy(O.graph(bgr, W, H, ws)[2].copy()).cuda()
    d_img = torch.from_numpy(img.reshape(-1).copy()).cuda()
    rf.setup(d_img, W, H, 4 * W, depix.LAYOUT_RGBA, graph, depix.params(), rp)
    pos = torch.zeros(2 * max(rf.counts()["nodes"], 1), dtype=torch.float32, device="cuda")
    rf.initial(pos)
    rf.run(rp, pos, energies=False)
    torch.cuda.synchronize()
    return pos


def test_one_capture_for_frames_to_and_fro(cuda):
    import depix
    rp = depix.refine_params(steps=20)
    shares = [1.0] + [0.8, 1.0, 0.75, 0.9, 0.6, 0.95, 0.45, 1.0] * 2
    rf = depix.Refiner(W * H)
    got = [refine(cuda, rf, img, rp) for img in frames(shares)]
    assert rf.debug_captures() == 1
    own = {}
    for s, img, pos in zip(shares, frames(shares), got):
        if s not in own:
            alone = depix.Refiner(W * H)
            own[s] = refine(cuda, alone, img, rp)
            alone.close()
        assert cuda.equal(pos, own[s])
    rf.close()


def test_other_parameters_are_captured_again(cuda):
    import depix
    img, = frames([1.0])
    rf = depix.Refiner(W * H)
    seen = 0
    for rp in (depix.refine_params(steps=20), depix.refine_params(steps=7), depix.refine_params(steps=7, lr=0.01),
               depix.refine_params(steps=7, lr=0.01, w_curvature=2.0), depix.refine_params(steps=7, lr=0.01, sigma=0.7)):
        pos = refine(cuda, rf, img, rp)
        seen += 1
        assert rf.debug_captures() == seen
        assert cuda.equal(refine(cuda, rf, img, rp), pos) and rf.debug_captures() == seen
        alone = depix.Refiner(W * H)
        assert cuda.equal(refine(cuda, alone, img, rp), pos)
        alone.close()
    rf.close()


def test_small_frames_after_a_large_one(cuda):
    import depix
    rp = depix.refine_params(steps=20)
    rf = depix.Refiner(W * H)
    for share in (1.0, 0.1, 0.0, 0.3, 1.0):
        img, = frames([share])
        pos = refine(cuda, rf, img, rp)
        alone = depix.Refiner(W * H)
        assert cuda.equal(refine(cuda, alone, img, rp), pos)
        alone.close()
    rf.close()
