"""The refiner's sample assignment against a search over all segments, in whole
numbers with the quotient rounded to double: distance keys that hold the slot
and (a frame of over 2^18 slots at x12) the two passes without it; and the
setup's counts and offsets: every sample once, ascending within its slot."""
import numpy as np
import pytest

from depix import synth

pytestmark = pytest.mark.gpu

WA = np.array([[0, 0, 0], [3, 1, 0], [4, 0, 0], [1, 3, 0], [1, 3, 0]])
WB = np.array([[0, 0, 0], [1, 3, 0], [3, 1, 0], [0, 4, 0], [0, 3, 1]])
BAND2 = 48 * 48


def image(kind, w, h):
    if kind == "frame":
        return synth.frame(w + h, w=w, h=h)
    img = np.random.default_rng(w * h).integers(0, 256, size=(h, w, 4)).astype(np.uint8)
    img[..., 3] = 255
    return img


@pytest.mark.parametrize("kind,w,h,scale", [("frame", 40, 33, 1), ("frame", 61, 47, 4), ("frame", 50, 40, 12),
                                            ("noise", 33, 30, 5), ("noise", 1, 9, 4), ("noise", 300, 260, 12)])
def test_assignment(cuda, kind, w, h, scale):
    import depix
    torch = cuda
    img = image(kind, w, h)
    r = depix.Refiner(w * h)
    p = depix.params(48, 7, 6, True, scale)
    rp = depix.refine_params()
    d_img = torch.from_numpy(np.ascontiguousarray(img).reshape(-1)).cuda()
    for _ in range(2):  # the second setup finds the first one's buffers
        r.setup(d_img, w, h, 4 * w, depix.LAYOUT_RGBA, None, p, rp)
    top = r.export()
    r.close()
    S, ow, oh = len(top["segs"]), w * scale, h * scale
    if kind == "noise" and scale == 12:
        assert S > 1 << 18
    x, slot = top["samples"][:, 0], top["samples"][:, 1]
    assert np.all(np.diff(slot) >= 0) and np.all(np.diff(x)[np.diff(slot) == 0] > 0)
    owner = np.full(ow * oh, -1)
    owner[x] = slot
    assert (owner >= 0).sum() == len(x)  # no sample twice
    live = np.nonzero(top["segs"][:, 3])[0]
    seg = top["segs"][live]
    q = top["q"][np.maximum(seg[:, :3], 0)].astype(np.int64)
    m = 2 * scale
    a, b = ((W[seg[:, 3]][..., None] * q).sum(1) * m for W in (WA, WB))
    a, b, ids = (torch.from_numpy(v).cuda() for v in (a, b, live))
    e = b - a
    L = (e * e).sum(1)
    rng = np.random.default_rng(scale)
    picks = np.concatenate([rng.integers(0, ow * oh, size=400), rng.choice(x, size=min(400, len(x))) if len(x) else x])
    for s in picks.astype(np.int64):
        v = torch.tensor([16 * (2 * (s % ow) + 1), 16 * (2 * (s // ow) + 1)], device="cuda") - a
        dot = (e * v).sum(1)
        cr = e[:, 0] * v[:, 1] - e[:, 1] * v[:, 0]
        u = v - e
        d = torch.where(dot <= 0, (v * v).sum(1).double(), torch.where(dot >= L, (u * u).sum(1).double(),
                                                                       (cr * cr).double() / L.clamp(min=1).double()))
        best = d.min().item() if len(d) else np.inf
        want = int(ids[d == best].min()) if best <= BAND2 else -1
        assert owner[s] == want, (s, best)
