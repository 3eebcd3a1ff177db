"""The roundings of a refinement step that decide where nodes with a gradient
near zero go: Adam over curvature and deviation alone (the coverage weighted by
zero, whose parts are then zeros) against the same float32 operations in numpy,
bit for bit. The fused ones are one rounding of a product and sum that
numpy.longdouble holds exactly, or to 64 bits of which a second rounding decides
once in 2^40."""
import numpy as np
import pytest

import oracle as O
from depix import synth

pytestmark = pytest.mark.gpu

f32, wide = np.float32, np.longdouble


def fma(a, b, c):
    return (wide(a) * np.asarray(b, wide) + np.asarray(c, wide)).astype(f32)


def adam(pos, pos0, free, nbr, rp):
    """rp.steps steps on float32 positions (a free node's neighbours are its two nbr)."""
    b1, b2, one = f32(0.9), f32(0.999), f32(1)
    n = f32(max(free.sum(), 1))
    curv, dev = f32(0.25) * (f32(rp.w_curvature) / n), f32(2) * (f32(rp.w_deviation) / n)
    k = np.nonzero(free)[0]
    a, b = nbr[k, 0], nbr[k, 1]
    m = np.zeros((len(k), 2), f32)
    v = np.zeros((len(k), 2), f32)
    c1 = c2 = 1.0

    def bend(x, at):  # second difference at the nodes `at`, zero where they are pinned
        on = free[at]
        p, q = np.where(on, nbr[at, 0], at), np.where(on, nbr[at, 1], at)
        return np.where(on[:, None], (x[p] - f32(2) * x[at]) + x[q], f32(0))

    x = pos.astype(f32)
    for _ in range(rp.steps):
        c1 *= float(b1)
        c2 *= float(b2)
        g = f32(-2) * ((x[a] - f32(2) * x[k]) + x[b])
        g = g + bend(x, a)
        g = g + bend(x, b)
        g = fma(curv, g, dev * (x[k] - pos0[k]))
        m = fma(one - b1, g, b1 * m)
        v = fma((one - b2) * g, g, b2 * v)
        y = x.copy()
        y[k] = x[k] - f32(rp.lr) * (m / f32(1.0 - c1)) / (np.sqrt(v / f32(1.0 - c2)) + f32(1e-8))
        x = y
    return x


@pytest.mark.parametrize("w,h,steps", [(64, 48, 1), (64, 48, 7), (33, 29, 40)])
def test_steps_without_coverage(cuda, w, h, steps):
    import depix
    torch = cuda
    img = synth.frame(5, w=w, h=h)
    bgr, ws = synth.rgba_to_bgr(img)
    graph = O.graph(bgr, w, h, ws)[2]
    rp = depix.refine_params(w_coverage=0.0, steps=steps)
    r = depix.Refiner(w * h)
    r.setup(torch.from_numpy(img.reshape(-1).copy()).cuda(), w, h, 4 * w, depix.LAYOUT_RGBA,
            torch.from_numpy(graph.copy()).cuda(), depix.params(), rp)
    top = r.export()
    free = (top["flags"] & 1) == 0
    assert free.sum() > 500
    pos0 = (top["q"] / 4).astype(f32)
    start = pos0.copy()
    start[free] += np.random.default_rng(w).normal(0, 0.05, (int(free.sum()), 2)).astype(f32)
    d_pos = torch.from_numpy(start.reshape(-1).copy()).cuda()
    r.run(rp, d_pos, energies=False)
    torch.cuda.synchronize()
    assert np.array_equal(d_pos.cpu().numpy().reshape(-1, 2), adam(start, pos0, free, top["nbr"], rp))
    r.close()
