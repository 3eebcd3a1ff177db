"""Refinement gives the same bits whenever it runs: gradients twice, 200 steps
twice, beside other work on the GPU, from another refiner of another capacity,
and with the steps launched one by one (a caller's capture) instead of replayed."""
import numpy as np
import pytest

import oracle as O
from depix import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,scale", [(24, 24, 2), (37, 61, 5), (256, 224, 4)])
def test_same_bits(cuda, w, h, scale):
    import depix
    torch = cuda
    img = synth.frame(9, w=w, h=h)
    bgr, ws = synth.rgba_to_bgr(img)
    d_img = torch.from_numpy(img.reshape(-1).copy()).cuda()
    d_graph = torch.from_numpy(O.graph(bgr, w, h, ws)[2].copy()).cuda()
    p, rp = depix.params(scale=scale), depix.refine_params(steps=200)

    def refiner(capacity):
        r = depix.Refiner(capacity)
        r.setup(d_img, w, h, 4 * w, depix.LAYOUT_RGBA, d_graph, p, rp)
        return r

    r = refiner(w * h)
    n = r.counts()["nodes"]
    start = torch.empty(2 * n, dtype=torch.float32, device="cuda")
    r.initial(start)
    top = r.export()
    moved = np.random.default_rng(1).normal(0, 0.05, (n, 2)).astype(np.float32)
    moved[top["flags"] & 1 == 1] = 0
    start += torch.from_numpy(moved.reshape(-1)).cuda()

    def gradient():
        g = torch.empty_like(start)
        r.energy_grad(rp, start, g)
        return g

    def positions(rf, run=None):
        pos = start.clone()
        (run or (lambda q: rf.run(rp, q, energies=False)))(pos)
        torch.cuda.synchronize()
        return pos

    g = gradient()
    for _ in range(3):
        assert torch.equal(gradient(), g)
    want = positions(r)
    assert not torch.equal(want, start)
    assert torch.equal(positions(r), want)

    side, other = torch.cuda.Stream(), refiner(w * h)
    a = torch.randn(2048, 2048, device="cuda")
    torch.cuda.synchronize()

    def beside(q):
        noise = start.clone()
        with torch.cuda.stream(side):
            for _ in range(8):
                a @ a
            other.run(rp, noise, stream=side, energies=False)
        r.run(rp, q, energies=False)

    for _ in range(3):
        assert torch.equal(positions(r, beside), want)

    def captured(q):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            r.run(rp, q, stream=torch.cuda.current_stream(), energies=False)
        graph.replay()

    torch.cuda.synchronize()
    assert torch.equal(positions(r, captured), want)
    larger = refiner(3 * w * h)
    assert torch.equal(positions(larger), want)
    for rf in (r, other, larger):
        rf.close()
