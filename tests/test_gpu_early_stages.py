"""Frames one after the other on a stream, whose stages may start while the one
before them ends: every pass's graph, labels and output against the oracle (the
output against the same frame run alone), through one context whose scratch each
pass overwrites. Sizes from one cell to both sides of the size up to which the
stages are launched early, odd widths (rows that start at any byte), with the
passes adjacent, with copies between them, and replayed from a captured graph."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (3, 2), (7, 5), (24, 24), (97, 61), (159, 143), (256, 224), (1024, 512), (1025, 512)]


def image(rng, w, h, kind):
    """0: few colours cell by cell; 1: long stripes; 2: noise."""
    img = np.zeros((h, w, 4), np.uint8)
    y, x = np.mgrid[0:h, 0:w]
    pal = rng.integers(0, 256, size=(4, 3)).astype(np.uint8)
    k = rng.integers(0, 3, size=(h, w)) if kind == 0 else ((x // 3 + y // 2) & 3 if kind == 1 else rng.integers(0, 4, size=(h, w)))
    img[..., :3] = pal[k]
    img[..., 3] = 255
    return img


@pytest.mark.parametrize("how", ["adjacent", "copies", "captured"])
@pytest.mark.parametrize("w,h", SIZES)
def test_frames_in_a_row(cuda, w, h, how):
    import depix
    torch = cuda
    rng = np.random.default_rng([w, h])
    p = depix.params(48, 7, 6, True, 2)
    ctx = depix.Context(w * h, 1)
    ws = (3 * w + 3) & ~3
    imgs, want = [], []
    for kind in range(3):
        img = image(rng, w, h, kind)
        buf = np.zeros((h, ws), np.uint8)
        buf[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
        res = O.graph(buf.reshape(-1), w, h, ws)[2]
        imgs.append(torch.from_numpy(img).cuda())
        out = torch.zeros((2 * h, 2 * w, 4), dtype=torch.uint8, device="cuda")
        ctx.frame(imgs[-1], w, h, 4 * w, depix.LAYOUT_RGBA, p, out)
        torch.cuda.synchronize()
        want.append((res, O.label_cc(res, w, h), out.cpu().numpy()))
    n = 12
    inp = torch.zeros_like(imgs[0])
    outs = [torch.zeros((2 * h, 2 * w, 4), dtype=torch.uint8, device="cuda") for _ in range(n)]
    graphs = [torch.zeros(w * h, dtype=torch.uint8, device="cuda") for _ in range(n)]
    labels = [torch.zeros(w * h, dtype=torch.int32, device="cuda") for _ in range(n)]

    def passes():
        for k in range(n):
            src = imgs[k % 3]
            if how == "copies":
                inp.copy_(src)
                src = inp
            ctx.frame(src, w, h, 4 * w, depix.LAYOUT_RGBA, p, outs[k], graphs[k], labels[k])

    if how == "captured":
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            passes()
        for _ in range(3):
            g.replay()
    else:
        for _ in range(3):
            passes()
    torch.cuda.synchronize()
    for k in range(n):
        res, lab, out = want[k % 3]
        assert np.array_equal(graphs[k].cpu().numpy(), res.reshape(-1)), k
        assert np.array_equal(labels[k].cpu().numpy(), np.asarray(lab).reshape(-1)), k
        assert np.array_equal(outs[k].cpu().numpy(), out), k
    ctx.close()


@pytest.mark.parametrize("scale", [1, 3, 4, 5, 8, 12, 13, None])
def test_labels_with_and_without_a_raster(cuda, scale):
    """The labels' roots, made by the raster up to scale 12 in every layout of its
    masks, beyond it and without an output by a kernel of their own: single frames,
    equal batches and uneven ones in each tile shape."""
    import depix
    torch = cuda
    rng = np.random.default_rng(scale or 99)
    s = scale or 1
    p = depix.params(48, 7, 6, True, s)
    sizes = [(1, 1), (5, 3), (33, 17), (32, 32), (95, 70), (130, 65)]
    want, imgs = [], []
    for k, (w, h) in enumerate(sizes):
        img = image(rng, w, h, k % 3)
        ws = (3 * w + 3) & ~3
        buf = np.zeros((h, ws), np.uint8)
        buf[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
        want.append(np.asarray(O.label_cc(O.graph(buf.reshape(-1), w, h, ws)[2], w, h)).reshape(-1))
        imgs.append(img)
        ctx = depix.Context(w * h, 1)
        d = torch.from_numpy(img).cuda()
        out = torch.zeros(w * h * s * s * 4, dtype=torch.uint8, device="cuda") if scale else None
        lab = torch.full((w * h,), -1, dtype=torch.int32, device="cuda")
        ctx.frame(d, w, h, 4 * w, depix.LAYOUT_RGBA, p, out, None, lab)
        assert np.array_equal(lab.cpu().numpy(), want[-1]), (w, h)
        ctx.close()
    if not scale:
        return
    for order, shapes in (([4] * 3, [None]), (range(len(sizes)), [(32, 32), (32, 16), (16, 16), (0, 0)])):
        ws, hs = [sizes[k][0] for k in order], [sizes[k][1] for k in order]
        io, oo, buf, ob = [], [], [], 0
        for k in order:
            io.append(sum(len(b) for b in buf))
            b = imgs[k].tobytes()
            buf.append(b + bytes(-len(b) % 16))
            oo.append(ob)
            ob += -(-len(b) * s * s // 16) * 16
        d = torch.from_numpy(np.frombuffer(b"".join(buf), np.uint8).copy()).cuda()
        out = torch.zeros(ob, dtype=torch.uint8, device="cuda")
        ctx = depix.Context(max(w * h for w, h in sizes), len(ws))
        for shape in shapes:
            if shape:
                ctx.set_launch_shape(1, *shape)
            lab = torch.full((sum(w * h for w, h in zip(ws, hs)),), -1, dtype=torch.int32, device="cuda")
            ctx.batch(ws, hs, io, oo, d, p, out, lab)
            assert np.array_equal(lab.cpu().numpy(), np.concatenate([want[k] for k in order])), shape
        ctx.close()
