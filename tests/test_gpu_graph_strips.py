"""The similarity-graph kernels' strips against the oracle, bit for bit: sizes
around the 64-column tiles, the four-column lanes and the strips of 1, 4 and 8
rows; aligned rows (TMA windows), unaligned ones and BGR; thresholds from 0 to
past the byte range; both luma arithmetics; with and without the trivial
removal; through the stage call, the frame path and the tile queue. Colours
are close to one another, so that every field's threshold decides some pairs."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 2), (4, 9), (5, 31), (63, 8), (64, 32), (65, 33), (68, 34), (130, 67), (640, 430), (1500, 1400)]
TR = [(0, 0, 0), (5, 7, 6), (48, 7, 6), (255, 255, 255), (400, 3, 256)]


def image(rng, w, h):
    base = rng.integers(0, 256, size=(1 + h // 6, 1 + w // 6, 3)).repeat(6, 0).repeat(6, 1)[:h, :w]
    img = base + rng.integers(-9, 10, size=(h, w, 3)) * (rng.random((h, w, 1)) < 0.5)
    img[rng.random((h, w)) < 0.1] = rng.integers(0, 256)  # grey levels: zero remainders of the luma sum
    img = np.clip(img, 0, 255).astype(np.uint8)
    return np.concatenate([img, rng.integers(0, 256, size=(h, w, 1)).astype(np.uint8)], 2)


def bgr_of(img, pad=0):
    h, w = img.shape[:2]
    ws = ((3 * w + 3) & ~3) + pad
    buf = np.zeros((h, ws), np.uint8)
    buf[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
    return buf.reshape(-1), ws


@pytest.mark.parametrize("yuv", [0, 1])
@pytest.mark.parametrize("tr", TR)
def test_graph_strips(cuda, tr, yuv):
    import depix
    torch = cuda
    rng = np.random.default_rng([*tr, yuv])
    p = depix.params(*tr, yuv=yuv)
    for w, h in SIZES:
        img = image(rng, w, h)
        buf, ws = bgr_of(img)
        raw, triv = O.graph(buf, w, h, ws, tr=tr, yuv=yuv)[:2]
        for layout in ("rgba", "rgba_unaligned", "bgr"):
            if layout == "bgr":
                src, s, lay = *bgr_of(img, pad=int(rng.integers(0, 5))), depix.LAYOUT_BGR
            else:
                s, lay = 4 * w + (4 if layout == "rgba_unaligned" else 0), depix.LAYOUT_RGBA
                src = np.zeros((h, s), np.uint8)
                src[:, :4 * w] = img.reshape(h, -1)
                src = src.reshape(-1)
            d_img = torch.from_numpy(src).cuda()
            for fuse, want in ((False, raw), (True, triv)):
                out = torch.full((w * h,), 255, dtype=torch.uint8, device="cuda")
                depix.graph(d_img, w, h, s, lay, p, out, fuse_trivial=fuse)
                assert np.array_equal(out.cpu().numpy(), want), (w, h, layout, fuse)


def test_graph_of_uneven_and_even_batches(cuda):
    import depix
    torch = cuda
    rng = np.random.default_rng(3)
    p = depix.params(48, 7, 6, True, 2)
    for sizes in (SIZES[:-2], [(64, 40)] * 3, [(67, 33)] * 3):
        imgs = [image(rng, w, h) for w, h in sizes]
        io = np.concatenate([[0], np.cumsum([(4 * w * h + 15) // 16 * 16 for w, h in sizes])])
        oo = np.concatenate([[0], np.cumsum([16 * w * h for w, h in sizes])])
        buf = np.zeros(int(io[-1]), np.uint8)
        for k, img in enumerate(imgs):
            buf[io[k]:io[k] + img.size] = img.reshape(-1)
        ctx = depix.Context(max(w * h for w, h in sizes), len(sizes))
        out = torch.zeros(int(oo[-1]), dtype=torch.uint8, device="cuda")
        lab = torch.zeros(sum(w * h for w, h in sizes), dtype=torch.int32, device="cuda")
        ctx.batch([w for w, _ in sizes], [h for _, h in sizes], io[:-1].astype(np.uint64), oo[:-1].astype(np.uint64),
                  torch.from_numpy(buf).cuda(), p, out, lab)
        out, lab = out.cpu().numpy(), lab.cpu().numpy()
        ctx.close()
        at = 0
        for k, (img, (w, h)) in enumerate(zip(imgs, sizes)):
            b, ws = bgr_of(img)
            f = O.frame(b, w, h, ws, True)
            assert np.array_equal(out[oo[k]:oo[k] + 16 * w * h].reshape(2 * h, 2 * w, 4), O.raster(f.pos, f.col, w, h, 2))
            assert np.array_equal(lab[at:at + w * h], O.label_cc(f.graph, w, h))
            at += w * h
