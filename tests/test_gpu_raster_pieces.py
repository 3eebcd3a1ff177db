"""The coverage-mask raster on arbitrary resolved graphs against the oracle's
VBO and raster contract, byte for byte: every scale of its three mask layouts,
random graph bytes (links that no neighbour returns, cut polygons that are not
star-shaped and go through the ear clip), images whose edge cells read through
the reference's linear addressing (every row padding, padding bytes that are
not zero, alpha bytes that are not 255), and sizes around the tiles."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# (w, h): one cell, one row, one column, each row padding of the RGBA layout,
# a tile and one cell beside it in either direction
SIZES = [(1, 1), (5, 1), (1, 6), (2, 2), (31, 17), (32, 16), (33, 33), (34, 9), (67, 35)]


def random_graph(rng, w, h, kind):
    """kind 0: any bytes; 1: sparse bytes; 2: symmetric edges, mostly four-linked."""
    if kind == 2:
        g = np.zeros((h, w), np.uint8)
        for e, (di, dj) in enumerate([(-1, 1), (0, 1), (1, 1), (-1, 0)]):
            p = 0.85 if e in (1, 3) else 0.25
            y0, y1, x0, x1 = 0, h - dj, max(0, -di), w - max(0, di)
            if y1 <= y0 or x1 <= x0:
                continue
            m = rng.random((y1 - y0, x1 - x0)) < p
            g[y0:y1, x0:x1] |= (m.astype(np.uint8) << e)
            g[y0 + dj:y1 + dj, x0 + di:x1 + di] |= (m.astype(np.uint8) << (7 - e))
        return g
    g = rng.integers(0, 256, size=(h, w)).astype(np.uint8)
    if kind == 1:
        g &= rng.integers(0, 256, size=(h, w)).astype(np.uint8)
    g[:, 0] &= 0xFF & ~0x29
    g[:, -1] &= 0xFF & ~0x94
    g[0, :] &= 0xFF & ~0xE0
    g[-1, :] &= 0xFF & ~0x07
    return g


@pytest.mark.parametrize("layout", ["rgba", "bgr"])
@pytest.mark.parametrize("scale", range(1, 13))
def test_raster_of_random_graphs(cuda, scale, layout):
    import depix
    torch = cuda
    rng = np.random.default_rng([scale, layout == "bgr"])
    for n, (w, h) in enumerate(SIZES):
        for kind in range(3):
            rgb = rng.integers(0, 3, size=(h, w, 3)).astype(np.uint8) * 90
            g = random_graph(rng, w, h, kind)
            sub = not (n + kind) % 4 == 3
            if layout == "bgr":
                ws = 3 * w + int(rng.integers(0, 6))
                buf = rng.integers(0, 2, size=(h, ws)).astype(np.uint8) * 90
                buf[:, :3 * w] = rgb[..., ::-1].reshape(h, -1)
                ref, ref_ws = buf.reshape(-1), ws
            else:
                ws, ref_ws = 4 * w, (3 * w + 3) & ~3
                buf = np.concatenate([rgb, rng.integers(0, 256, size=(h, w, 1)).astype(np.uint8)], 2)
                ref = np.zeros((h, ref_ws), np.uint8)
                ref[:, :3 * w] = rgb[..., ::-1].reshape(h, -1)
                ref = ref.reshape(-1)
            f = O.frame(ref, w, h, ref_ws, sub, graph_in=g.reshape(-1))
            want = O.raster(f.pos, f.col, w, h, scale)
            d_img = torch.from_numpy(np.ascontiguousarray(buf).reshape(-1)).cuda()
            out = torch.zeros(w * h * scale * scale * 4, dtype=torch.uint8, device="cuda")
            depix.raster(d_img, w, h, ws, depix.LAYOUT_BGR if layout == "bgr" else depix.LAYOUT_RGBA,
                         torch.from_numpy(g.reshape(-1).copy()).cuda(), depix.params(48, 7, 6, sub, scale), out)
            got = out.cpu().numpy().reshape(h * scale, w * scale, 4)
            assert np.array_equal(got, want), (w, h, kind, sub)


@pytest.mark.parametrize("tile", [(32, 32), (32, 16), (16, 16)])
@pytest.mark.parametrize("scale", [1, 3, 4, 5, 7, 8, 9, 12])
def test_queue_tiles_of_every_layout(cuda, scale, tile):
    """Uneven batches through each raster tile, on images of mostly shared
    blocks (a random colour per pixel of three) and flat ones."""
    import depix
    torch = cuda
    rng = np.random.default_rng([scale, *tile])
    sizes = [(1, 1), (33, 31), (16, 17), (40, 64), (64, 33)]
    imgs = [rng.integers(0, 3 if k % 2 else 1, size=(h, w, 4)).astype(np.uint8) * 90 for k, (w, h) in enumerate(sizes)]
    io = np.concatenate([[0], np.cumsum([(4 * w * h + 15) // 16 * 16 for w, h in sizes])])
    oo = np.concatenate([[0], np.cumsum([(4 * w * h * scale * scale + 15) // 16 * 16 for w, h in sizes])])
    buf = np.zeros(int(io[-1]), np.uint8)
    for k, img in enumerate(imgs):
        buf[io[k]:io[k] + img.size] = img.reshape(-1)
    ctx = depix.Context(max(w * h for w, h in sizes), len(sizes))
    ctx.set_launch_shape(2, *tile)
    out = torch.zeros(int(oo[-1]), dtype=torch.uint8, device="cuda")
    ctx.batch([w for w, _ in sizes], [h for _, h in sizes], io[:-1].astype(np.uint64), oo[:-1].astype(np.uint64),
              torch.from_numpy(buf).cuda(), depix.params(48, 7, 6, True, scale), out)
    out = out.cpu().numpy()
    ctx.close()
    for k, (w, h) in enumerate(sizes):
        ws = (3 * w + 3) & ~3
        ref = np.zeros((h, ws), np.uint8)
        ref[:, :3 * w] = imgs[k][..., 2::-1].reshape(h, -1)
        f = O.frame(ref.reshape(-1), w, h, ws, True)
        want = O.raster(f.pos, f.col, w, h, scale)
        assert np.array_equal(out[oo[k]:oo[k] + want.size].reshape(want.shape), want), (w, h)


@pytest.mark.parametrize("scale,size,ns", [(2, (96, 97), (25, 26)), (3, (97, 96), (25, 26)), (4, (96, 97), (25, 26)),
                                           (5, (64, 49), (19, 20)), (8, (64, 49), (19, 20)), (12, (65, 48), (16, 17))])
def test_threads_by_tiles(cuda, scale, size, ns):
    """Equal batches on both sides of the tile counts (304 up to x4, 152 above) at
    which the raster's blocks change their size, widths with and without TMA."""
    import depix
    torch = cuda
    w, h = size
    rng = np.random.default_rng(scale)
    imgs = [rng.integers(0, 3, size=(h, w, 4)).astype(np.uint8) * 90 for _ in range(3)]
    want = []
    for img in imgs:
        ws = (3 * w + 3) & ~3
        ref = np.zeros((h, ws), np.uint8)
        ref[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
        f = O.frame(ref.reshape(-1), w, h, ws, True)
        want.append(O.raster(f.pos, f.col, w, h, scale))
    for n in ns:
        step, ostep = (4 * w * h + 15) // 16 * 16, (4 * w * h * scale * scale + 15) // 16 * 16
        buf = np.zeros((n, step), np.uint8)
        for k in range(n):
            buf[k, :4 * w * h] = imgs[k % 3].reshape(-1)
        out = torch.zeros((n, ostep), dtype=torch.uint8, device="cuda")
        ctx = depix.Context(w * h, n)
        ctx.batch([w] * n, [h] * n, [k * step for k in range(n)], [k * ostep for k in range(n)],
                  torch.from_numpy(buf).cuda(), depix.params(48, 7, 6, True, scale), out)
        got = out.cpu().numpy()[:, :4 * w * h * scale * scale]
        ctx.close()
        for k in range(n):
            assert np.array_equal(got[k].reshape(want[k % 3].shape), want[k % 3]), (n, k)
