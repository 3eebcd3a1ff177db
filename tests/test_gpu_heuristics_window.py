"""Heuristic resolution against the oracle, bit for bit, where the kernel's
tiles, windows and lists can go wrong: curves that leave a tile's window (8
rows, 16 columns around a 64x16 tile) before they end or reach the walk's 31
steps, crossings on tile borders and corners, tiles full of crossings, graphs
whose links no neighbour returns or that point outside, rows that TMA can and
cannot load; the reference's tests and the vote; with labels in the frame path
and the tile queue."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

DI = (-1, 0, 1, -1, 1, -1, 0, 1)
DJ = (1, 1, 1, 0, 0, -1, -1, -1)
SIZES = [(1, 1), (2, 2), (64, 16), (65, 17), (63, 40), (160, 96), (161, 97), (320, 50)]


def curves(rng, w, h):
    """Crossings whose four arms are curves of 0 to 40 links."""
    g = np.zeros((h, w), np.uint8)
    for _ in range(max(1, w * h // 500)):
        if w < 2 or h < 2:
            break
        i, j = int(rng.integers(0, w - 1)), int(rng.integers(0, h - 1))
        if rng.random() < 0.5:  # at a tile's corner
            i, j = min((i // 64) * 64 + 63, w - 2), min((j // 16) * 16 + 15, h - 2)
        for (x, y, e) in ((i, j, 5), (i + 1, j + 1, 2), (i + 1, j, 7), (i, j + 1, 0)):
            g[y, x] |= 1 << (7 - e)
            for _ in range(int(rng.integers(0, 41))):
                nx, ny = x + DI[e], y + DJ[e]
                if not (0 <= nx < w and 0 <= ny < h):
                    break
                g[y, x] |= 1 << e
                g[ny, nx] |= 1 << (7 - e)
                x, y = nx, ny
                if rng.random() < 0.1:
                    e = int(rng.choice((e, (0, 1, 2, 4, 7, 6, 5, 3)[((0, 1, 2, 4, 7, 6, 5, 3).index(e) + 1) % 8])))
    return g


def dense(rng, w, h):
    """All diagonals of most blocks: crossings everywhere."""
    g = np.zeros((h, w), np.uint8)
    for e in (0, 2):
        for y in range(h - 1):
            for x in range(max(0, -DI[e]), w - max(0, DI[e])):
                if rng.random() < 0.9:
                    g[y, x] |= 1 << e
                    g[y + 1, x + DI[e]] |= 1 << (7 - e)
    return g


def bytes_(rng, w, h):
    return rng.integers(0, 256, size=(h, w)).astype(np.uint8)


@pytest.mark.parametrize("vote", [False, True])
@pytest.mark.parametrize("make", [curves, dense, bytes_])
def test_heuristics(cuda, make, vote):
    import depix
    torch = cuda
    rng = np.random.default_rng([len(make.__name__), vote])
    for w, h in SIZES:
        for rep in range(3):
            g = make(rng, w, h)
            want = O.heuristics(g, w, h, vote)
            d = torch.from_numpy(g.reshape(-1).copy()).cuda()
            out = torch.zeros_like(d)
            depix.resolve_heuristics(d, w, h, out, vote=vote)
            assert np.array_equal(out.cpu().numpy(), want), (w, h, rep)
            if not vote:
                assert depix.lib().depix_resolve_heuristics_static(depix.ptr(d), w, h, depix.stream_ptr()) == 0
                assert np.array_equal(d.cpu().numpy(), want), (w, h, rep)


def lines(rng, w, h):
    """A dark image with crossing one-pixel diagonals and dithered areas."""
    img = np.zeros((h, w, 4), np.uint8)
    img[..., 3] = 255
    for _ in range(max(2, w * h // 300)):
        x, y, dx, dy = int(rng.integers(0, w)), int(rng.integers(0, h)), *(int(v) for v in rng.choice((-1, 1), size=2))
        col = rng.integers(0, 256, size=3)
        for _ in range(int(rng.integers(2, 50))):
            if 0 <= x < w and 0 <= y < h:
                img[y, x, :3] = col
            x, y = x + dx, y + dy
    yy, xx = np.mgrid[0:h, 0:w]
    img[((xx + yy) & 1 == 0) & (xx > 2 * w // 3)] = (200, 40, 90, 255)
    return img


@pytest.mark.parametrize("vote", [False, True])
def test_frames_with_labels(cuda, vote):
    import depix
    torch = cuda
    rng = np.random.default_rng(7 + vote)
    p = depix.params(48, 7, 6, True, 2, vote=vote)
    imgs = [lines(rng, w, h) for w, h in SIZES]
    refs = []
    for img in imgs:
        h, w = img.shape[:2]
        ws = (3 * w + 3) & ~3
        buf = np.zeros((h, ws), np.uint8)
        buf[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
        res = O.graph(buf.reshape(-1), w, h, ws, vote=vote)[2]
        refs.append((res, O.label_cc(res, w, h)))
        ctx = depix.Context(w * h, 1)
        g = torch.zeros(w * h, dtype=torch.uint8, device="cuda")
        lab = torch.zeros(w * h, dtype=torch.int32, device="cuda")
        ctx.frame(torch.from_numpy(img.reshape(-1).copy()).cuda(), w, h, 4 * w, depix.LAYOUT_RGBA, p, None, g, lab)
        assert np.array_equal(g.cpu().numpy(), res), (w, h)
        assert np.array_equal(lab.cpu().numpy(), refs[-1][1]), (w, h)
        ctx.close()
    sizes = [(i.shape[1], i.shape[0]) for i in imgs]
    io = np.concatenate([[0], np.cumsum([(4 * w * h + 15) // 16 * 16 for w, h in sizes])])
    oo = np.concatenate([[0], np.cumsum([16 * w * h for w, h in sizes])])
    buf = np.zeros(int(io[-1]), np.uint8)
    for k, img in enumerate(imgs):
        buf[io[k]:io[k] + img.size] = img.reshape(-1)
    ctx = depix.Context(max(w * h for w, h in sizes), len(sizes))
    lab = torch.zeros(sum(w * h for w, h in sizes), dtype=torch.int32, device="cuda")
    ctx.batch([w for w, _ in sizes], [h for _, h in sizes], io[:-1].astype(np.uint64), oo[:-1].astype(np.uint64),
              torch.from_numpy(buf).cuda(), p, torch.zeros(int(oo[-1]), dtype=torch.uint8, device="cuda"), lab)
    assert np.array_equal(lab.cpu().numpy(), np.concatenate([r[1] for r in refs]))
    ctx.close()


@pytest.mark.parametrize("n", [15, 16, 25, 26])
@pytest.mark.parametrize("vote", [False, True])
def test_threads_by_tiles(cuda, n, vote):
    """Equal batches on both sides of the tile counts at which the blocks change
    their size (48 tiles a frame: 720, 768, 1200 and 1248; one frame above and
    below each), resolved graphs by way of the labels."""
    import depix
    torch = cuda
    w, h = 192, 241
    rng = np.random.default_rng(n)
    imgs = np.stack([lines(rng, w, h) for _ in range(3)])
    want = []
    for img in imgs:
        ws = (3 * w + 3) & ~3
        buf = np.zeros((h, ws), np.uint8)
        buf[:, :3 * w] = img[..., 2::-1].reshape(h, -1)
        want.append(np.asarray(O.label_cc(O.graph(buf.reshape(-1), w, h, ws, vote=vote)[2], w, h)).reshape(-1))
    p = depix.params(48, 7, 6, True, 1, vote=vote)
    ctx = depix.Context(w * h, n)
    d = torch.from_numpy(imgs[np.arange(n) % 3].copy()).cuda()
    out = torch.zeros(n * w * h * 4, dtype=torch.uint8, device="cuda")
    lab = torch.zeros(n * w * h, dtype=torch.int32, device="cuda")
    off = [k * w * h * 4 for k in range(n)]
    ctx.batch([w] * n, [h] * n, off, off, d, p, out, lab)
    got = lab.cpu().numpy().reshape(n, -1)
    for k in range(n):
        assert np.array_equal(got[k], want[k % 3]), k
    ctx.close()
