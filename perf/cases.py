"""The work that users of this library have it do, as cases that can be timed.

A case is a dict of plain values. ``listed()`` names the representative ones,
``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` makes what
a program has in hand before the call (inputs on the GPU, buffers, the context
or refiner it keeps), ``run(state)`` is one pass through the public entry
points, ``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the floating outputs in 64 bits.

Kinds of case:

* ``frame``   -- one frame through ``Context.frame`` (the per-frame drop-in path);
* ``batch``   -- equal-size frames through ``Context.batch``, device resident;
* ``sprites`` -- frames of uneven sizes through ``Context.batch``;
* ``host``    -- a batch from and to pinned host buffers, ``Context.batch_host``;
* ``walks``   -- border walks of resolved graphs, ``depix.border_walks``;
* ``refine``  -- one frame of a stream with refinement: topology setup, warm
                 start from the previous frame, Adam steps;
* ``grad``    -- energy and adjoint at given positions (an outer optimiser's call);
* ``vbo``     -- the reference's own frame driver (host image in, VBO, graph and
                 triangulated points out), ``depix.launch_kernel_compat``.

Images follow the generators of ``depix.synth`` (palette scenes of rectangles
and ellipses with dark outlines, checkerboard dithering, single-pixel noise in
the large frames), drawn here on the GPU so that a thousand distinct frames
take a fraction of a second.
"""
import ctypes
import math
import os
import sys
import weakref

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pixel-art-remaster-gpu_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import depix  # noqa: E402

KINDS = ("frame", "batch", "sprites", "host", "walks", "refine", "grad", "vbo")
LAYOUTS = {"rgba": depix.LAYOUT_RGBA, "bgr": depix.LAYOUT_BGR}
DEV = "cuda"


def listed():
    return [
        # a single sprite as it is loaded or edited: the smallest call, all latency
        dict(name="frame_24x24_x4", kind="frame", w=24, h=24, scale=4, layout="rgba", labels=True, subdivide=True,
             vote=False),
        # the plain path: one console frame at a time, as an emulator hands them over
        dict(name="frame_256x224_x4", kind="frame", w=256, h=224, scale=4, layout="rgba", labels=True,
             subdivide=True, vote=False),
        # a stream in batches of 8 (low latency)
        dict(name="batch_8_256x224_x4", kind="batch", n=8, w=256, h=224, scale=4, labels=True, subdivide=True,
             vote=False, noisy=False),
        # bulk conversion of a video: the headline batch
        dict(name="batch_1024_256x224_x4", kind="batch", n=1024, w=256, h=224, scale=4, labels=True, subdivide=True,
             vote=False, noisy=False),
        # larger noisy frames to print size
        dict(name="batch_16_640x480_x8", kind="batch", n=16, w=640, h=480, scale=8, labels=True, subdivide=True,
             vote=False, noisy=True),
        # handheld captures with a cropped column and row (odd sizes, no
        # 16-byte rows), resolved by the weighted vote, no labels
        dict(name="batch_32_159x143_x3_vote", kind="batch", n=32, w=159, h=143, scale=3, labels=False,
             subdivide=True, vote=True, noisy=False),
        # a game's sprite sheet cut into its sprites: uneven sizes in one call
        dict(name="sprites_4096_x4", kind="sprites", n=4096, lo=8, hi=64, scale=4, labels=True, subdivide=True),
        # frames that live in host memory, results back there
        dict(name="host_64_256x224_x4", kind="host", n=64, w=256, h=224, scale=4, labels=True),
        # spline export of a batch of frames
        dict(name="walks_128_256x224", kind="walks", n=128, w=256, h=224),
        # one frame of the refined stream
        dict(name="refine_256x224_x4_20", kind="refine", w=256, h=224, scale=4, steps=20),
        # the adjoint alone, called by an outer optimiser
        dict(name="grad_256x224_x4", kind="grad", w=256, h=224, scale=4),
        # an existing caller of the reference's frame driver
        dict(name="vbo_256x224", kind="vbo", w=256, h=224, subdivide=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: every kind, sizes log-uniform
    (odd ones as they come), the options that each kind takes."""
    kind = rng.choice(KINDS)
    w, h = _log(rng, 12, 512), _log(rng, 12, 400)
    scale = rng.choice((2, 3, 4, 4, 4, 5, 6, 8, 10, 12))
    c = dict(kind=kind)
    if kind == "frame":
        c |= dict(w=w, h=h, scale=scale, layout=rng.choice(("rgba", "rgba", "bgr")), labels=rng.random() < 0.7,
                  subdivide=rng.random() < 0.8, vote=rng.random() < 0.2)
    elif kind in ("batch", "host"):
        most = (2.0e9 if kind == "batch" else 1.2e8) / (w * h * (8.0 + 4.0 * scale * scale))
        n = max(2, min(_log(rng, 2, 1024 if kind == "batch" else 64), int(most)))
        c |= dict(n=n, w=w, h=h, scale=scale, labels=rng.random() < 0.7)
        if kind == "batch":
            c |= dict(subdivide=rng.random() < 0.85, vote=rng.random() < 0.2, noisy=rng.random() < 0.3)
    elif kind == "sprites":
        hi = rng.randint(24, 64)
        c |= dict(n=_log(rng, 48, 4096), lo=rng.randint(8, 16), hi=hi, scale=rng.choice((2, 3, 4, 4, 5, 6)),
                  labels=rng.random() < 0.7, subdivide=rng.random() < 0.85)
    elif kind == "walks":
        c |= dict(n=_log(rng, 1, 128), w=min(w, 320), h=min(h, 240))
    elif kind in ("refine", "grad"):
        c |= dict(w=max(24, min(w, 320)), h=max(24, min(h, 240)), scale=rng.choice((2, 3, 4, 4, 5, 6)))
        if kind == "refine":
            c |= dict(steps=_log(rng, 5, 200))
    else:
        c |= dict(w=w, h=h, subdivide=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ inputs


def _scenes(rng, ws, hs, W, H, lo_col, hi_col, lo_shapes, hi_shapes, size_hi, outline_p, dither, noise, empty_p=0.0):
    """One scene per entry of ws/hs on W x H canvases: an (n, H, W) int32
    tensor of RGBA8 words (R in the low byte)."""
    n = len(ws)
    ws, hs = np.asarray(ws), np.asarray(hs)
    n_col = rng.integers(lo_col, hi_col + 1, size=n)
    palette = rng.integers(0, 256, size=(n, hi_col, 3)).astype(np.int64)
    n_shapes = rng.integers(lo_shapes, hi_shapes + 1, size=n)
    empty = rng.random(n) < empty_p

    def pick():
        return palette[np.arange(n), rng.integers(0, 1 << 30, size=n) % n_col]

    def words(rgb, alpha=255):
        v = rgb[:, 0] | rgb[:, 1] << 8 | rgb[:, 2] << 16 | alpha << 24
        return torch.from_numpy(v.astype(np.uint32).view(np.int32)).to(DEV)

    bg = pick()
    bg[empty] = 0
    first = np.where(empty, 0, 255)
    img = words(bg, first)[:, None, None].expand(n, H, W).contiguous()
    xs = np.arange(-1, W + 1)[None, :]
    ys = np.arange(-1, H + 1)[None, :]
    for k in range(hi_shapes):
        sw, sh = rng.integers(4, size_hi + 1, size=n), rng.integers(4, size_hi + 1, size=n)
        x0 = rng.integers(0, 1 << 30, size=n) % np.maximum(ws, 1) - sw // 2
        y0 = rng.integers(0, 1 << 30, size=n) % np.maximum(hs, 1) - sh // 2
        ell = rng.random(n) < 0.45
        col = pick()
        outlined = (rng.random(n) < outline_p) | empty
        off = k >= n_shapes

        def profile(c, at, size):
            inside = (c >= at[:, None]) & (c < (at + size)[:, None])
            d = (c - (at + (size - 1) / 2.0)[:, None]) / (size / 2.0)[:, None]
            f = np.where(ell[:, None], d * d, np.where(inside, 0.0, 4.0))
            f[off] = 4.0
            return torch.from_numpy(f.astype(np.float32)).to(DEV)

        fx, fy = profile(xs, x0, sw), profile(ys, y0, sh)
        cx, cy = fx[:, None, 1:-1], fy[:, 1:-1, None]
        mask = cx + cy <= 1.0
        img = torch.where(mask, words(col)[:, None, None], img)
        if outlined.any():
            nx = torch.maximum(fx[:, :-2], fx[:, 2:])[:, None, :]
            ny = torch.maximum(fy[:, :-2], fy[:, 2:])[:, :, None]
            edge = mask & ~((nx + cy <= 1.0) & (cx + ny <= 1.0))
            edge &= torch.from_numpy(outlined).to(DEV)[:, None, None]
            img = torch.where(edge, words(col // 4)[:, None, None], img)
    gx = torch.arange(W, device=DEV)[None, None, :]
    gy = torch.arange(H, device=DEV)[None, :, None]
    checker = ((gx + gy) & 1) == 0
    for _ in range(max(1, int(round(dither * W * H / 342.0)))):
        dw, dh = rng.integers(4, 33, size=n), rng.integers(4, 33, size=n)
        x0 = rng.integers(0, 1 << 30, size=n) % np.maximum(ws - dw, 1)
        y0 = rng.integers(0, 1 << 30, size=n) % np.maximum(hs - dh, 1)
        mx = torch.from_numpy((xs[:, 1:-1] >= x0[:, None]) & (xs[:, 1:-1] < (x0 + dw)[:, None])).to(DEV)[:, None, :]
        my = torch.from_numpy((ys[:, 1:-1] >= y0[:, None]) & (ys[:, 1:-1] < (y0 + dh)[:, None])).to(DEV)[:, :, None]
        img = torch.where(mx & my & checker, words(pick())[:, None, None], img)
    if noise > 0:
        g = torch.Generator(device=DEV)
        g.manual_seed(int(rng.integers(0, 1 << 31)))
        hit = torch.rand((n, H, W), device=DEV, generator=g) < noise
        which = torch.randint(0, int(n_col.min()), (n, H, W), device=DEV, generator=g)
        flat = palette[..., 0] | palette[..., 1] << 8 | palette[..., 2] << 16 | 255 << 24
        pal = torch.from_numpy(flat.astype(np.uint32).view(np.int32)).to(DEV)
        img = torch.where(hit, torch.gather(pal, 1, which.reshape(n, -1)).reshape(n, H, W), img)
    return img


def _frames(rng, n, w, h, noisy=False):
    """n equal-size frames as an (n, h, w) int32 tensor of RGBA8 words: the
    console frame's scene, or the large noisy one's; shapes by the area."""
    share = max(6, int(round((200 if noisy else 70) * w * h / float(640 * 480 if noisy else 256 * 224))))
    out = torch.empty((n, h, w), dtype=torch.int32, device=DEV)
    step = max(1, (1 << 23) // (w * h))
    for a in range(0, n, step):
        m = min(step, n - a)
        out[a:a + m] = _scenes(rng, [w] * m, [h] * m, w, h, 64 if noisy else 16, 64 if noisy else 16, share, share,
                               48, 0.5, 0.10 if noisy else 0.05, 0.02 if noisy else 0.0)
    return out


def _align16(v):
    return (v + 15) // 16 * 16


def _bgr(img):
    """An (h, w) frame of RGBA words in the reference's image layout (host)."""
    px = img.cpu().numpy().view(np.uint8).reshape(img.shape[0], img.shape[1], 4)
    ws = (3 * img.shape[1] + 3) & ~3
    buf = np.zeros((img.shape[0], ws), np.uint8)
    buf[:, :3 * img.shape[1]].reshape(img.shape[0], img.shape[1], 3)[...] = px[..., 2::-1]
    return buf.reshape(-1), ws


def _params(case):
    return depix.params(48, 7, 6, case.get("subdivide", True), case.get("scale", 4), case.get("vote", False))


def _resolved(img, w, h, p):
    """The resolved graph of one device frame (h, w int32 words)."""
    ctx = depix.Context(w * h, 1)
    g = torch.empty(w * h, dtype=torch.uint8, device=DEV)
    ctx.frame(img, w, h, 4 * w, depix.LAYOUT_RGBA, p, None, g, None)
    torch.cuda.synchronize()
    ctx.close()
    return g


def _packed(rng, case):
    """(widths, heights, input offsets, output offsets, input tensor, output
    bytes, pixels) of a batch."""
    s2 = 4 * case["scale"] ** 2
    if case["kind"] == "sprites":
        n, lo, hi = case["n"], case["lo"], case["hi"]
        sheet = np.random.default_rng([0x9A57, n, lo, hi])  # the sizes belong to the case, the pictures to the seed
        ws, hs = sheet.integers(lo, hi + 1, size=n), sheet.integers(lo, hi + 1, size=n)
        px = ws * hs
        io = np.concatenate([[0], np.cumsum(_align16(4 * px))])
        buf = torch.zeros(int(io[-1]) // 4, dtype=torch.int32, device=DEV)
        step = max(1, (1 << 23) // (hi * hi))
        for a in range(0, n, step):
            w, h = ws[a:a + step], hs[a:a + step]
            img = _scenes(rng, w, h, hi, hi, 4, 16, 1, 8, min(48, hi), 0.5, 0.05, 0.0, empty_p=0.3)
            x = torch.arange(hi, device=DEV)[None, None, :]
            y = torch.arange(hi, device=DEV)[None, :, None]
            tw, th = torch.from_numpy(w).to(DEV)[:, None, None], torch.from_numpy(h).to(DEV)[:, None, None]
            at = torch.from_numpy(io[a:a + len(w)] // 4).to(DEV)[:, None, None] + y * tw + x
            ok = (x < tw) & (y < th)
            buf[at[ok]] = img[ok]
    else:
        n, w, h = case["n"], case["w"], case["h"]
        img = _frames(rng, n, w, h, case.get("noisy", False))
        ws, hs, px = np.full(n, w), np.full(n, h), np.full(n, w * h)
        io = np.arange(n + 1) * _align16(4 * w * h)
        buf = torch.zeros((n, int(io[1]) // 4), dtype=torch.int32, device=DEV)
        buf[:, :w * h] = img.reshape(n, -1)
        buf = buf.reshape(-1)
    oo = np.concatenate([[0], np.cumsum(_align16(px * s2))])
    return (ws.astype(np.int32), hs.astype(np.int32), io[:-1].astype(np.uint64), oo[:-1].astype(np.uint64), buf,
            int(oo[-1]), int(px.sum()))


def _refined_pair(rng, w, h):
    """Two consecutive frames of a stream: a background with 24 sprites moved
    by 0-3 pixels in each direction, wrapping around."""
    size = max(8, min(48, w // 2, h // 2))
    sw, sh = rng.integers(8, size + 1, size=24), rng.integers(8, size + 1, size=24)
    sp = _scenes(rng, sw, sh, size, size, 4, 16, 1, 8, size, 0.5, 0.05, 0.0, empty_p=0.3).cpu().numpy()
    bg = _frames(rng, 1, w, h)[0].cpu().numpy()
    at = rng.integers(0, (w, h), size=(24, 2))
    vel = rng.integers(0, 4, size=(24, 2))
    out = []
    for f in (0, 1):
        img = bg.copy()
        for k in range(24):
            s = sp[k, :sh[k], :sw[k]]
            ix = np.ix_((at[k, 1] + vel[k, 1] * f + np.arange(sh[k])) % h, (at[k, 0] + vel[k, 0] * f + np.arange(sw[k])) % w)
            img[ix] = np.where(s < 0, s, img[ix])  # alpha 255: a negative word
        out.append(torch.from_numpy(img).to(DEV))
    return out


def _set_up(img, w, h, p, rp):
    g = _resolved(img, w, h, p)
    r = depix.Refiner(w * h)
    r.setup(img, w, h, 4 * w, depix.LAYOUT_RGBA, g, p, rp)
    return r, g


def _moved(r, pos, seed):
    """Positions some optimiser steps away from r's start: free nodes off by a
    few hundredths of a pixel."""
    r.initial(pos)
    top = r.export()
    n = len(top["flags"])
    step = np.random.default_rng(seed).normal(0.0, 0.05, size=(n, 2)).astype(np.float32)
    step[(top["flags"] & 1) == 1] = 0.0
    pos[:2 * n] += torch.from_numpy(step.reshape(-1)).to(DEV)
    return top


def prepare(case, seed):
    rng = np.random.default_rng([0x9A57, int(seed)])
    kind = case["kind"]
    if kind == "frame":
        w, h, s = case["w"], case["h"], case["scale"]
        img = _frames(rng, 1, w, h)[0]
        ws = 4 * w
        if case["layout"] == "bgr":
            buf, ws = _bgr(img)
            img = torch.from_numpy(buf).to(DEV)
        return dict(kind=kind, ctx=depix.Context(w * h, 1), img=img, w=w, h=h, ws=ws, layout=LAYOUTS[case["layout"]],
                    p=_params(case), out=torch.zeros((h * s, w * s, 4), dtype=torch.uint8, device=DEV),
                    graph=torch.zeros((h, w), dtype=torch.uint8, device=DEV),
                    labels=torch.zeros((h, w), dtype=torch.int32, device=DEV) if case["labels"] else None)
    if kind in ("batch", "sprites", "host"):
        ws, hs, io, oo, buf, out_bytes, px = _packed(rng, case)
        host = dict(pin_memory=True) if kind == "host" else dict(device=DEV)
        if kind == "host":
            buf = torch.empty(buf.shape, dtype=buf.dtype, pin_memory=True).copy_(buf)
        return dict(kind=kind, ctx=depix.Context(int((ws.astype(np.int64) * hs).max()), case["n"]), ws=ws, hs=hs,
                    io=io, oo=oo, img=buf, p=_params(case), out=torch.zeros(out_bytes, dtype=torch.uint8, **host),
                    labels=torch.zeros(px, dtype=torch.int32, **host) if case["labels"] else None)
    if kind == "walks":
        w, h, n = case["w"], case["h"], case["n"]
        imgs = _frames(rng, n, w, h)
        ctx = depix.Context(w * h, 1)
        g = torch.empty((n, w * h), dtype=torch.uint8, device=DEV)
        for k in range(n):
            ctx.frame(imgs[k], w, h, 4 * w, depix.LAYOUT_RGBA, _params(case), None, g[k], None)
        torch.cuda.synchronize()
        most, walks = w * h + 16, w * h // 4 + 16
        return dict(kind=kind, g=g, w=w, h=h, n=n, most=most, walks=walks,
                    scratch=torch.empty(n * w * h, dtype=torch.uint8, device=DEV),
                    nodes=torch.zeros((n, most), dtype=torch.int32, device=DEV),
                    edges=torch.zeros((n, most), dtype=torch.int8, device=DEV),
                    offsets=torch.zeros((n, walks + 1), dtype=torch.int32, device=DEV),
                    counts=torch.zeros((n, 3), dtype=torch.int32, device=DEV))
    if kind in ("refine", "grad"):
        w, h = case["w"], case["h"]
        p, rp = _params(case), depix.refine_params(steps=case.get("steps", 1))
        a, b = _refined_pair(rng, w, h)
        pos = torch.zeros(2 * (4 * w + 3) * (4 * h + 3), dtype=torch.float32, device=DEV)
        prev, _ = _set_up(a, w, h, p, rp)
        top = _moved(prev, pos, int(seed))
        if kind == "grad":
            return dict(kind=kind, r=prev, rp=rp, pos=pos, n=len(top["flags"]), grad=torch.zeros_like(pos), img=a)
        return dict(kind=kind, prev=prev, prev_pos=pos, r=depix.Refiner(w * h), img=b, graph=_resolved(b, w, h, p),
                    w=w, h=h, p=p, rp=rp, pos=torch.zeros_like(pos))
    w, h = case["w"], case["h"]
    img, ws = _bgr(_frames(rng, 1, w, h)[0])
    n = w * h * depix.CELL
    return dict(kind=kind, img=img, w=w, h=h, ws=ws, subdivide=case["subdivide"],
                pos=torch.zeros((n, 2), dtype=torch.float32, device=DEV),
                col=torch.zeros((n, 4), dtype=torch.uint8, device=DEV), ec=np.zeros(w * h, np.int32),
                graph=np.zeros(w * h, np.uint8))


# --------------------------------------------------------------------- run


_free = ctypes.CDLL(None).free
_free.argtypes = [ctypes.c_void_p]


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["ctx"].frame(s["img"], s["w"], s["h"], s["ws"], s["layout"], s["p"], s["out"], s["graph"], s["labels"])
        return dict(out=s["out"], graph=s["graph"], labels=s["labels"])
    if kind in ("batch", "sprites"):
        s["ctx"].batch(s["ws"], s["hs"], s["io"], s["oo"], s["img"], s["p"], s["out"], s["labels"])
        return dict(out=s["out"], labels=s["labels"])
    if kind == "host":
        s["ctx"].batch_host(s["ws"], s["hs"], s["io"], s["oo"], s["img"], s["img"].numel() * 4, s["p"], s["out"],
                            s["out"].numel(), s["labels"])
        return dict(out=s["out"], labels=s["labels"])
    if kind == "walks":
        depix.border_walks(s["g"], s["w"], s["h"], s["n"], s["scratch"], s["nodes"], s["edges"], s["offsets"],
                           s["most"], s["walks"], s["counts"])
        return dict(nodes=s["nodes"], edges=s["edges"], offsets=s["offsets"], counts=s["counts"])
    if kind == "refine":
        r = s["r"]
        r.setup(s["img"], s["w"], s["h"], 4 * s["w"], depix.LAYOUT_RGBA, s["graph"], s["p"], s["rp"])
        r.warm_start(s["prev"], s["prev_pos"], s["pos"], count=False)
        r.run(s["rp"], s["pos"], energies=False)
        return dict(pos=s["pos"])
    if kind == "grad":
        e = s["r"].energy_grad(s["rp"], s["pos"], s["grad"])
        return dict(energy=np.array(e), grad=s["grad"])
    a = depix.launch_kernel_compat(s["pos"], s["col"], s["img"], s["w"], s["h"], s["ws"], s["ec"], s["graph"],
                                   s["subdivide"])
    points = np.ctypeslib.as_array(ctypes.cast(a, ctypes.POINTER(ctypes.c_float)), (s["w"] * s["h"] * depix.CELL, 2))
    weakref.finalize(points, _free, a)  # the caller owns the points
    return dict(points=points, pos=s["pos"], col=s["col"], edge_count=s["ec"], graph=s["graph"])


# -------------------------------------------------------------------- work


def work(case):
    kind = case["kind"]
    s2 = case.get("scale", 1) ** 2
    if kind == "sprites":
        px = case["n"] * ((case["lo"] + case["hi"]) / 2.0) ** 2
    else:
        px = float(case.get("n", 1) * case["w"] * case["h"])
    lab = 4 if case.get("labels") else 0
    if kind == "frame":
        return dict(bytes=px * ((4 if case["layout"] == "rgba" else 3) + 4 * s2 + 1 + lab), flops=0)
    if kind in ("batch", "sprites", "host"):
        return dict(bytes=px * (4 + 4 * s2 + lab), flops=0)
    if kind == "walks":
        return dict(bytes=px * (1 + 5 * 0.25), flops=0)  # about a node in four is on a border
    if kind in ("refine", "grad"):
        # about 0.2 nodes and 2.2 samples (at x4) a pixel, 90 operations a sample and 70 a node
        samples, nodes = px * 0.55 * case["scale"], px * 0.2
        return dict(bytes=px * 5 + nodes * 16, flops=case.get("steps", 1) * (90 * samples + 70 * nodes))
    return dict(bytes=px * (3 + depix.CELL * (8 + 8 + 4) + 5), flops=0)


# ------------------------------------------------------------------- exact

# ends of a segment over its three nodes, by type (none, middle, pinned start,
# pinned end, corner)
_WA = torch.tensor([[0, 0, 0], [3, 1, 0], [4, 0, 0], [1, 3, 0], [1, 3, 0]], dtype=torch.float64) / 4
_WB = torch.tensor([[0, 0, 0], [1, 3, 0], [3, 1, 0], [0, 4, 0], [0, 3, 1]], dtype=torch.float64) / 4


def _phi(z):
    return 0.5 * (1.0 + torch.erf(z / math.sqrt(2.0)))


class _Energy:
    """The refinement energy of a frozen topology in 64 bits."""

    def __init__(self, top, img, scale, rp):
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        h, w = img.shape
        self.p0 = to(top["q"]).double() / 4
        self.free = to(np.nonzero((top["flags"] & 1) == 0)[0])
        nbr = to(top["nbr"]).long()
        self.a, self.b = nbr[self.free, 0], nbr[self.free, 1]
        seg = to(top["segs"])[to(top["samples"])[:, 1].long()].long()
        self.nodes = seg[:, :3].clamp(min=0)
        self.wa, self.wb = _WA.to(DEV)[seg[:, 3]][..., None], _WB.to(DEV)[seg[:, 3]][..., None]
        col = to(top["cols"].astype(np.int64))[to(top["samples"])[:, 1].long()]
        rgb = lambda c: torch.stack([c & 255, (c >> 8) & 255, (c >> 16) & 255], -1).double()  # noqa: E731
        self.left, self.right = rgb(col[:, 0]), rgb(col[:, 1])
        at = to(top["samples"])[:, 0].long()
        xo, yo = at % (w * scale), at // (w * scale)
        self.x = torch.stack([(xo + 0.5) / scale, (yo + 0.5) / scale], 1).double()
        self.sig = rp.sigma / scale
        self.w = rp.w_curvature, rp.w_deviation, rp.w_coverage
        self.norm = rp.w_coverage / (3.0 * w * scale * h * scale)
        px = rgb(img.long() & 0xFFFFFF)
        ix, iy = xo // scale, yo // scale
        self.target = torch.zeros_like(self.left)
        for dj in (-1, 0, 1):
            for di in (-1, 0, 1):
                i, j = ix + di, iy + dj
                cx = _phi((self.x[:, 0] - i) / self.sig) - _phi((self.x[:, 0] - i - 1) / self.sig)
                cy = _phi((self.x[:, 1] - j) / self.sig) - _phi((self.x[:, 1] - j - 1) / self.sig)
                ok = (i >= 0) & (i < w) & (j >= 0) & (j < h)
                self.target += torch.where(ok, cx * cy, 0.0)[:, None] * px[j.clamp(0, h - 1), i.clamp(0, w - 1)]

    def parts(self, pos):
        f = max(len(self.free), 1)
        p = pos[self.free]
        t = pos[self.a] - 2 * p + pos[self.b]
        d = p - self.p0[self.free]
        q = pos[self.nodes]
        A, B = (self.wa * q).sum(1), (self.wb * q).sum(1)
        e, v = B - A, self.x - A
        dist = (e[:, 0] * v[:, 1] - e[:, 1] * v[:, 0]) / e.square().sum(1).sqrt()
        r = self.right + (self.left - self.right) * _phi(dist / self.sig)[:, None]
        return torch.stack([self.w[0] * 0.125 * t.square().sum() / f, self.w[1] * d.square().sum() / f,
                            self.norm * ((r - self.target) / 255.0).square().sum()])

    def grad(self, pos):
        """(three terms and their sum, gradient with zeros at pinned nodes)"""
        pos = pos.detach().requires_grad_(True)
        e = self.parts(pos)
        g, = torch.autograd.grad(e.sum(), pos)
        out = torch.zeros_like(g)
        out[self.free] = g[self.free]
        return torch.cat([e.detach(), e.detach().sum()[None]]), out


def _same_tiles(img_a, g_a, img_b, g_b, w, h):
    """Per 16x16 tile: its pixels' colours and graph bytes, and its one-pixel
    ring's, are those of the other frame."""
    same = ((img_a & 0xFFFFFF) == (img_b & 0xFFFFFF)).cpu().numpy() & (g_a == g_b).reshape(h, w).cpu().numpy()
    return np.array([[same[max(y - 1, 0):y + 17, max(x - 1, 0):x + 17].all() for x in range(0, w, 16)]
                     for y in range(0, h, 16)])


def exact(case, seed):
    """Rasters, graphs, labels and walks are whole numbers. The frame driver's
    points are sums of whole and quarter-multiple numbers that 32 bits hold
    exactly. The energies, the gradient and the refined positions follow from
    the frozen topology (whole numbers), by plain 64-bit arithmetic."""
    if case["kind"] not in ("refine", "grad"):
        return None
    s = prepare(case, seed)
    if case["kind"] == "grad":
        top = s["r"].export()
        e, g = _Energy(top, s["img"], case["scale"], s["rp"]).grad(s["pos"][:2 * s["n"]].double().reshape(-1, 2))
        out = torch.zeros_like(s["pos"], dtype=torch.float64)
        out[:2 * s["n"]] = g.reshape(-1)
        return dict(energy=e, grad=out)
    w, h, r, prev = s["w"], s["h"], s["r"], s["prev"]
    r.setup(s["img"], w, h, 4 * w, depix.LAYOUT_RGBA, s["graph"], s["p"], s["rp"])
    top, old = r.export(), prev.export()
    rng = np.random.default_rng([0x9A57, int(seed)])
    before, _ = _refined_pair(rng, w, h)
    same = _same_tiles(before, _resolved(before, w, h, s["p"]), s["img"], s["graph"], w, h)
    pos = top["q"] / 4.0
    was = {tuple(q): k for k, q in enumerate(old["q"].tolist())}
    old_pos = s["prev_pos"][:2 * len(old["q"])].double().reshape(-1, 2).cpu().numpy()
    for k, (x, y) in enumerate(top["q"].tolist()):
        j = was.get((x, y))
        if j is not None and same[min(max(y >> 2, 0), h - 1) // 16, min(max(x >> 2, 0), w - 1) // 16]:
            pos[k] = old_pos[j]
    E = _Energy(top, s["img"], case["scale"], s["rp"])
    pos = torch.from_numpy(pos).to(DEV)
    m, v = torch.zeros_like(pos), torch.zeros_like(pos)
    lr = s["rp"].lr
    for t in range(1, case["steps"] + 1):
        _, g = E.grad(pos)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        pos = pos - lr * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    out = torch.zeros_like(s["pos"], dtype=torch.float64)
    out[:2 * len(pos)] = pos.reshape(-1)
    return dict(pos=out)
