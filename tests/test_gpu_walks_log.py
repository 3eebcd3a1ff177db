"""Border walks whose paths come from the log of dropped walks, against the
oracle: frames where most starts run into the same obstacles, every split of
shared memory (log and index whole, cut short, absent; the 32-bit offset table
of wide frames; frames that do not fit), graphs whose walks never close or
close only from the log, and capacities that end a frame early."""
import numpy as np
import pytest

import oracle as O
from depix import synth

pytestmark = pytest.mark.gpu

# whole log; cut short; none; too large for shared memory; 32-bit table
SIZES = [(256, 224), (340, 300), (420, 380), (520, 400), (5000, 13)]


def frame_graph(rng, w, h):
    img = synth.draw_scene(rng, w, h, 16, max(4, w * h // 1500), max(3, w * h // 2000), dither_frac=0.05)
    bgr, ws = synth.rgba_to_bgr(img)
    return O.graph(bgr, w, h, ws)[2]


def ragged(rng, w, h):
    """Symmetric links of random density with solid areas: borders with many
    obstacles."""
    g = np.zeros((h, w), np.uint8)
    solid = rng.random((h // 8 + 1, w // 8 + 1)).repeat(8, 0).repeat(8, 1)[:h, :w]
    for e, (di, dj) in ((0, (-1, 1)), (1, (0, 1)), (2, (1, 1)), (3, (-1, 0))):
        a, b = solid[0:h - dj, max(0, -di):w - max(0, di)], solid[dj:h, max(0, di):w - max(0, -di)]
        m = (np.minimum(a, b) > 0.3) | (rng.random(a.shape) < 0.5)
        if e in (0, 2):
            m &= rng.random(a.shape) < 0.15
        g[0:h - dj, max(0, -di):w - max(0, di)] |= (m << e).astype(np.uint8)
        g[dj:h, max(0, di):w - max(0, -di)] |= (m << (7 - e)).astype(np.uint8)
    return g.reshape(-1)


@pytest.mark.parametrize("make", [frame_graph, ragged])
@pytest.mark.parametrize("w,h", SIZES)
def test_walks(cuda, w, h, make):
    import depix
    g = make(np.random.default_rng([w, h, make is ragged]), w, h)
    (walks, trunc), = depix.border_walk_lists(cuda.from_numpy(g.copy()).cuda(), w, h, max_nodes=2 * w * h, max_walks=w * h)
    assert not trunc
    assert walks == [(list(a), list(b)) for a, b in O.border_walks(g, w, h)]


def test_arbitrary_bytes(cuda):
    import depix
    rng = np.random.default_rng(5)
    for w, h in ((1, 1), (2, 3), (16, 2), (40, 33), (129, 65)):
        gs = [(rng.integers(0, 256, w * h) & rng.integers(0, 256, w * h) if k % 2 else rng.integers(0, 256, w * h)).astype(np.uint8)
              for k in range(8)]
        res = depix.border_walk_lists(cuda.from_numpy(np.concatenate(gs)).cuda(), w, h, nframes=len(gs),
                                      max_nodes=9 * w * h + 9, max_walks=w * h)
        for g, (walks, trunc) in zip(gs, res):
            assert not trunc
            assert walks == [(list(a), list(b)) for a, b in O.border_walks(g, w, h)]


@pytest.mark.parametrize("max_nodes,max_walks", [(1, 10 ** 5), (777, 10 ** 5), (5000, 10 ** 5), (10 ** 5, 1), (10 ** 5, 40)])
def test_capacities(cuda, max_nodes, max_walks):
    import depix
    w, h = 150, 120
    g = ragged(np.random.default_rng(9), w, h)
    full = [(list(a), list(b)) for a, b in O.border_walks(g, w, h)]
    (walks, trunc), = depix.border_walk_lists(cuda.from_numpy(g.copy()).cuda(), w, h, max_nodes=max_nodes, max_walks=max_walks)
    fit = 0
    while fit < len(full) and fit < max_walks and sum(len(a) for a, _ in full[:fit + 1]) <= max_nodes:
        fit += 1
    assert walks == full[:fit] and trunc == (fit < len(full))
