"""The walks' shared-memory kernel on the CPU, its lanes scheduled apart: the
kernel's source compiled as C++, every lane a fiber that runs from one barrier,
ballot or shuffle to the next before another lane runs. A store that another lane
has still to read around, with no barrier in between, shows as lanes at different
barriers or as another result; walks equal the oracle's whatever the order."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.join(HERE, "..", "pixel-art-remaster-gpu_gb300", "csrc", "depix_walks.cu")

SHIM = r"""
#include <ucontext.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#define __device__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(n)
#define __align__(n)
#define __shared__ static
struct uint4 { uint32_t x, y, z, w; };
struct Dim { unsigned x; };
static Dim threadIdx, blockIdx, blockDim;
static uint8_t g_smem[256 * 1024] __attribute__((aligned(16)));
static inline int __popc(unsigned v) { return __builtin_popcount(v); }
static inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
template <typename T> static inline T __ldg(const T* p) { return *p; }
static inline uint32_t atomicOr(uint32_t* p, uint32_t v) { uint32_t o = *p; *p |= v; return o; }

enum { RUNS, AT_WARP, AT_BLOCK, GONE };
struct Lane { ucontext_t ctx; std::vector<char> stack; int state, site, arg; uint32_t in, out; };
static std::vector<Lane> lanes;
static ucontext_t g_main;
static int g_now;
static bool g_apart;
static uint32_t meet(int state, int site, uint32_t in, int arg)
{
    Lane& l = lanes[g_now];
    l.state = state, l.site = site, l.in = in, l.arg = arg;
    swapcontext(&l.ctx, &g_main);
    return lanes[g_now].out;
}
// arg: 0 barrier or ballot, 1 + lane a shuffle from it, -o one from o lanes below
#define __syncwarp() ((void)meet(AT_WARP, __LINE__, 0, 0))
#define __syncthreads() ((void)meet(AT_BLOCK, __LINE__, 0, 0))
#define __ballot_sync(m, p) meet(AT_WARP, __LINE__, (p) ? 1u : 0u, 0)
#define __shfl_sync(m, v, s) (int)meet(AT_WARP, __LINE__, (uint32_t)(v), 1 + (int)(s))
#define __shfl_up_sync(m, v, o) meet(AT_WARP, __LINE__, (uint32_t)(v), -(int)(o))

static void (*g_body)();
static void entry() { g_body(); lanes[g_now].state = GONE; swapcontext(&lanes[g_now].ctx, &g_main); }

// order 0: lanes ascending, 1: descending, else drawn anew for each round
static bool run_block(int n, void (*body)(), int order)
{
    g_body = body;
    g_apart = false;
    lanes = std::vector<Lane>(n);
    for (int k = 0; k < n; k++) {
        Lane& l = lanes[k];
        l.stack.resize(64 * 1024);
        getcontext(&l.ctx);
        l.ctx.uc_stack.ss_sp = l.stack.data();
        l.ctx.uc_stack.ss_size = l.stack.size();
        l.ctx.uc_link = nullptr;
        l.state = RUNS;
        makecontext(&l.ctx, entry, 0);
    }
    srand(order);
    for (;;) {
        std::vector<int> at(n);
        for (int k = 0; k < n; k++) at[k] = order == 1 ? n - 1 - k : k;
        if (order > 1) for (int k = n - 1; k > 0; k--) std::swap(at[k], at[rand() % (k + 1)]);
        int ran = 0, gone = 0, block = 0;
        for (int k : at)
            if (lanes[k].state == RUNS) {
                g_now = k;
                threadIdx.x = k;
                swapcontext(&g_main, &lanes[k].ctx);
                ran++;
            }
        for (auto& l : lanes) gone += l.state == GONE, block += l.state == AT_BLOCK;
        if (gone == n) return true;
        bool freed = false;
        for (int w = 0; w < n; w += 32) { // a warp meets when all of it is at one place
            Lane* l = &lanes[w];
            int here = 0;
            uint32_t votes = 0;
            for (int k = 0; k < 32; k++) {
                here += l[k].state == AT_WARP;
                votes |= l[k].in << k;
            }
            if (!here) continue;
            for (int k = 0; k < 32; k++)
                if (l[k].state != AT_WARP || l[k].site != l[0].site) { g_apart = true; return false; }
            for (int k = 0; k < 32; k++) {
                const int a = l[k].arg;
                l[k].out = a == 0 ? votes : a > 0 ? l[a - 1].in : l[k + a < 0 ? k : k + a].in;
            }
            for (int k = 0; k < 32; k++) l[k].state = RUNS;
            freed = true;
        }
        if (!freed && block && block + gone == n) {
            for (auto& l : lanes) if (l.state == AT_BLOCK) l.state = RUNS;
            freed = true;
        }
        if (!freed) { g_apart = true; return false; }
    }
}

static const int kDi[8] = {-1, 0, 1, -1, 1, -1, 0, 1}, kDj[8] = {1, 1, 1, 0, 0, -1, -1, -1};
static inline int dir_di(int e) { return kDi[e]; }
static inline int dir_dj(int e) { return kDj[e]; }
static unsigned inside_mask(int x, int y, int w, int h)
{
    unsigned m = 0;
    for (int e = 0; e < 8; e++)
        if (x + kDi[e] >= 0 && x + kDi[e] < w && y + kDj[e] >= 0 && y + kDj[e] < h) m |= 1u << e;
    return m;
}
"""

MAIN = r"""
static struct { const uint8_t* g; int w, h; WalkSizes z; int32_t* on; int8_t* oe; int32_t* oo; int mn, mw; int32_t* cnt; } C;
template <typename T> static void body() { k_border_walks_smem<T>(C.g, C.w, C.h, C.z, C.on, C.oe, C.oo, C.mn, C.mw, C.cnt); }
extern "C" int walks(const uint8_t* g, int w, int h, int most, int wide, int mn, int mw, int order, int32_t* on, int8_t* oe,
                     int32_t* oo, int32_t* cnt)
{
    blockDim.x = kWalkThreads;
    C = {g, w, h, wide ? walk_sizes<int32_t>((size_t)w * h, most) : walk_sizes<uint16_t>((size_t)w * h, most), on, oe, oo, mn, mw, cnt};
    if (C.z.bytes > sizeof(g_smem)) return 2;
    return run_block(kWalkThreads, wide ? body<int32_t> : body<uint16_t>, order) && !g_apart ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def kernel(tmp_path_factory):
    text = open(SOURCE).read()
    text = text[:text.index("// larger frames: the graph from global memory, the state in the scratch")]
    for a, b in (('#include "depix_internal.h"', ""), ("extern __shared__ __align__(16) uint8_t sm[];", "uint8_t* sm = g_smem;")):
        assert text.count(a) == 1
        text = text.replace(a, b)
    d = tmp_path_factory.mktemp("walks")
    src, lib = str(d / "walks.cpp"), str(d / "walks.so")
    with open(src, "w") as f:
        f.write(SHIM + text + "\n}  // namespace depix\nusing namespace depix;\n" + MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-o", lib, src])
    return ctypes.CDLL(lib).walks


def graph(rng, w, h, lone):
    """Symmetric links between random pixels, a share of them without any."""
    g = np.zeros((h, w), np.uint8)
    on = rng.random((h, w)) >= lone
    for e, (di, dj) in ((0, (-1, 1)), (1, (0, 1)), (2, (1, 1)), (3, (-1, 0))):
        ys, xs = slice(0, h - dj), slice(max(0, -di), w - max(0, di))
        yt, xt = slice(dj, h), slice(max(0, di), w + min(0, di))
        m = on[ys, xs] & on[yt, xt] & (rng.random((h - dj, w - abs(di))) < (0.8 if e in (1, 3) else 0.15))
        g[ys, xs] |= (m << e).astype(np.uint8)
        g[yt, xt] |= (m << (7 - e)).astype(np.uint8)
    return g.reshape(-1)


def run(kernel, g, w, h, most, wide, order, mn=None, mw=None):
    mn, mw = mn or 9 * w * h + 9, mw or w * h
    on, oe = np.full(mn, -7, np.int32), np.full(mn, -7, np.int8)
    oo, cnt = np.zeros(mw + 1, np.int32), np.zeros(3, np.int32)
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (np.ascontiguousarray(g), on, oe, oo, cnt)]
    assert kernel(p[0], w, h, most, wide, mn, mw, order, *p[1:]) == 0, "lanes at different barriers"
    return [(on[a:b].tolist(), oe[a:b].tolist()) for a, b in zip(oo[:cnt[0]], oo[1:cnt[0] + 1])], bool(cnt[2])


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("most,wide", [(224 * 1024, 0), (12 * 1024, 0), (224 * 1024, 1)])  # log whole; absent; 32-bit table
def test_lanes_agree(kernel, order, most, wide):
    rng = np.random.default_rng([order, most, wide])
    for w, h, lone in ((1, 1, 1), (33, 1, 1), (40, 9, 0.9), (64, 21, 0.5), (31, 40, 0.1), (70, 33, 0.0)):
        g = graph(rng, w, h, lone)
        walks, cut = run(kernel, g, w, h, most, wide, order)
        assert not cut and walks == [(list(a), list(b)) for a, b in O.border_walks(g, w, h)]
    g = (rng.integers(0, 256, 29 * 17) & rng.integers(0, 256, 29 * 17)).astype(np.uint8)  # links on one side only
    assert run(kernel, g, 29, 17, most, wide, order)[0] == [(list(a), list(b)) for a, b in O.border_walks(g, 29, 17)]


@pytest.mark.parametrize("order", [0, 1, 4])
@pytest.mark.parametrize("mn,mw", [(1, 999), (100, 999), (9999, 1), (9999, 30)])
def test_lanes_agree_at_capacities(kernel, order, mn, mw):
    w, h = 48, 20
    g = graph(np.random.default_rng(3), w, h, 0.3)
    full = [(list(a), list(b)) for a, b in O.border_walks(g, w, h)]
    fit = 0
    while fit < min(len(full), mw) and sum(len(a) for a, _ in full[:fit + 1]) <= mn:
        fit += 1
    walks, cut = run(kernel, g, w, h, 224 * 1024, 0, order, mn, mw)
    assert walks == full[:fit] and cut == (fit < len(full))
