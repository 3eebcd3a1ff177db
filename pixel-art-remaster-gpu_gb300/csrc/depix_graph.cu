// depix_graph.cu -- similarity graph, crossing resolution and component
// labelling kernels.
//
// Frames are addressed through FrameRef so the same tile functions serve a
// single frame (grid.z = 1) and a batch of equal-size frames (grid.z = frame).
#include "depix_internal.h"

namespace depix {

// ------------------------------------------------------------ graph stage

// set when a bounded wait for a TMA tile load gave up (that tile of the
// graph was left unwritten); read and cleared by depix_take_device_faults
__device__ int g_graph_fault;
__device__ int g_heur_fault; // the same for the heuristics stage
// Test switch (depix_debug_tma_timeout): the TMA graph kernel issues no tile
// load and its wait gives up after kTestPolls polls, with nothing in flight.
__device__ int g_graph_tma_timeout_test;
constexpr int kTestPolls = 16;

// A block of kGThreads threads makes a tile of 64 x (4 GH) nodes: it turns the
// tile's pixel window (one pixel around it, more on the sides for the 16-byte
// alignment of the TMA box) into comparable words in shared memory, once a
// pixel; then each group of 16 lanes marches up a strip of GH rows, four
// columns a lane, holding two rows of words in registers, the pairs of four
// columns as the bytes of one register and the node bytes of four columns as
// another.
//
// Bound: issue. What a pixel costs is its word (about 25 instructions), four
// pair tests of three instructions and a quarter of the packed node assembly;
// a thread per pixel over byte arrays in shared memory took five times as
// many. 1024 frames of 256x224: 512 us before, 175 us now (85 instructions a pixel).
constexpr int kGTW = 64;          // tile width (pixels): 16 lanes of four columns
constexpr int kGThreads = 64;     // four groups of 16 lanes, strips of GH rows above each other
constexpr int kGBoxW = kGTW + 8;  // window from x0 - 4
// rows of a strip: 8 in large batches (the pairs of the row below a strip are
// made twice, 1/8 of them), 4 up to 2^21 pixels and 1 up to 2^18, where blocks
// are what is missing (8 frames of 256x224: 10.5 us with 8 rows, 9.9 with 4; one
// frame: 7.8 us with 2 rows, 7.1 with 1; 1024 frames: 198 us with 4 rows, 175
// with 8), 4 in the tile queue (its 64x16 tiles); the left column's pairs take
// a lane a row, so at most 15
constexpr int kGStrip = 8, kGStripSmall = 4, kGStripFrame = 1, kGStripQueue = 4;

// Comparable form of a packed Y/U/V word (yuv_word): its byte fields in slots
// of 10 bits, whose bit 9 is a guard. With A = a + guards + thresholds, the
// slots of E = A - b hold 512 + t + (a - b) and those of C - E, C = 2 (guards
// + thresholds), 512 + t - (a - b): a and b are similar (every field within
// its threshold) when both keep all guard bits. kNoPixel, outside the image,
// is similar to no pixel: its lowest slot is further from any byte than any
// threshold reaches.
constexpr uint32_t kGuards = 1u << 9 | 1u << 19 | 1u << 29;
constexpr uint32_t kNoPixel = 511u;

__device__ __forceinline__ uint32_t spread_fields(uint32_t w)
{
    return (w & 0xFFu) + ((w & 0xFF00u) << 2) + ((w & 0xFF0000u) << 4);
}

// Spread words of four RGBA pixels, yuv_word's arithmetic on integers, exact
// over every input: the quotient of 0..255000 by 1000; 0.492f and 0.877f
// times -255..255 rounded to float and truncated (no product of a negative
// difference is whole, so truncation is the floor plus one). Negative fields
// borrow from the next slot as they do from the next byte of the word. The
// double evaluation only where a luma sum leaves no remainder, as yuv_word
// explains; one branch for the four.
__device__ __forceinline__ void pixel_fields(const uint32_t (&px)[4], int mode, uint32_t (&out)[4])
{
    int y[4], sum[4];
    bool whole = false;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        // in the reference's byte order B plays r and R plays b: 299 B + 587 G + 114 R
        sum[q] = (int)__dp4a(px[q], 0x002B4B72u, 256u * __dp4a(px[q], 0x00010200u, 0u));
        y[q] = (int)__umulhi((unsigned)sum[q], 4294968u);
        whole |= sum[q] == y[q] * 1000;
    }
    if (whole) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (sum[q] != y[q] * 1000 || sum[q] == 0) continue;
            const double r = (double)(int)((px[q] >> 16) & 0xFFu), g = (double)(int)((px[q] >> 8) & 0xFFu);
            const double b = (double)(int)(px[q] & 0xFFu);
            const double t = mode == DEPIX_YUV_HOST
                                 ? __dadd_rn(__dadd_rn(__dmul_rn(0.299, r), __dmul_rn(0.587, g)), __dmul_rn(0.114, b))
                                 : __fma_rn(0.114, b, __fma_rn(0.299, r, __dmul_rn(0.587, g)));
            y[q] = __double2int_rz(t);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int du = (int)(px[q] & 0xFFu) - y[q], dv = (int)((px[q] >> 16) & 0xFFu) - y[q];
        const int u = ((du * 32245) >> 16) + (int)((unsigned)du >> 31);
        const int v = ((dv * 57475) >> 16) + (int)((unsigned)dv >> 31);
        out[q] = (uint32_t)(y[q] * (1 << 20) + u * (1 << 10) + v) & 0x0FF3FCFFu;
    }
}

// bit k set in the packed bytes when a (as A) and b are similar
__device__ __forceinline__ uint32_t pair_bit(uint32_t A, uint32_t b, uint32_t C, uint32_t bit)
{
    const uint32_t E = A - b;
    return (~(E & (C - E)) & kGuards) == 0 ? bit : 0u;
}

template <int LAYOUT, int GH, bool TMA = false>
__device__ __forceinline__ void graph_tile(const FrameRef f, int x0, int y0, uint32_t thr, bool fuse_trivial,
                                           const CUtensorMap* pix_map = nullptr, int frame = 0)
{
    static_assert(GH < 16, "a lane for each row's left pair");
    constexpr int TH = GH * (kGThreads / 16), RH = TH + 2, RW = kGBoxW;
    __shared__ __align__(128) uint32_t win[RH][RW]; // pixel (x, y) at win[y - y0 + 1][x - x0 + 4]
    const int w = f.w, h = f.h, mode = yuv_mode_of(thr);
    if constexpr (TMA) {
        __shared__ uint64_t bar;
        __shared__ int ok;
        if (threadIdx.x == 0) {
            const bool test_timeout = *(volatile int*)&g_graph_tma_timeout_test != 0;
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, (uint32_t)sizeof(win));
            if (!test_timeout) tma_load_3d(&win[0][0], pix_map, x0 - 4, y0 - 1, frame, &bar);
            ok = tma_wait_or_flag(&bar, &g_graph_fault, test_timeout ? kTestPolls : kTmaPolls) ? 1 : 0;
        }
        __syncthreads();
        if (!ok) return;
    }
    // ---- words of the window, four a thread (outer columns of the box that no
    // pair reads are made too: they keep the rows 16-byte aligned)
    const bool inside = x0 >= 4 && y0 >= 1 && x0 + kGTW + 4 <= w && y0 + TH + 1 <= h;
    for (int k = threadIdx.x; k < RH * (RW / 4); k += kGThreads) {
        const int ry = k / (RW / 4), rx = 4 * (k % (RW / 4));
        const int gx = x0 - 4 + rx, gy = y0 - 1 + ry;
        uint32_t px[4];
        if constexpr (TMA) {
            const uint4 v = *reinterpret_cast<const uint4*>(&win[ry][rx]);
            px[0] = v.x; px[1] = v.y; px[2] = v.z; px[3] = v.w;
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                px[q] = 0;
                if (gx + q < 0 || gx + q >= w || gy < 0 || gy >= h) continue;
                if (LAYOUT == DEPIX_LAYOUT_RGBA) {
                    px[q] = __ldg(reinterpret_cast<const uint32_t*>(f.img + (size_t)gy * f.ws) + gx + q);
                } else {
                    const uint32_t c = load_bgr(f.img, f.ws, LAYOUT, gx + q, gy);
                    px[q] = ((c >> 16) & 0xFFu) | (c & 0xFF00u) | ((c & 0xFFu) << 16);
                }
            }
        }
        uint32_t fd[4];
        pixel_fields(px, mode, fd);
        if (!inside) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (gx + q < 0 || gx + q >= w || gy < 0 || gy >= h) fd[q] = kNoPixel;
        }
        *reinterpret_cast<uint4*>(&win[ry][rx]) = make_uint4(fd[0], fd[1], fd[2], fd[3]);
    }
    __syncthreads();
    // ---- strips
    const uint32_t GT = kGuards + spread_fields(thr & 0x00FFFFFFu), C = 2u * GT;
    const int gl = threadIdx.x & 15, base = GH * (threadIdx.x >> 4); // window row of y0 - 1 + base
    // pairs of a column c with the row above (words lo: row, hi: row above): bit
    // 0 right, 1 up, 2 up-right, 3 right's up-left, 4 the block's four sides
    // all similar (its trivial crossing goes, crossCheck_4)
    // the column left of the tile, a row a lane
    uint32_t edge = 0;
    if (gl <= GH) {
        const uint32_t* lo = &win[base + gl][3];
        const uint32_t* hi = &win[base + gl + 1][3];
        const uint32_t a0 = lo[0] + GT, a1 = lo[1] + GT;
        edge = pair_bit(a0, lo[1], C, 1u) | pair_bit(a0, hi[0], C, 2u) | pair_bit(a0, hi[1], C, 4u) |
               pair_bit(a1, hi[0], C, 8u);
        if (fuse_trivial && (edge & 3u) == 3u && pair_bit(a1, hi[1], C, 1u) && pair_bit(hi[0] + GT, hi[1], C, 1u)) edge |= 16u;
    }
    auto row_words = [&](int r, uint32_t (&v)[5]) {
        const uint4 q = *reinterpret_cast<const uint4*>(&win[r][4 + 4 * gl]);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        v[4] = win[r][8 + 4 * gl];
    };
    auto right_pairs = [&](const uint32_t (&A)[5], const uint32_t (&v)[5]) {
        return pair_bit(A[0], v[1], C, 1u) | pair_bit(A[1], v[2], C, 1u << 8) | pair_bit(A[2], v[3], C, 1u << 16) |
               pair_bit(A[3], v[4], C, 1u << 24);
    };
    uint32_t A[5], n[5];
    row_words(base, n);
#pragma unroll
    for (int q = 0; q < 5; q++) A[q] = n[q] + GT;
    uint32_t R = right_pairs(A, n), below = 0, below_left = 0;
    const int gx = x0 + 4 * gl;
    uint8_t* out = f.graph + (ptrdiff_t)(y0 + base - 1) * w + gx;
    const bool wide = gx + 3 < w && ((w | (int)reinterpret_cast<uintptr_t>(f.graph)) & 3) == 0;
#pragma unroll
    for (int r = 0; r <= GH; r++) {
        row_words(base + r + 1, n);
        uint32_t P = R, U = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            U |= pair_bit(A[q], n[q], C, 1u << (8 * q));
            P |= pair_bit(A[q], n[q + 1], C, 4u << (8 * q)) | pair_bit(A[q + 1], n[q], C, 8u << (8 * q));
        }
        const uint32_t U4 = pair_bit(A[4], n[4], C, 1u << 24);
#pragma unroll
        for (int q = 0; q < 5; q++) A[q] = n[q] + GT;
        const uint32_t Rn = right_pairs(A, n);
        P |= U << 1;
        if (fuse_trivial) P |= (R & Rn & U & (U >> 8 | U4)) << 4;
        R = Rn;
        uint32_t left = __shfl_up_sync(0xFFFFFFFFu, P, 1, 16) >> 24;
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, edge, r, 16);
        if (gl == 0) left = e;
        const uint32_t L = P << 8 | left; // the pairs of the column to the left
        if (r > 0) {
            constexpr uint32_t k1 = 0x01010101u;
            uint32_t node = (L >> 3 & k1) | (P & 2 * k1) | (P & 4 * k1) | (L & k1) << 3 | (P & k1) << 4 |
                            (below_left & 4 * k1) << 3 | (below & 2 * k1) << 5 | (below & 8 * k1) << 4;
            // the blocks at whose corners the node is lose their crossing diagonals
            node &= ~((L >> 4 & k1) | (P >> 2 & 4 * k1) | (below_left & 16 * k1) << 1 | (below & 16 * k1) << 3);
            if (y0 + base + r - 1 < h) {
                uint8_t* o = out + (size_t)r * w;
                if (wide) {
                    *reinterpret_cast<uint32_t*>(o) = node;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (gx + q < w) o[q] = (uint8_t)(node >> (8 * q));
                }
            }
        }
        below = P;
        below_left = L;
    }
}

template <int LAYOUT, int GH>
__global__ void __launch_bounds__(kGThreads) k_graph(FrameBatch b, uint32_t thr, int fuse_trivial)
{
    early_start();
    FrameRef f = b.frame(blockIdx.z);
    graph_tile<LAYOUT, GH>(f, blockIdx.x * kGTW, blockIdx.y * 4 * GH, thr, fuse_trivial != 0);
}

// RGBA frames whose base, rows and frame stride are 16-byte aligned: the
// pixel windows come by TMA
template <int GH>
__global__ void __launch_bounds__(kGThreads) k_graph_tma(FrameBatch b, uint32_t thr, int fuse_trivial,
                                                         const __grid_constant__ CUtensorMap pix_map)
{
    early_start();
    FrameRef f = b.frame(blockIdx.z);
    graph_tile<DEPIX_LAYOUT_RGBA, GH, true>(f, blockIdx.x * kGTW, blockIdx.y * 4 * GH, thr, fuse_trivial != 0, &pix_map,
                                            (int)blockIdx.z);
}

// Trivial removal on a graph in place (crossCheck_4, graph_functions.cu:1211-1274).
// Only orthogonal bits are read and only diagonal bits written: race-free.
__global__ void k_trivial(uint8_t* g, int w, int h)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || j >= h) return;
    auto at = [&](int x, int y) -> unsigned {
        return (x < 0 || y < 0 || x >= w || y >= h) ? 0u : (unsigned)g[(size_t)y * w + x];
    };
    unsigned c = at(i, j), l = at(i - 1, j), r = at(i + 1, j), u = at(i, j + 1), d = at(i, j - 1);
    unsigned ul = at(i - 1, j + 1), ur = at(i + 1, j + 1), dl = at(i - 1, j - 1), dr = at(i + 1, j - 1);
    unsigned out = c;
    if (bitof(l, 1) && bitof(l, 4) && bitof(ul, 6) && bitof(ul, 4) && bitof(c, 3) && bitof(c, 1) && bitof(u, 6) &&
        bitof(u, 3))
        out &= ~1u;
    if (bitof(c, 1) && bitof(c, 4) && bitof(u, 6) && bitof(u, 4) && bitof(r, 3) && bitof(r, 1) && bitof(ur, 6) &&
        bitof(ur, 3))
        out &= ~4u;
    if (bitof(dl, 1) && bitof(dl, 4) && bitof(l, 6) && bitof(l, 4) && bitof(d, 3) && bitof(d, 1) && bitof(c, 6) &&
        bitof(c, 3))
        out &= ~32u;
    if (bitof(d, 1) && bitof(d, 4) && bitof(c, 6) && bitof(c, 4) && bitof(dr, 3) && bitof(dr, 1) && bitof(r, 6) &&
        bitof(r, 3))
        out &= ~128u;
    if (out != c) g[(size_t)j * w + i] = (uint8_t)out;
}

// ------------------------------------------------------- heuristics stage

constexpr int kHTW = 64, kHTH = 16;
// Window of a tile: 16 columns (TMA's alignment) and 8 rows around it, which
// hold the 8x8 windows of the vote and nearly all curve-length walks; a walk
// moves at most 31 steps from its block, and one that leaves the window reads
// the snapshot in global memory. (A halo of 32 that held every walk was 10 KB
// to load and keep for the tile's 1 KB.)
constexpr int kHaloX = 16, kHaloY = 8;
constexpr int kHRW = kHTW + 2 * kHaloX, kHRH = kHTH + 2 * kHaloY;
// Threads of a tile. With few tiles a tile's time is the call's, and more threads
// shorten its lists of crossings and joins (a call with labels at x4, us with
// 128 / 256 / 512 threads: a 256x224 frame, 56 tiles, 36.5 / 33.6 / 28.8; 8 of
// them 51.6 / 41.1 / 39.0; 12 of them, 672 tiles, 58.8 / 54.7 / 53.9; 16 of them
// 61.0 / 58.6 / 62.0; 20 of them, 1120, 68.2 / 66.5 / 66.6; 24 72.4 / 72.5 / 72.5).
// With many, blocks of 128 leave less waiting at barriers (heuristics of 1024
// frames 244 / 309 with 256).
constexpr int kHThreads = 128;
// The lines, 760 and 1216 tiles of the 152 SMs measured, are kept per SM.
constexpr int kTilesPerSm512 = 5, kTilesPerSm256 = 8;

struct SnapTile {
    const uint8_t (*s)[kHRW];
    int ox, oy; // image coordinates of s[0][0]
    const uint8_t* g;
    int w, h;
    __device__ __forceinline__ unsigned at(int x, int y) const { return s[y - oy][x - ox]; } // inside the window
    __device__ __forceinline__ unsigned far(int x, int y) const
    {
        if ((unsigned)(x - ox) < (unsigned)kHRW && (unsigned)(y - oy) < (unsigned)kHRH) return s[y - oy][x - ox];
        return (unsigned)x < (unsigned)w && (unsigned)y < (unsigned)h ? g[(size_t)y * w + x] : 0u;
    }
};

// set bits of node other than bit e; last = the highest such bit in the
// scan order e+1 .. e+7 (mod 8)
__device__ __forceinline__ int others(unsigned node, int e, int& last)
{
    unsigned rest = (node & 0xFFu) & ~(1u << e);
    int s = __popc(rest);
    if (s) {
        // scan order e+1, ..., 7, 0, ..., e-1: the last in that order is the
        // highest set bit below e if any, else the highest set bit overall
        unsigned below = rest & ((1u << e) - 1u);
        last = below ? 31 - __clz(below) : 31 - __clz(rest);
    }
    return s;
}

// Block decision codes: bit 1 remove "/" (bits 2/5), bit 2 remove "\" (bits
// 0/7); kDecWalk: the curve lengths decide.
constexpr unsigned kDecSlash = 2, kDecBack = 4, kDecWalk = 8;

// Curve length of arm q of the block whose lower-left node is (i, j)
// (calcVal2PathSize, graph_functions.cu:541-573): from its node on, away from
// the block, while the curve does not branch or end, at most 31 steps. Arms 0
// and 1 are "/", 2 and 3 "\". The reference walks the second arm of a diagonal
// on the first one's count and stops at 31: min(31, the two lengths).
constexpr int kMaxCurve = 31;
__device__ __forceinline__ int arm_length(const SnapTile& t, int i, int j, int q)
{
    int x = i + (q == 1 || q == 2), y = j + (q & 1), e = q == 0 ? 2 : q == 1 ? 5 : q == 2 ? 0 : 7;
    int len = 0;
    for (; len < kMaxCurve; len++) {
        int k = 0;
        if (others(t.far(x, y), e, k) != 1) break;
        x += dir_di(k);
        y += dir_dj(k);
        e = 7 - k;
    }
    return len;
}

// Block decision (processHeuristics2, graph_functions.cu:761-849) as far as the
// block's own nodes make it; where no arm goes on, both curves have length 0
// and "/" goes.
__device__ __forceinline__ unsigned block_decision(const SnapTile& t, int i, int j)
{
    unsigned n1 = t.at(i, j), n2 = t.at(i, j + 1), n3 = t.at(i + 1, j), n4 = t.at(i + 1, j + 1);
    int dummy;
    int o1 = others(n1, 2, dummy), o4 = others(n4, 5, dummy), o3 = others(n3, 0, dummy), o2 = others(n2, 7, dummy);
    if (o1 == 1 && o4 == 1) return kDecBack;       // curve through "/"
    if (o3 == 1 && o2 == 1) return kDecSlash;      // curve through "\"
    bool v1 = o1 == 0, v4 = o4 == 0, v3 = o3 == 0, v2 = o2 == 0;
    if ((v1 || v4) && !v3 && !v2) return kDecBack; // island
    if (v3 || (v2 && !v1 && !v4)) return kDecSlash; // island, reference precedence (graph_functions.cu:805)
    return o1 == 1 || o2 == 1 || o3 == 1 || o4 == 1 ? kDecWalk : kDecSlash;
}

// Size of the component of `seed` in an 8x8 window whose bit r*8+c is the
// pixel in window row r, column c; m[e] holds the pixels with edge e. The
// fill follows the edges inside the window only (a move off the window's
// columns is masked, one off its rows shifts out).
__device__ __forceinline__ int window_component(const uint64_t (&m)[8], uint64_t seed)
{
    constexpr uint64_t kCol0 = 0x0101010101010101ull, kCol7 = 0x8080808080808080ull;
    uint64_t c = seed, prev;
    do {
        prev = c;
        c |= ((prev & m[0]) << 7) & ~kCol7; // (-1, +1)
        c |= (prev & m[1]) << 8;            // ( 0, +1)
        c |= ((prev & m[2]) << 9) & ~kCol0; // (+1, +1)
        c |= ((prev & m[3]) >> 1) & ~kCol7; // (-1,  0)
        c |= ((prev & m[4]) << 1) & ~kCol0; // (+1,  0)
        c |= ((prev & m[5]) >> 9) & ~kCol7; // (-1, -1)
        c |= (prev & m[6]) >> 8;            // ( 0, -1)
        c |= ((prev & m[7]) >> 7) & ~kCol0; // (+1, -1)
    } while (c != prev);
    return __popcll(c);
}

// Weighted vote of the three heuristics of Kopf and Lischinski,
// "Depixelizing Pixel Art" (SIGGRAPH 2011), section 3.2, for the block whose
// lower-left node is (i, j); not in the reference, which decides by the
// ordered tests of block_decision. Each heuristic votes for the diagonal to
// keep: curves by the difference of the two curve lengths (the same walks as
// block_decision), sparse pixels by the difference of the sizes of the two
// diagonals' components inside the 8x8 window centred on the block (the
// sparser one is kept), islands with weight 5 for a diagonal whose removal
// would leave one of its ends without edges. The diagonal with fewer votes
// is removed; a tie removes both.
//
// Four lanes a block (all lanes of the warp call it): each has the length of
// its arm, takes two of the window's eight edge masks off its bytes (the
// product gathers four bytes' bits) and gets the others by shuffle; two lanes
// fill a diagonal's component each.
__device__ __forceinline__ unsigned vote_decision(const SnapTile& t, int i, int j, int seg, int seg2)
{
    unsigned n1 = t.at(i, j), n2 = t.at(i, j + 1), n3 = t.at(i + 1, j), n4 = t.at(i + 1, j + 1);
    int dummy;
    int o1 = others(n1, 2, dummy), o4 = others(n4, 5, dummy), o3 = others(n3, 0, dummy), o2 = others(n2, 7, dummy);
    int keep_slash = 0, keep_back = 0;
    if (seg > seg2) keep_slash += seg - seg2;
    else keep_back += seg2 - seg;
    if (o1 == 0 || o4 == 0) keep_slash += 5;
    if (o3 == 0 || o2 == 0) keep_back += 5;
    // window columns i-3 .. i+4, rows j-3 .. j+4 (inside the snapshot halo)
    const int q = threadIdx.x & 3, cx = i - 3 - t.ox;
    const uint32_t* row = reinterpret_cast<const uint32_t*>(&t.s[j - 3 - t.oy][cx & ~3]);
    uint64_t mine[2] = {0, 0};
#pragma unroll
    for (int r = 0; r < 8; r++, row += kHRW / 4) {
        const uint32_t lo = __funnelshift_r(row[0], row[1], 8 * (cx & 3)), hi = __funnelshift_r(row[1], row[2], 8 * (cx & 3));
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t bits = ((lo >> (2 * q + k) & 0x01010101u) * 0x01020408u >> 24) |
                                  ((hi >> (2 * q + k) & 0x01010101u) * 0x01020408u >> 24) << 4;
            mine[k] |= (uint64_t)bits << (8 * r);
        }
    }
    uint64_t m[8];
#pragma unroll
    for (int e = 0; e < 8; e++) m[e] = __shfl_sync(0xFFFFFFFFu, (unsigned long long)mine[e & 1], e >> 1, 4);
    // i1 = (i, j) is window bit 27 (with i4 on "/"), i2 = (i, j + 1) bit 35
    int size = 0;
    if (q < 2) size = window_component(m, 1ull << (q == 0 ? 27 : 35));
    const int size_slash = __shfl_sync(0xFFFFFFFFu, size, 0, 4), size_back = __shfl_sync(0xFFFFFFFFu, size, 1, 4);
    if (size_slash < size_back) keep_slash += size_back - size_slash;
    else keep_back += size_slash - size_back;
    if (keep_slash > keep_back) return kDecBack;
    if (keep_back > keep_slash) return kDecSlash;
    return kDecSlash | kDecBack;
}

constexpr int kMaxJoins = (kHTH - 1) * 3 * kHTW; // every upward edge of a tile
template <int NT>
__device__ void tile_labels(const uint8_t (*node)[kHTW], uint16_t* joins, int32_t* L, int w, int h, int x0, int y0);

// Heuristic resolution of one 64x16 tile; with L set, the tile's local
// component labels too (union-find over the resolved bytes, still in shared
// memory), which leaves the label stage only the merge across tile borders
// and the roots.
//
// Crossings are few, so four 2x2 blocks a thread are tested for one at a time
// in packed bytes, the crossings go to a list, and a lane decides each (once:
// its four corner nodes each lose a bit of the decision). Bound: issue (79 %);
// 1024 frames of 256x224 with labels: 636 us when every node tested its four
// blocks over bytes and every lane ran a row's join masks, 244 us now (the
// vote on 32 frames of 159x143: 68 us before, 25 now). The window by 16-byte
// asynchronous copies instead of TMA: 255.
template <int NT, bool TMA = false, bool VOTE = false>
__device__ __forceinline__ void heuristics_tile(const uint8_t* snap, uint8_t* out, int w, int h, int x0, int y0,
                                                int32_t* L = nullptr, const CUtensorMap* map = nullptr,
                                                int frame = 0)
{
    // the window, later the labels' list of joins
    __shared__ __align__(128) uint8_t buf[kHRH * kHRW > 2 * kMaxJoins ? kHRH * kHRW : 2 * kMaxJoins];
    static_assert(sizeof(buf) >= kHRH * kHRW + 2 * (kHTW + 1) * (kHTH + 1), "a second list behind the window");
    uint8_t(*s)[kHRW] = reinterpret_cast<uint8_t(*)[kHRW]>(buf);
    __shared__ __align__(16) uint8_t res[kHTH][kHTW]; // resolved nodes
    // blocks touching the tile that hold a crossing: column - (x0 - 1) | row - (y0 - 1) << 8
    __shared__ uint16_t list[(kHTW + 1) * (kHTH + 1)];
    __shared__ int count, count2;
    const int ox = x0 - kHaloX, oy = y0 - kHaloY;
    if constexpr (TMA) {
        // the window as one TMA box (x0 - 16 is a multiple of 16 bytes);
        // bytes outside the image read as zero
        __shared__ uint64_t bar;
        __shared__ int ok;
        if (threadIdx.x == 0) {
            count = count2 = 0;
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, (uint32_t)(kHRH * kHRW));
            tma_load_3d(&s[0][0], map, ox, oy, frame, &bar);
            ok = tma_wait_or_flag(&bar, &g_heur_fault) ? 1 : 0;
        }
        __syncthreads();
        if (!ok) return;
    } else {
        if (threadIdx.x == 0) count = count2 = 0;
        constexpr int RW4 = kHRW / 4;
        for_each_batched<2>(
            kHRH * RW4, [&](int k) { return row_bytes4(snap, w, h, ox + 4 * (k % RW4), oy + k / RW4); },
            [&](int k, uint32_t v) { *reinterpret_cast<uint32_t*>(&s[k / RW4][4 * (k % RW4)]) = v; });
        __syncthreads();
    }
    const SnapTile t{s, ox, oy, snap, w, h};
    // ---- crossings, four blocks of a row at a time: rows y0 - 1 .. y0 + 15,
    // columns x0 - 4 .. x0 + 63 of which the first word gives x0 - 1 only.
    // Blocks reaching outside the image read zeros and are never crossings.
    constexpr int NW = kHTW / 4 + 1;
    for (int k = threadIdx.x; k < NW * (kHTH + 1); k += NT) {
        const int wc = k % NW, by = k / NW;
        const uint32_t* a = reinterpret_cast<const uint32_t*>(&s[by + kHaloY - 1][kHaloX - 4 + 4 * wc]);
        const uint32_t* b = a + kHRW / 4;
        const uint32_t a0 = a[0], b0 = b[0];
        const uint32_t a1 = __funnelshift_r(a0, a[1], 8), b1 = __funnelshift_r(b0, b[1], 8); // one column on
        uint32_t cross = (a0 >> 2) & (b0 >> 7) & a1 & (b1 >> 5) & 0x01010101u;
        if (wc == 0) cross &= 0x01000000u;
        if (wc > 0 && by > 0) *reinterpret_cast<uint32_t*>(&res[by - 1][4 * wc - 4]) = a0;
        if (cross) {
            int slot = atomicAdd(&count, __popc(cross));
            while (cross) {
                const int q = (__ffs(cross) - 1) >> 3;
                cross &= cross - 1;
                list[slot++] = (uint16_t)((4 * wc + q - 3) | by << 8);
            }
        }
    }
    __syncthreads();
    const int n = count;
    // the block's nodes lose their bits of a removed diagonal, those inside the tile
    auto apply = [&](int bx, int by, unsigned d) {
        auto drop = [&](int tx, int ty, unsigned bit) {
            if ((unsigned)tx < (unsigned)kHTW && (unsigned)ty < (unsigned)kHTH)
                atomicAnd(reinterpret_cast<unsigned*>(&res[ty][tx & ~3]), ~(bit << (8 * (tx & 3))));
        };
        if (d & kDecSlash) {
            drop(bx - 1, by - 1, 4u);
            drop(bx, by, 32u);
        }
        if (d & kDecBack) {
            drop(bx, by - 1, 1u);
            drop(bx - 1, by, 128u);
        }
    };
    // decided by their own nodes; those that need curve lengths to a second
    // list (behind the window), so that four lanes can walk a block's arms at
    // once (8 frames of 256x224: 14.6 us when a lane walked all four, 12.9 now;
    // the vote on 32 frames of 159x143: 28.7 us, 24.9 now)
    const uint16_t* walks = list;
    int nwalks = n;
    if constexpr (!VOTE) {
        uint16_t* more = reinterpret_cast<uint16_t*>(buf + kHRH * kHRW);
        for (int k = threadIdx.x; k < n; k += NT) {
            const int bx = list[k] & 0xFF, by = list[k] >> 8;
            const unsigned d = block_decision(t, x0 - 1 + bx, y0 - 1 + by);
            if (d == kDecWalk) more[atomicAdd(&count2, 1)] = list[k];
            else apply(bx, by, d);
        }
        __syncthreads();
        walks = more;
        nwalks = count2;
    }
    for (int k0 = 0; k0 < nwalks; k0 += NT / 4) {
        const int k = k0 + (threadIdx.x >> 2), q = threadIdx.x & 3;
        if (k0 + ((int)threadIdx.x & ~31) / 4 >= nwalks) break; // whole warps
        const int it = walks[k < nwalks ? k : nwalks - 1], bx = it & 0xFF, by = it >> 8;
        const int i = x0 - 1 + bx, j = y0 - 1 + by;
        int len = arm_length(t, i, j, q);
        len = min(kMaxCurve, len + __shfl_xor_sync(0xFFFFFFFFu, len, 1));
        const int seg = __shfl_sync(0xFFFFFFFFu, len, 0, 4), seg2 = __shfl_sync(0xFFFFFFFFu, len, 2, 4);
        unsigned d;
        if constexpr (VOTE) d = vote_decision(t, i, j, seg, seg2);
        else d = seg2 < seg ? kDecBack : kDecSlash;
        if (k < nwalks && q == 0) apply(bx, by, d);
    }
    __syncthreads();
    // ---- output, four nodes a thread; for the labels the nodes on the image's
    // edge lose their bits toward outside
    const bool edge = x0 == 0 || y0 == 0 || x0 + kHTW >= w || y0 + kHTH >= h;
    for (int k = threadIdx.x; k < kHTW / 4 * kHTH; k += NT) {
        const int tx = 4 * (k % (kHTW / 4)), ty = k / (kHTW / 4);
        const int i = x0 + tx, j = y0 + ty;
        const uint32_t v = *reinterpret_cast<const uint32_t*>(&res[ty][tx]);
        if (j < h && i < w) {
            uint8_t* o = out + (size_t)j * w + i;
            if (i + 3 < w && (reinterpret_cast<uintptr_t>(o) & 3) == 0) {
                *reinterpret_cast<uint32_t*>(o) = v;
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (i + q < w) o[q] = (uint8_t)(v >> (8 * q));
            }
        }
        if (L && edge) {
            uint32_t m = 0;
            if (j < h) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (i + q < w) m |= inside_mask(i + q, j, w, h) << (8 * q);
            }
            *reinterpret_cast<uint32_t*>(&res[ty][tx]) = v & m;
        }
    }
    if (L) {
        if (edge) __syncthreads();
        tile_labels<NT>(res, reinterpret_cast<uint16_t*>(buf), L, w, h, x0, y0);
    }
}

// VOTE: the weighted vote instead of the reference's ordered tests; L may be
// NULL
template <bool VOTE, int NT>
__global__ void __launch_bounds__(NT) k_heuristics(GraphBatch b, int32_t* L)
{
    follow_last();
    const uint8_t* snap = b.snap + b.frame_stride * blockIdx.z;
    uint8_t* out = b.out + b.frame_stride * blockIdx.z;
    heuristics_tile<NT, false, VOTE>(snap, out, b.w, b.h, blockIdx.x * kHTW, blockIdx.y * kHTH,
                                 L ? L + b.frame_stride * blockIdx.z : nullptr);
}

// the same with the graph windows by TMA (width and frame stride multiples of
// 16 bytes, 16-byte aligned base)
template <bool VOTE, int NT>
__global__ void __launch_bounds__(NT) k_heuristics_tma(GraphBatch b, int32_t* L, const __grid_constant__ CUtensorMap map)
{
    follow_last();
    const uint8_t* snap = b.snap + b.frame_stride * blockIdx.z;
    uint8_t* out = b.out + b.frame_stride * blockIdx.z;
    heuristics_tile<NT, true, VOTE>(snap, out, b.w, b.h, blockIdx.x * kHTW, blockIdx.y * kHTH,
                                L ? L + b.frame_stride * blockIdx.z : nullptr, &map, (int)blockIdx.z);
}

// -------------------------------------------------- component labelling

// lock-free union with the smaller root winning: the final root of every
// component is its minimum index
__device__ __forceinline__ void uf_unite(int32_t* L, int a, int b)
{
    for (;;) {
        // both finds' loads in flight together
        int pa = L[a], pb = L[b];
        while (pa != a || pb != b) {
            a = pa;
            b = pb;
            pa = L[a];
            pb = L[b];
        }
        if (a == b) return;
        if (a > b) {
            int t = a;
            a = b;
            b = t;
        }
        int old = atomicMin(&L[b], a);
        if (old == b) return;
        b = old;
    }
}

// Component labels in three passes: union-find inside tiles in shared memory
// (local roots are the tile-local minima, which are also the minima in global
// index order), then unions across tile borders on the global label array,
// then one flattening pass. The frame and batch paths make the tile-local
// labels inside the 64x16 heuristics tiles (tile_labels), merge with
// merge_tile_borders and flatten in the raster's tiles (flatten_tile), or with
// k_cc_flatten where no mask raster follows; the stage API
// (depix_label_components) runs its own 32x32 tiles over a graph in global memory (cc_local_core: a warp
// owns a row, horizontal runs from one ballot, one union per pair of touching
// runs).
constexpr int kLT = 32;

// find with path compression, for the passes that follow the unions (no
// union in flight: every parent lowered is lowered to its final root)
__device__ __forceinline__ int s_find(int* L, int x)
{
    int r = x;
    while (L[r] != r) r = L[r];
    while (L[x] > r) {
        int nx = L[x];
        atomicMin(&L[x], r);
        x = nx;
    }
    return r;
}

// root without compression, for the unions themselves
__device__ __forceinline__ int s_root(const int* L, int x)
{
    while (L[x] != x) x = L[x];
    return x;
}

// Lock-free union, the smaller root winning. Its finds do not compress:
// with compression interleaved with the unions of other threads, joins
// were lost on the GPU (tile-local labels of 4096-sprite batches wrong in
// about one tile in 10^5, one in 10^4 with volatile loads; none in 560
// batches, 6.2 million tiles, without it).
__device__ __forceinline__ void s_unite(int* L, int a, int b)
{
    for (;;) {
        a = s_root(L, a);
        b = s_root(L, b);
        if (a == b) return;
        if (a > b) {
            int t = a;
            a = b;
            b = t;
        }
        int old = atomicMin(&L[b], a);
        if (old == b) return;
        b = old;
    }
}

// position of the set bit of rank j (from 0, counted from bit 0) of m;
// j < popcount(m)
__device__ __forceinline__ int nth_set_bit64(uint64_t m, int j)
{
    const unsigned lo = (unsigned)m;
    const int nlo = __popc(lo);
    return j < nlo ? (int)__fns(lo, 0, j + 1) : 32 + (int)__fns((unsigned)(m >> 32), 0, j - nlo + 1);
}

// 64-bit row mask from the ballots of a warp's two 32-pixel segments
__device__ __forceinline__ uint64_t ballot64(bool lo, bool hi)
{
    return (uint64_t)__ballot_sync(0xFFFFFFFFu, lo) | (uint64_t)__ballot_sync(0xFFFFFFFFu, hi) << 32;
}

// the run start at or before position c of a line whose run starts are S
__device__ __forceinline__ int run_start(uint64_t S, int c) { return 63 - __clzll(S & (~0ull >> (63 - c))); }

// Which edges between two lines of at most 64 pixels, r and q, need a union
// when the pixels joined along each line are already one set. Edge e at
// position c joins r[c] and q[c + e - 1]; Sr and Sq mark where the lines'
// runs start; q_end marks positions past the end of q (another tile, so
// another set). An edge is skipped where another edge joins the same two
// runs: an e = 1 edge defers to the e = 1 edge one position before it, an
// e = 0 edge to the e = 0 or e = 1 edge one position before it, an e = 2
// edge to the e = 2 edge one position before it or the e = 1 edge one
// position after it, each when both runs are the same there. Every chain of
// deferrals ends at an edge that is kept (e = 0 and e = 1 edges defer only
// to lower positions, and an e = 2 edge to a lower position or to an e = 1
// edge), so the kept edges join the same sets as all of them.
__device__ __forceinline__ uint64_t join_mask(int e, uint64_t Sr, uint64_t Sq, uint64_t E0, uint64_t E1, uint64_t E2,
                                              uint64_t q_end)
{
    if (e == 0) return E0 & ~(~Sr & (((E0 & ~Sq) << 1) | (E1 << 1)));
    if (e == 1) return E1 & ~((E1 << 1) & ~Sr & ~Sq);
    return E2 & ~(((E2 << 1) & ~Sr & ~((Sq >> 1) | q_end)) | ((E1 & ~Sr) >> 1));
}
__device__ __forceinline__ void join_masks(uint64_t Sr, uint64_t Sq, uint64_t E0, uint64_t E1, uint64_t E2,
                                           uint64_t q_end, uint64_t (&need)[3])
{
#pragma unroll
    for (int e = 0; e < 3; e++) need[e] = join_mask(e, Sr, Sq, E0, E1, E2, q_end);
}

// fn(e, c) for every set bit c of need[e], spread over the warp's lanes
// (one union per lane in turn)
template <typename Fn>
__device__ __forceinline__ void for_each_join(const uint64_t (&need)[3], Fn fn)
{
    const int lane = threadIdx.x & 31;
    const int n0 = __popcll(need[0]), n01 = n0 + __popcll(need[1]), n = n01 + __popcll(need[2]);
    for (int i = lane; i < n; i += 32) {
        const int e = i < n0 ? 0 : i < n01 ? 1 : 2;
        const uint64_t m = e == 0 ? need[0] : e == 1 ? need[1] : need[2];
        fn(e, nth_set_bit64(m, i - (e == 0 ? 0 : e == 1 ? n0 : n01)));
    }
}

// Component labels of a 64x16 tile of a symmetric graph (each edge held by
// both of its nodes, as in the resolved graph; 0 outside the image), as global
// indices of the tile-local roots. A run's parent is kept at its leftmost
// pixel. The rows' run starts and upward edges become 64-bit masks, eight columns
// a thread: a product gathers a bit of four packed bytes at once. A lane then
// lists the edges of one kind between half a row and the row above it that
// join_mask keeps (three warps, one a kind); all threads unite along the listed
// edges, one each (a lane that united its own edges in turn waited
// for a chain of finds per edge: 8.4 k cycles of a tile's 26 k); then the
// listed runs, which are all that are not their own root, are pointed at their
// roots, and each pixel reads its run's parent (following the chains from
// there cost 6.8 k cycles).
template <int NT>
__device__ void tile_labels(const uint8_t (*node)[kHTW], uint16_t* joins, int32_t* L, int w, int h, int x0, int y0)
{
    static_assert(kHTW == 64 && kHTH == 16 && NT >= 128, "lanes of the joins");
    __shared__ __align__(16) int sl[kHTH * kHTW];
    __shared__ uint64_t rows[4][kHTH]; // run starts, up-left, up, up-right edges
    __shared__ int njoins;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) njoins = 0;
    if (NT == 128 || threadIdx.x < 128) {
        // eight columns a thread: bit planes of its two words as bytes of the
        // row masks (the product gathers a word's four bits in its top byte)
        const int r = threadIdx.x >> 3, g = threadIdx.x & 7;
        const uint2 v = *reinterpret_cast<const uint2*>(&node[r][8 * g]);
        auto plane = [&](int bit) -> unsigned {
            return ((v.x >> bit & 0x01010101u) * 0x01020408u >> 24) | ((v.y >> bit & 0x01010101u) * 0x01020408u >> 24) << 4;
        };
        const unsigned first = g == 0, last = g == 7 ? 0x80u : 0u;
        auto put = [&](int k, unsigned m) { reinterpret_cast<uint8_t*>(&rows[k][r])[g] = (uint8_t)m; };
        put(0, ~plane(3) | first);
        put(1, plane(0) & ~first); // edges within the tile
        put(2, plane(1));
        put(3, plane(2) & ~last);
        const int p = 8 * threadIdx.x;
        int4* q = reinterpret_cast<int4*>(&sl[p]);
        q[0] = make_int4(p, p + 1, p + 2, p + 3);
        q[1] = make_int4(p + 4, p + 5, p + 6, p + 7);
    }
    __syncthreads();
    // joins as position in the tile | kind << 10
    if (warp < 3 && lane < 2 * (kHTH - 1)) {
        const int r = lane >> 1, half = lane & 1;
        const uint64_t need = join_mask(warp, rows[0][r], rows[0][r + 1], rows[1][r], rows[2][r], rows[3][r], 1ull << 63);
        uint32_t m = (uint32_t)(need >> (32 * half));
        int slot = m ? atomicAdd(&njoins, __popc(m)) : 0;
        while (m) {
            joins[slot++] = (uint16_t)(r * kHTW + 32 * half + __ffs(m) - 1 | warp << 10);
            m &= m - 1;
        }
    }
    __syncthreads();
    const int n = njoins;
    auto runs = [&](int i, int& a, int& b) {
        const int p = joins[i] & 1023, e = joins[i] >> 10, r = p / kHTW, c = p % kHTW;
        a = r * kHTW + run_start(rows[0][r], c);
        b = (r + 1) * kHTW + run_start(rows[0][r + 1], c + e - 1);
    };
    for (int i = threadIdx.x; i < n; i += NT) {
        int a, b;
        runs(i, a, b);
        s_unite(sl, a, b);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += NT) {
        int a, b;
        runs(i, a, b);
        // no union in flight: both ends have one root, and a store only ever
        // shortens another thread's way to it
        const int root = s_root(sl, a);
        sl[a] = root;
        sl[b] = root;
    }
    __syncthreads();
    // four pixels a thread: their runs' roots, stored at once where the row allows
    const bool wide = ((w | x0 | (int)(reinterpret_cast<uintptr_t>(L) >> 2)) & 3) == 0;
#pragma unroll
    for (int k = threadIdx.x; k < kHTW / 4 * kHTH; k += NT) {
        const int r = k / (kHTW / 4), c = 4 * (k % (kHTW / 4)), x = x0 + c, y = y0 + r;
        const uint64_t S = rows[0][r];
        int run = run_start(S, c);
        const unsigned s4 = (unsigned)(S >> c);
        int lab[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (q && (s4 >> q & 1u)) run = c + q;
            const int root = sl[r * kHTW + run];
            lab[q] = (y0 + root / kHTW) * w + x0 + root % kHTW;
        }
        if (y >= h || x >= w) continue;
        int32_t* o = L + (size_t)y * w + x;
        if (wide) {
            *reinterpret_cast<int4*>(o) = make_int4(lab[0], lab[1], lab[2], lab[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (x + q < w) o[q] = lab[q];
        }
    }
}

// Union-find over a TW x TH tile whose graph bytes are in shared memory (sg,
// row-major, 0 outside the image): local roots as global indices. A warp
// owns a row and walks its 32-pixel segments left to right: horizontal runs
// from one ballot per segment (a run's root is its leftmost pixel, carried
// across segments), rows joined with one union per pair of touching runs.
template <int TW, int TH>
__device__ void cc_local_core(const uint8_t* sg, int* sl, uint16_t* run, int32_t* L, int w, int h, int x0, int y0)
{
    static_assert(TW % 32 == 0 && TW * TH <= 65536, "tile shape");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int r = warp; r < TH; r += nwarp) {
        int carry = r * TW;
#pragma unroll
        for (int sgm = 0; sgm < TW / 32; sgm++) {
            const int c = sgm * 32 + lane, p = r * TW + c;
            const bool link = c > 0 && (bitof(sg[p], 3) || bitof(sg[p - 1], 4));
            const unsigned starts = __ballot_sync(0xFFFFFFFFu, !link);
            const unsigned upto = lane == 31 ? starts : (starts & ((2u << lane) - 1u));
            const int root = upto ? r * TW + sgm * 32 + (31 - __clz(upto)) : carry;
            run[p] = (uint16_t)root;
            sl[p] = root;
            carry = __shfl_sync(0xFFFFFFFFu, root, 31);
        }
    }
    __syncthreads();
    for (int r = warp; r < TH - 1; r += nwarp) {
#pragma unroll
        for (int sgm = 0; sgm < TW / 32; sgm++) {
            const int c = sgm * 32 + lane, p = r * TW + c;
            const unsigned node = sg[p];
#pragma unroll
            for (int e = 0; e <= 2; e++) { // up-left, up, up-right
                const int nc = c + dir_di(e);
                if (nc < 0 || nc >= TW) continue;
                const int q = p + TW + dir_di(e);
                if (!(bitof(node, e) || bitof(sg[q], 7 - e))) continue;
                // the pixel to the left already joins the same two runs
                if (c > 0 && nc > 0 && run[p - 1] == run[p] && run[q - 1] == run[q] &&
                    (bitof(sg[p - 1], e) || bitof(sg[q - 1], 7 - e)))
                    continue;
                s_unite(sl, run[p], run[q]);
            }
        }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < TW * TH; p += blockDim.x) {
        const int x = x0 + p % TW, y = y0 + p / TW;
        if (x >= w || y >= h) continue;
        const int r = s_find(sl, p);
        L[(size_t)y * w + x] = (y0 + r / TW) * w + (x0 + r % TW);
    }
}

// union-find inside one 32x32 tile (x0, y0) of a graph in global memory
__device__ void cc_local_tile(const uint8_t* g, int32_t* L, int w, int h, int x0, int y0)
{
    __shared__ int sl[kLT * kLT];
    __shared__ uint16_t run[kLT * kLT];
    __shared__ uint8_t sg[kLT * kLT];
    for (int p = threadIdx.x; p < kLT * kLT; p += blockDim.x) {
        int x = x0 + p % kLT, y = y0 + p / kLT;
        sg[p] = (x < w && y < h) ? g[(size_t)y * w + x] & inside_mask(x, y, w, h) : 0;
    }
    __syncthreads();
    cc_local_core<kLT, kLT>(sg, sl, run, L, w, h, x0, y0);
}

__global__ void __launch_bounds__(256) k_cc_local(const uint8_t* g, int32_t* L, int w, int h, size_t frame_stride)
{
    cc_local_tile(g + frame_stride * blockIdx.z, L + frame_stride * blockIdx.z, w, h, blockIdx.x * kLT,
                  blockIdx.y * kLT);
}

// unions across tile borders: every set bit whose neighbour lies in another
// tile (each symmetric pair is seen from both ends; uniting twice is
// harmless). One thread per border pixel of a tile (4 * 32 - 4 of them).
constexpr int kLBorder = 4 * kLT - 4;

// unions of border pixel q (of 4 kLT - 4) of tile `tile` in the kLT x kLT
// tiling with neighbours in other tiles
__device__ __forceinline__ void cc_merge_border(const uint8_t* g, int32_t* L, int w, int h, int tile, int q)
{
    constexpr int TW = kLT, TH = kLT;
    const int tiles_x = (w + TW - 1) / TW;
    // border position q: bottom row, top row, then left and right columns
    int lx, ly;
    if (q < TW) { lx = q; ly = 0; }
    else if (q < 2 * TW) { lx = q - TW; ly = TH - 1; }
    else if (q < 2 * TW + TH - 2) { lx = 0; ly = q - 2 * TW + 1; }
    else { lx = TW - 1; ly = q - (2 * TW + TH - 2) + 1; }
    const int i = (tile % tiles_x) * TW + lx, j = (tile / tiles_x) * TH + ly;
    if (i >= w || j >= h) return;
    const int k = j * w + i;
    unsigned node = g[k];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        if (!bitof(node, e)) continue;
        int ni = i + dir_di(e), nj = j + dir_dj(e);
        if (ni < 0 || nj < 0 || ni >= w || nj >= h) continue;
        if (ni / TW == i / TW && nj / TH == j / TH) continue;
        uf_unite(L, k, nj * w + ni);
    }
}

// Unions across two borders of the 64x16 tile (tx, ty) of a symmetric
// graph, by one warp. Rows y0 + 15 and y0 + 16: the edges from row y0 + 15
// to (x - 1, y + 1), (x, y + 1), (x + 1, y + 1), the first reaching from
// column x0 into the tile at (tx - 1, ty + 1) and the last from column
// x0 + 63 into (tx + 1, ty + 1). Columns x0 + 63 and x0 + 64 over rows
// y0 .. y0 + 15 (runs along the columns: the pixels joined by their (x, y + 1)
// edge): the edges (x + 1, y) of every row, (x + 1, y + 1) of rows y0 ..
// y0 + 14 and, from column x0 + 64, (x - 1, y + 1) of those rows; the two
// diagonals from row y0 + 15 belong to the row pairs of this tile and of
// tile (tx + 1, ty). Every cross-tile pair is joined by exactly one tile, and
// of the edges between the same two runs only one (join_masks).
// unite(a, b) joins the sets of pixels a and b (frame indices); rows, columns:
// which of the two borders.
template <typename Unite>
__device__ void merge_tile_borders(const uint8_t* g, int w, int h, int tx, int ty, bool rows, bool columns, Unite unite)
{
    const int lane = threadIdx.x & 31;
    const int x0 = tx * kHTW, y0 = ty * kHTH;
    const int yr = y0 + kHTH - 1, yq = yr + 1;
    if (rows && yq < h) {
        unsigned a[2], b[2];
#pragma unroll
        for (int sgm = 0; sgm < 2; sgm++) {
            const int x = x0 + 32 * sgm + lane;
            a[sgm] = x < w ? g[(size_t)yr * w + x] & inside_mask(x, yr, w, h) : 0u;
            b[sgm] = x < w ? g[(size_t)yq * w + x] & inside_mask(x, yq, w, h) : 0u;
        }
        const uint64_t Sr = ballot64(lane == 0 || !bitof(a[0], 3), !bitof(a[1], 3));
        const uint64_t Sq = ballot64(lane == 0 || !bitof(b[0], 3), !bitof(b[1], 3));
        uint64_t need[3];
        join_masks(Sr, Sq, ballot64(bitof(a[0], 0), bitof(a[1], 0)), ballot64(bitof(a[0], 1), bitof(a[1], 1)),
                   ballot64(bitof(a[0], 2), bitof(a[1], 2)), 1ull << 63, need);
        for_each_join(need, [&](int e, int c) {
            const int nc = c + e - 1, qc = nc < 0 || nc >= kHTW ? nc : run_start(Sq, nc);
            unite(yr * w + x0 + run_start(Sr, c), yq * w + x0 + qc);
        });
    }
    const int xr = x0 + kHTW - 1, xq = xr + 1;
    if (columns && xq < w) {
        const int y = y0 + lane;
        unsigned a = 0, b = 0;
        if (lane < kHTH && y < h) {
            a = g[(size_t)y * w + xr] & inside_mask(xr, y, w, h);
            b = g[(size_t)y * w + xq] & inside_mask(xq, y, w, h);
        }
        // runs along the columns: row y starts one unless row y - 1 links up
        const uint64_t Sr = ~((uint64_t)__ballot_sync(0xFFFFFFFFu, bitof(a, 1)) << 1);
        const uint64_t Sq = ~((uint64_t)__ballot_sync(0xFFFFFFFFu, bitof(b, 1)) << 1);
        const uint64_t E1 = __ballot_sync(0xFFFFFFFFu, bitof(a, 4));
        const uint64_t E2 = __ballot_sync(0xFFFFFFFFu, bitof(a, 2)) & 0x7FFFu;
        const uint64_t E0 = (uint64_t)(__ballot_sync(0xFFFFFFFFu, bitof(b, 0)) & 0x7FFFu) << 1;
        uint64_t need[3];
        join_masks(Sr, Sq, E0, E1, E2, 1ull << 63, need);
        for_each_join(need, [&](int e, int c) {
            unite((y0 + run_start(Sr, c)) * w + xr, (y0 + run_start(Sq, c + e - 1)) * w + xq);
        });
    }
}

// the same on the global labels
__device__ __forceinline__ void cc_merge_tile_warp(const uint8_t* g, int32_t* L, int w, int h, int tx, int ty, bool rows,
                                                   bool columns)
{
    merge_tile_borders(g, w, h, tx, ty, rows, columns, [&](int a, int b) { uf_unite(L, a, b); });
}

// two warps per 64x16 tile, one per border: the unions are chains of global
// loads, and the two borders' run at once (8 frames of 256x224: 10.5 us when one
// warp did both and each union's finds ran one after the other, 8.5 now)
__global__ void __launch_bounds__(128) k_cc_merge_tiles(const uint8_t* g, int32_t* L, int w, int h, size_t frame_stride)
{
    follow_last();
    const int tiles_x = (w + kHTW - 1) / kHTW, tiles = tiles_x * ((h + kHTH - 1) / kHTH);
    const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), t = k >> 1;
    if (t >= tiles) return;
    cc_merge_tile_warp(g + frame_stride * blockIdx.z, L + frame_stride * blockIdx.z, w, h, t % tiles_x,
                       t / tiles_x, !(k & 1), k & 1);
}

__global__ void k_cc_merge(const uint8_t* g, int32_t* L, int w, int h, size_t frame_stride)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int tiles = ((w + kLT - 1) / kLT) * ((h + kLT - 1) / kLT);
    if (t / kLBorder >= tiles) return;
    cc_merge_border(g + frame_stride * blockIdx.z, L + frame_stride * blockIdx.z, w, h, t / kLBorder, t % kLBorder);
}

// the roots of all labels, where no raster follows that makes them
__global__ void k_cc_flatten(int32_t* L, int n, size_t frame_stride)
{
    follow_last();
    const int k = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= n) return;
    L += frame_stride * blockIdx.z;
    flatten4(L, L + k, min(4, n - k));
}

// ------------------------------------------------ uneven batches (queue)

__global__ void __launch_bounds__(kGThreads) k_graph_queue(QueueBatch q)
{
    const QueueHeader* H = q.hdr;
    const int n = H->n;
    queue_loop(q.counters + QC_GRAPH, (int)H->total[QS_GRAPH], q.gran[QS_GRAPH], [&](int t) {
        const uint32_t* base = H->base + QS_GRAPH * (n + 1);
        const int f = queue_frame(base, n, (uint32_t)t);
        const QueueFrame fr = H->frames[f];
        const int lt = t - (int)base[f], tx = (fr.w + kGTW - 1) / kGTW;
        FrameRef ref{H->img + fr.in_off, fr.w, fr.h, 4 * fr.w, q.graph_a + fr.px_off};
        graph_tile<DEPIX_LAYOUT_RGBA, kGStripQueue>(ref, (lt % tx) * kGTW, (lt / tx) * 4 * kGStripQueue, H->thr, true);
    });
}

template <bool VOTE>
__global__ void __launch_bounds__(kHThreads) k_heur_queue(QueueBatch q)
{
    const QueueHeader* H = q.hdr;
    const int n = H->n;
    queue_loop(q.counters + QC_HEUR, (int)H->total[QS_HEUR], q.gran[QS_HEUR], [&](int t) {
        const uint32_t* base = H->base + QS_HEUR * (n + 1);
        const int f = queue_frame(base, n, (uint32_t)t);
        const QueueFrame fr = H->frames[f];
        const int lt = t - (int)base[f], tx = (fr.w + kHTW - 1) / kHTW;
        heuristics_tile<kHThreads, false, VOTE>(q.graph_a + fr.px_off, q.graph_b + fr.px_off, fr.w, fr.h, (lt % tx) * kHTW,
                                     (lt / tx) * kHTH, H->labels ? H->labels + fr.px_off : nullptr);
    });
}


__global__ void __launch_bounds__(128) k_label_merge_queue(QueueBatch q)
{
    // the local labels came with the heuristics stage: its tiles
    const QueueHeader* H = q.hdr;
    const int n = H->n;
    warp_queue_loop(q.counters + QC_MERGE, (int)H->total[QS_LABEL], q.gran[QS_LABEL], [&](int t) {
        const uint32_t* base = H->base + QS_LABEL * (n + 1);
        const int f = queue_frame(base, n, (uint32_t)t);
        const QueueFrame fr = H->frames[f];
        const int lt = t - (int)base[f], tx = (fr.w + kHTW - 1) / kHTW;
        cc_merge_tile_warp(q.graph_b + fr.px_off, H->labels + fr.px_off, fr.w, fr.h, lt % tx, lt / tx, true, true);
    });
}

cudaError_t queue_graph(const QueueBatch& q, int blocks, cudaStream_t s)
{
    k_graph_queue<<<blocks, kGThreads, 0, s>>>(q);
    return cudaGetLastError();
}

cudaError_t queue_heuristics(const QueueBatch& q, int blocks, cudaStream_t s)
{
    if (q.vote) k_heur_queue<true><<<blocks, kHThreads, 0, s>>>(q);
    else k_heur_queue<false><<<blocks, kHThreads, 0, s>>>(q);
    return cudaGetLastError();
}

cudaError_t queue_labels(const QueueBatch& q, int blocks, cudaStream_t s)
{
    // local labels were made by the heuristics stage; the raster makes the roots
    k_label_merge_queue<<<blocks, 128, 0, s>>>(q);
    return cudaGetLastError();
}

static_assert(kQGraphTW == kGTW && kQGraphTH == 4 * kGStripQueue, "graph queue tile");
static_assert(kQHeurTW == kHTW && kQHeurTH == kHTH, "heuristics queue tile");

template <typename K>
static int occupancy(K kernel, int threads)
{
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, 0) != cudaSuccess) return 0;
    return nb;
}

int queue_blocks_per_sm(int stage, const QueueBatch& q)
{
    switch (stage) {
    case QS_GRAPH: return occupancy(k_graph_queue, kGThreads);
    case QS_HEUR: return q.vote ? occupancy(k_heur_queue<true>, kHThreads) : occupancy(k_heur_queue<false>, kHThreads);
    case QS_LABEL: return occupancy(k_label_merge_queue, 128);
    default: return queue_raster_blocks_per_sm(q);
    }
}

__global__ void k_yuv_words(const uint8_t* px3, size_t n, int mode, uint32_t* out)
{
    size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    out[k] = yuv_word(px3[3 * k], px3[3 * k + 1], px3[3 * k + 2], mode);
}

// ----------------------------------------------------------------- launch

cudaError_t launch_yuv_words(const uint8_t* px3, size_t n, int mode, uint32_t* out, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_yuv_words<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(px3, n, mode, out);
    return cudaGetLastError();
}

cudaError_t set_graph_tma_timeout_test(int on)
{
    int v = on ? 1 : 0;
    return cudaMemcpyToSymbol(g_graph_tma_timeout_test, &v, sizeof(int));
}

cudaError_t take_graph_fault(int* out)
{
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_graph_fault, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_graph_fault, &zero, sizeof(int));
    return e;
}

template <int GH>
static cudaError_t launch_graph_t(const FrameBatch& b, int nframes, uint32_t thr, bool fuse_trivial, cudaStream_t s)
{
    dim3 grid((b.w + kGTW - 1) / kGTW, (b.h + 4 * GH - 1) / (4 * GH), nframes);
    CUtensorMap map;
    if (b.layout == DEPIX_LAYOUT_RGBA &&
        rgba_tensor_map(b.img, b.w, b.h, b.ws, b.img_stride, nframes, kGBoxW, 4 * GH + 2, &map))
        k_graph_tma<GH><<<grid, kGThreads, 0, s>>>(b, thr, fuse_trivial ? 1 : 0, map);
    else if (b.layout == DEPIX_LAYOUT_RGBA)
        k_graph<DEPIX_LAYOUT_RGBA, GH><<<grid, kGThreads, 0, s>>>(b, thr, fuse_trivial ? 1 : 0);
    else
        k_graph<DEPIX_LAYOUT_BGR, GH><<<grid, kGThreads, 0, s>>>(b, thr, fuse_trivial ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_graph(const FrameBatch& b, int nframes, uint32_t thr, bool fuse_trivial, cudaStream_t s)
{
    const long long px = (long long)b.w * b.h * nframes;
    // tiles of four rows only where grid.y takes them all (one column of 2^18 rows has one too many)
    if (px <= 1 << 18 && b.h <= 65535 * 4 * kGStripFrame) return launch_graph_t<kGStripFrame>(b, nframes, thr, fuse_trivial, s);
    if (px <= 1 << 21) return launch_graph_t<kGStripSmall>(b, nframes, thr, fuse_trivial, s);
    return launch_graph_t<kGStrip>(b, nframes, thr, fuse_trivial, s);
}

cudaError_t launch_trivial(uint8_t* g, int w, int h, cudaStream_t s)
{
    dim3 blk(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    k_trivial<<<grid, blk, 0, s>>>(g, w, h);
    return cudaGetLastError();
}

template <int NT>
static cudaError_t heuristics_t(bool tma, bool early, dim3 grid, cudaStream_t s, const GraphBatch& b, int32_t* labels,
                                const CUtensorMap& map)
{
    if (tma)
        return launch_early(early, b.vote ? k_heuristics_tma<true, NT> : k_heuristics_tma<false, NT>, grid, NT, 0, s, b,
                            labels, map);
    return launch_early(early, b.vote ? k_heuristics<true, NT> : k_heuristics<false, NT>, grid, NT, 0, s, b, labels);
}

cudaError_t launch_heuristics(const GraphBatch& b, int nframes, int32_t* labels, cudaStream_t s)
{
    dim3 grid((b.w + kHTW - 1) / kHTW, (b.h + kHTH - 1) / kHTH, nframes);
    const bool early = early_stages((long long)b.w * b.h * nframes);
    CUtensorMap map;
    const bool tma = u8_tensor_map(b.snap, b.w, b.h, b.frame_stride, nframes, kHRW, kHRH, &map);
    const long long tiles = (long long)grid.x * grid.y * nframes, sms = sm_count();
    if (tiles <= kTilesPerSm512 * sms) return heuristics_t<512>(tma, early, grid, s, b, labels, map);
    if (tiles <= kTilesPerSm256 * sms) return heuristics_t<256>(tma, early, grid, s, b, labels, map);
    return heuristics_t<kHThreads>(tma, early, grid, s, b, labels, map);
}

cudaError_t take_heuristics_fault(int* out)
{
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_heur_fault, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_heur_fault, &zero, sizeof(int));
    return e;
}

cudaError_t launch_labels_after_heuristics(const uint8_t* g, int32_t* labels, int w, int h, int nframes,
                                          size_t frame_stride, bool flatten, cudaStream_t s)
{
    const int n = w * h;
    const int tiles = ((w + kHTW - 1) / kHTW) * ((h + kHTH - 1) / kHTH);
    const bool early = early_stages((long long)n * nframes);
    const cudaError_t e =
        launch_early(early, k_cc_merge_tiles, dim3((tiles + 1) / 2, 1, nframes), 128, 0, s, g, labels, w, h, frame_stride);
    return e == cudaSuccess && flatten
               ? launch_early(early, k_cc_flatten, dim3((n + 1023) / 1024, 1, nframes), 256, 0, s, labels, n, frame_stride)
               : e;
}

cudaError_t launch_labels(const uint8_t* g, int32_t* labels, int w, int h, int nframes, size_t frame_stride,
                          cudaStream_t s)
{
    int n = w * h;
    dim3 tiles((w + kLT - 1) / kLT, (h + kLT - 1) / kLT, nframes);
    k_cc_local<<<tiles, 256, 0, s>>>(g, labels, w, h, frame_stride);
    const int borders = tiles.x * tiles.y * kLBorder;
    k_cc_merge<<<dim3((borders + 127) / 128, 1, nframes), 128, 0, s>>>(g, labels, w, h, frame_stride);
    dim3 grid((n + 1023) / 1024, 1, nframes);
    k_cc_flatten<<<grid, 256, 0, s>>>(labels, n, frame_stride);
    return cudaGetLastError();
}

}  // namespace depix
