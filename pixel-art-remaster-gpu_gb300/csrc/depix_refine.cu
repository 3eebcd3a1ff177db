// depix_refine.cu -- spline refinement: node positions of the colour
// boundaries optimised against curvature, deviation and a soft-coverage
// raster loss, with a hand-written adjoint.
//
// The reference has no such stage (its frame path ends at the VBO fill,
// kernel.cu:439-520). Its definition here:
//
// Topology, extracted once per frame and frozen:
//   * cells are the hulls of the resolved graph's cell patterns (the hull
//     table); split at every hull vertex lying inside an edge, the cells'
//     edges pair up exactly with reversed twins in 8-neighbour cells;
//   * a split edge whose twin belongs to a dissimilar cell is a curve edge,
//     kept once (from the lower-indexed cell, along its counter-clockwise
//     hull: its colour on the left);
//   * nodes are curve-edge vertices in global quarter-pixel units, numbered
//     in vertex-grid order; pinned when not of degree 2, on an edge without
//     a twin (the frame), or where the two edges turn by 90 degrees or more;
//   * one Chaikin round gives the segments: the middle of each edge (slot
//     3e+1), the piece from a pinned end to the first cut point (3e, 3e+2)
//     and the cut corner of each free node (3E + node);
//   * every output sample within 1.5 output pixels of a segment is assigned
//     to the nearest one (distances in whole numbers; ties to the lower
//     slot).
// Energy (every term a mean): w_curv * 1/F sum_free |a - 2p + b|^2 / 8
//   + w_dev * 1/F sum_free |p - p0|^2
//   + w_cov * 1/(3 Ws Hs) sum_samples sum_rgb ((r - t)/255)^2,
//   r = cR + (cL - cR) Phi(d / sigma), d the sample's signed distance from
//   its segment's line, t the nearest-neighbour target under the same
//   Gaussian coverage. The adjoint recomputes each segment's Chaikin points
//   from the nodes in the backward pass instead of storing them.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "depix_internal.h"

namespace depix {

namespace {

constexpr int kBand = 48;          // 1.5 output pixels in 1/(32 s) source pixel
constexpr int kMaxRefineScale = 12;
enum SegType { SEG_NONE = 0, SEG_MID = 1, SEG_PIN_U = 2, SEG_PIN_V = 3, SEG_CORNER = 4 };
// weights (x4) of a segment's ends over its three node slots, per type, as
// 4-bit fields (type * 12 + slot * 4): A {-, 3 1 0, 4 0 0, 1 3 0, 1 3 0},
// B {-, 1 3 0, 3 1 0, 0 4 0, 0 3 1}
constexpr unsigned long long kSegWA = 0x031031004013000ull;
constexpr unsigned long long kSegWB = 0x130040013031000ull;
__host__ __device__ constexpr int seg_wa(int type, int k) { return (int)((kSegWA >> (type * 12 + k * 4)) & 0xF); }
__host__ __device__ constexpr int seg_wb(int type, int k) { return (int)((kSegWB >> (type * 12 + k * 4)) & 0xF); }
static_assert(seg_wa(1, 0) == 3 && seg_wa(1, 1) == 1 && seg_wa(2, 0) == 4 && seg_wa(3, 1) == 3 && seg_wa(4, 1) == 3,
              "segment weights A");
static_assert(seg_wb(1, 1) == 3 && seg_wb(2, 0) == 3 && seg_wb(2, 1) == 1 && seg_wb(3, 1) == 4 && seg_wb(4, 2) == 1 &&
              seg_wb(4, 1) == 3 && seg_wb(4, 0) == 0, "segment weights B");

// vertex grid word: bit 0 a hull vertex, bit 1 on an edge without a twin,
// bits 8.. the number of curve edges
constexpr uint32_t kVUsed = 1, kVFrame = 2;
constexpr int kDegShift = 8;

// ---------------------------------------------------------------- scans

constexpr int kScanBlock = 1024, kScanItems = 4, kScanTile = kScanBlock * kScanItems;

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s; // inclusive
    }
    __syncthreads();
    const T base = warp > 0 ? warp_sums[warp - 1] : T(0);
    __syncthreads();
    return base + x - v;
}

// An exclusive scan left in two parts: out within tiles of kScanTile, and the
// tiles' own sums before them. Readers add the two (at), which spares a pass
// over the array.
template <typename T>
struct Scan {
    T* out;
    T* tiles;
    T* total;
    int* ticket; // zero between scans
    __device__ __forceinline__ T at(int k) const { return out[k] + tiles[k / kScanTile]; }
};

// Exclusive scan of load(0) .. load(n - 1) in one launch: every block scans its
// tile, the last one to finish scans the tiles' sums (none waits for another).
template <typename T, typename Load>
__global__ void __launch_bounds__(kScanBlock) k_scan(Load load, int n, Scan<T> S)
{
    follow_last();
    __shared__ T ws[32];
    __shared__ int last;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    T v[kScanItems], s = T(0);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? load(base + k) : T(0);
        s += v[k];
    }
    T ex = block_exclusive_scan(s, ws);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) S.out[base + k] = ex;
        ex += v[k];
    }
    if (threadIdx.x == blockDim.x - 1) {
        S.tiles[blockIdx.x] = ex;
        __threadfence();
        last = atomicAdd(S.ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    T carry = T(0);
    for (int b = 0; b < (int)gridDim.x; b += kScanBlock) {
        const int k = b + threadIdx.x;
        const T t = k < (int)gridDim.x ? __ldcg(S.tiles + k) : T(0);
        const T e = block_exclusive_scan(t, ws);
        if (k < (int)gridDim.x) S.tiles[k] = carry + e;
        if (threadIdx.x == blockDim.x - 1) ws[0] = e + t;
        __syncthreads();
        carry += ws[0];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *S.total = carry;
        *S.ticket = 0;
    }
}

template <typename T, typename Load>
cudaError_t exclusive_scan(Load load, int n, const Scan<T>& S, cudaStream_t s)
{
    return launch_early(true, k_scan<T, Load>, std::max(1, (n + kScanTile - 1) / kScanTile), kScanBlock, 0, s, load, n, S);
}

struct Geo {
    const uint8_t* img;
    int ws, layout;
    const uint8_t* g;
    int w, h;
    int gw, gh;         // vertex grid: (4w + 3) x (4h + 3), origin at quarter (-1, -1)
    const uint64_t* lut;
    const uint32_t* box; // per-pattern hull boxes (k_rf_boxes)
    uint32_t thr;
};

__device__ __forceinline__ uint64_t cell_hull(const Geo& G, int idx)
{
    const int n = G.w * G.h;
    const unsigned node = G.g[idx];
    const unsigned left = idx > 0 ? G.g[idx - 1] : 0u;
    const unsigned right = idx + 1 < n ? G.g[idx + 1] : 0u;
    return __ldg(&G.lut[cell_pattern(node, left, right)]);
}

// hull vertex t in global quarter units
__device__ __forceinline__ int qvx(uint64_t e, int t, int i) { return 4 * i + (int)((e >> (4 + 6 * t)) & 7u) - 1; }
__device__ __forceinline__ int qvy(uint64_t e, int t, int j) { return 4 * j + (int)((e >> (7 + 6 * t)) & 7u) - 1; }
__device__ __forceinline__ int vindex(const Geo& G, int x, int y) { return (y + 1) * G.gw + (x + 1); }

// the unit step of a hull edge on the quarter grid and how many it takes
__device__ __forceinline__ int edge_steps(int dx, int dy, int& sx, int& sy)
{
    const int ax = abs(dx), ay = abs(dy);
    int g = max(ax, ay);
    if (ax && ay && ax != ay) { // neither along an axis nor a diagonal
        int u = ax, v = ay;
        while (v) {
            const int t = u % v;
            u = v;
            v = t;
        }
        g = u;
        sx = dx / g;
        sy = dy / g;
        return g;
    }
    sx = (dx > 0) - (dx < 0);
    sy = (dy > 0) - (dy < 0);
    return g;
}

// v -> u lies on p -> q in the same direction
__device__ __forceinline__ bool reversed_on(int px, int py, int qx, int qy, int ux, int uy, int vx, int vy)
{
    const int ex = qx - px, ey = qy - py;
    if (ex * (vy - py) - ey * (vx - px) != 0 || ex * (uy - py) - ey * (ux - px) != 0) return false;
    if (ex * (ux - vx) + ey * (uy - vy) <= 0) return false;
    const int L = ex * ex + ey * ey;
    const int tv = ex * (vx - px) + ey * (vy - py), tu = ex * (ux - px) + ey * (uy - py);
    return tv >= 0 && tu <= L;
}

__device__ __forceinline__ uint32_t cell_word(const Geo& G, int i, int j)
{
    return word_of_bgr(load_bgr(G.img, G.ws, G.layout, i, j), G.thr);
}

// Walks the split edges of hull edge t of cell idx; for each, the twin's owner:
// the first 8-neighbour (in bit order) with a hull edge that holds the reversed
// split edge. A neighbour is only searched when its hull's bounding box (the
// per-pattern box table) holds the split edge. npat, nbox: the neighbours'
// patterns (-1 outside the frame) and boxes, in shared memory (in registers,
// with the loop over them unrolled, they left room for 16 warps an SM).
// fn(ux, uy, vx, vy, owner, B).
template <typename Fn>
__device__ __forceinline__ void walk_split_edges(const Geo& G, const uint32_t* vgrid, int i, int j, uint64_t e, int t,
                                                 const int* npat, const uint32_t* nbox, Fn fn)
{
    const int k = (int)(e & 0xF), t1 = t + 1 == k ? 0 : t + 1;
    const int ax = qvx(e, t, i), ay = qvy(e, t, j), bx = qvx(e, t1, i), by = qvy(e, t1, j);
    int sx, sy;
    const int gcd = edge_steps(bx - ax, by - ay, sx, sy);
    int px = ax, py = ay;
    for (int st = 1; st <= gcd; st++) {
        const int cx = ax + st * sx, cy = ay + st * sy;
        if (st < gcd && !(vgrid[vindex(G, cx, cy)] & kVUsed)) continue;
        int owner = -1;
        // the split edge relative to the cell's own quarter origin
        const int lx0 = min(px, cx) - 4 * i, lx1 = max(px, cx) - 4 * i;
        const int ly0 = min(py, cy) - 4 * j, ly1 = max(py, cy) - 4 * j;
#pragma unroll 1
        for (int d = 0; d < 8 && owner < 0; d++) {
            if (npat[d] < 0) continue;
            const uint32_t bb = nbox[d];
            const int ox = 4 * dir_di(d), oy = 4 * dir_dj(d);
            if (lx0 < (int)(bb & 0xFF) - 8 + ox || lx1 > (int)((bb >> 8) & 0xFF) - 8 + ox ||
                ly0 < (int)((bb >> 16) & 0xFF) - 8 + oy || ly1 > (int)(bb >> 24) - 8 + oy)
                continue;
            const int ni = i + dir_di(d), nj = j + dir_dj(d);
            const uint64_t ne = __ldg(&G.lut[npat[d]]);
            const int nk = (int)(ne & 0xF);
            for (int s = 0; s < nk; s++) {
                const int s1 = s + 1 == nk ? 0 : s + 1;
                if (reversed_on(qvx(ne, s, ni), qvy(ne, s, nj), qvx(ne, s1, ni), qvy(ne, s1, nj), px, py, cx, cy)) {
                    owner = d;
                    break;
                }
            }
        }
        const int B = owner < 0 ? -1 : (j + dir_dj(owner)) * G.w + (i + dir_di(owner));
        fn(px, py, cx, cy, owner, B);
        px = cx;
        py = cy;
    }
}

// per pattern: the hull's bounding box in local quarter units, each bound + 8
__global__ void k_rf_boxes(const uint64_t* lut, uint32_t* box)
{
    const int pat = blockIdx.x * blockDim.x + threadIdx.x;
    if (pat >= 4096) return;
    const uint64_t e = lut[pat];
    const int k = (int)(e & 0xF);
    int x0 = 99, x1 = -99, y0 = 99, y1 = -99;
    for (int t = 0; t < k; t++) {
        const int x = qvx(e, t, 0), y = qvy(e, t, 0);
        x0 = min(x0, x);
        x1 = max(x1, x);
        y0 = min(y0, y);
        y1 = max(y1, y);
    }
    box[pat] = k ? (uint32_t)(x0 + 8) | (uint32_t)(x1 + 8) << 8 | (uint32_t)(y0 + 8) << 16 | (uint32_t)(y1 + 8) << 24
                 : 0xFFu; // empty: x0 beyond every edge
}

__global__ void k_rf_mark_vertices(Geo G, uint32_t* vgrid)
{
    follow_last();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= G.w * G.h) return;
    const int i = idx % G.w, j = idx / G.w;
    const uint64_t e = cell_hull(G, idx);
    const int k = (int)(e & 0xF);
    for (int t = 0; t < k; t++) atomicOr(&vgrid[vindex(G, qvx(e, t, i), qvy(e, t, j))], kVUsed);
}

// A cell whose node and neighbours all link their four sides and no diagonal
// (byte 90) is a square among squares: its edges are shared whole with the
// four cells beside it.
__device__ __forceinline__ bool square_among_squares(const Geo& G, int i, int j)
{
    if (i == 0 || j == 0 || i == G.w - 1 || j == G.h - 1) return false;
    const uint8_t* q = G.g + (size_t)j * G.w + i;
    bool all = true;
#pragma unroll
    for (int dj = -1; dj <= 1; dj++)
#pragma unroll
        for (int di = -1; di <= 1; di++) all &= q[dj * G.w + di] == 90;
    return all;
}

// Curve edges per cell, the frame marks, and the edges themselves, 16 bits each
// at slots + cell * max_split: the ends relative to the cell's corner (quarter
// units + 1, 3 bits a coordinate: u, v) and the owner's direction (bits 12-14).
// A block takes kEdgeCells cells; those that are not squares among similar
// squares go to a list (about four in ten), of which eight lanes take a cell, a
// hull edge each (a hull has at most eight): one cell's walk is a long chain,
// and a lane per cell spent 38 us on a 256x224 frame, once to count and once
// more to emit (57 us with the list and a lane per cell: too few warps). It is
// 33 us now and the emission, from the slots, 5.
constexpr int kEdgeCells = 32, kEdgeThreads = 128;
__global__ void __launch_bounds__(kEdgeThreads) k_rf_count_edges(Geo G, uint32_t* vgrid, int max_split, int* count,
                                                                 uint16_t* slots)
{
    follow_last();
    __shared__ int list[kEdgeCells], n;
    __shared__ int npat[kEdgeThreads];
    __shared__ uint32_t nbox[kEdgeThreads];
    if (threadIdx.x == 0) n = 0;
    __syncthreads();
    if (threadIdx.x < kEdgeCells) {
        const int idx = blockIdx.x * kEdgeCells + threadIdx.x;
        if (idx < G.w * G.h) {
            const int i = idx % G.w, j = idx / G.w;
            bool flat = square_among_squares(G, i, j);
            if (flat) {
                // the later of its neighbours are to the right and above
                const uint32_t me = cell_word(G, i, j);
                flat = similar(me, cell_word(G, i + 1, j), G.thr) && similar(me, cell_word(G, i, j + 1), G.thr);
            }
            if (flat) count[idx] = 0;
            else list[atomicAdd(&n, 1)] = idx;
        }
    }
    __syncthreads();
    const int t = threadIdx.x & 7;
    for (int k0 = 0; k0 < n; k0 += kEdgeThreads / 8) {
        const int k = k0 + (threadIdx.x >> 3);
        if (k0 + ((int)threadIdx.x & ~31) / 8 >= n) break; // whole warps
        const bool have = k < n;
        const int idx = list[have ? k : n - 1], i = idx % G.w, j = idx / G.w;
        // a neighbour's pattern and box a lane
        {
            const int ni = i + dir_di(t), nj = j + dir_dj(t);
            int mine = -1;
            if (ni >= 0 && ni < G.w && nj >= 0 && nj < G.h) {
                const int nidx = nj * G.w + ni, last = G.w * G.h;
                mine = cell_pattern(G.g[nidx], nidx > 0 ? G.g[nidx - 1] : 0u, nidx + 1 < last ? G.g[nidx + 1] : 0u);
                nbox[threadIdx.x] = __ldg(&G.box[mine]);
            }
            npat[threadIdx.x] = mine;
        }
        __syncwarp();
        const uint64_t e = cell_hull(G, idx);
        const uint32_t me = cell_word(G, i, j);
        uint64_t found = 0; // up to four split edges of a hull edge, 16 bits each
        int c = 0;
        if (have && t < (int)(e & 0xF))
            walk_split_edges(G, vgrid, i, j, e, t, npat + (threadIdx.x & ~7), nbox + (threadIdx.x & ~7), [&](int ux, int uy, int vx, int vy, int owner, int B) {
                if (owner < 0) {
                    atomicOr(&vgrid[vindex(G, ux, uy)], kVFrame);
                    atomicOr(&vgrid[vindex(G, vx, vy)], kVFrame);
                } else if (B > idx && !similar(me, cell_word(G, i + dir_di(owner), j + dir_dj(owner)), G.thr)) {
                    found |= (uint64_t)((ux - 4 * i + 1) | (uy - 4 * j + 1) << 3 | (vx - 4 * i + 1) << 6 |
                                        (vy - 4 * j + 1) << 9 | owner << 12)
                             << (16 * c++);
                }
            });
        int upto = c;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, upto, o, 8);
            if (t >= o) upto += y;
        }
        if (have) {
            uint16_t* slot = slots + (size_t)idx * max_split + (upto - c);
            for (int q = 0; q < c; q++) slot[q] = (uint16_t)(found >> (16 * q));
            if (t == 7) count[idx] = upto;
        }
        __syncwarp();
    }
}

// the curve edges at their offsets; degrees and up to two neighbours (vertex,
// edge) per vertex
__global__ void k_rf_emit_edges(Geo G, uint32_t* vgrid, int max_split, const int* count, Scan<int> off,
                                const uint16_t* slots, int4* edges, int2* nb_v, int2* nb_e)
{
    follow_last();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= G.w * G.h) return;
    const int c = count[idx];
    if (!c) return;
    const int i = idx % G.w, j = idx / G.w, o0 = off.at(idx);
    const uint16_t* slot = slots + (size_t)idx * max_split;
    for (int k = 0; k < c; k++) {
        const unsigned e = slot[k];
        const int u = vindex(G, 4 * i + (int)(e & 7u) - 1, 4 * j + (int)(e >> 3 & 7u) - 1);
        const int v = vindex(G, 4 * i + (int)(e >> 6 & 7u) - 1, 4 * j + (int)(e >> 9 & 7u) - 1);
        const int d = (int)(e >> 12), o = o0 + k;
        edges[o] = make_int4(u, v, idx, (j + dir_dj(d)) * G.w + i + dir_di(d));
        const uint32_t su = atomicAdd(&vgrid[u], 1u << kDegShift) >> kDegShift;
        const uint32_t sv = atomicAdd(&vgrid[v], 1u << kDegShift) >> kDegShift;
        if (su < 2) {
            (&nb_v[u].x)[su] = v;
            (&nb_e[u].x)[su] = o;
        }
        if (sv < 2) {
            (&nb_v[v].x)[sv] = u;
            (&nb_e[v].x)[sv] = o;
        }
    }
}

// scan inputs: vertices with curve edges, free nodes
struct NodeFlag {
    const uint32_t* vgrid;
    __device__ __forceinline__ int operator()(int v) const { return (vgrid[v] >> kDegShift) > 0; }
};
struct FreeFlag {
    const int* flags;
    __device__ __forceinline__ int operator()(int k) const { return !(flags[k] & 1); }
};
struct CellCount {
    const int* count;
    __device__ __forceinline__ int operator()(int k) const { return count[k]; }
};
// samples of a slot (low word) and whether it has any (high word)
struct SampleCount {
    const int* count;
    __device__ __forceinline__ unsigned long long operator()(int k) const
    {
        const unsigned c = (unsigned)count[k];
        return c | (unsigned long long)(c > 0) << 32;
    }
};

// The segments that read a free node: the middles of its two edges (parts 0 and
// 1), its own corner (2) and, across each edge, the neighbour's corner or pinned
// piece (3 and 4). Each keeps its part of the node's coverage gradient in a place
// of its own and the node pass sums them, so that a run's positions do not depend
// on what else runs, or on how the steps are launched: by float atomics the sum
// had another rounding with every order of arrival, and where it should be zero
// Adam makes a step of full length of its last bits.
constexpr int kParts = 5;

struct NodeOut {
    int2* q;        // quarter coordinates
    int* flags;     // bit 0 pinned, 1 frame, 2 corner; degree << 4
    int2* nbr;      // neighbours of degree-2 nodes (ascending), else -1
    int2* nbr_edge; // the edges to them
    float2* pos0;
    float2* gcov;   // kParts parts of n each, zeroed
    int n;          // nodes
};

__global__ void k_rf_make_nodes(Geo G, const uint32_t* vgrid, Scan<int> nid, const int2* nb_v, const int2* nb_e, NodeOut N)
{
    follow_last();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= G.gw * G.gh) return;
    const uint32_t word = vgrid[v];
    const int deg = (int)(word >> kDegShift);
    if (deg == 0) return;
    const int k = nid.at(v);
    const int x = v % G.gw - 1, y = v / G.gw - 1;
    int f = min(deg, 15) << 4;
    if (word & kVFrame) f |= 2;
    int2 nb = make_int2(-1, -1), ne = make_int2(-1, -1);
    if (deg == 2) {
        int a = nid.at(nb_v[v].x), b = nid.at(nb_v[v].y);
        int ea = nb_e[v].x, eb = nb_e[v].y;
        const int va = nb_v[v].x, vb = nb_v[v].y;
        int vax = va % G.gw - 1, vay = va / G.gw - 1, vbx = vb % G.gw - 1, vby = vb / G.gw - 1;
        if (a > b) {
            int t = a; a = b; b = t;
            t = ea; ea = eb; eb = t;
            t = vax; vax = vbx; vbx = t;
            t = vay; vay = vby; vby = t;
        }
        nb = make_int2(a, b);
        ne = make_int2(ea, eb);
        if ((x - vax) * (vbx - x) + (y - vay) * (vby - y) <= 0) f |= 4;
    }
    if (deg != 2 || (f & 6)) f |= 1;
    N.q[k] = make_int2(x, y);
    N.flags[k] = f;
    N.nbr[k] = nb;
    N.nbr_edge[k] = ne;
    N.pos0[k] = make_float2(0.25f * x, 0.25f * y);
#pragma unroll
    for (int q = 0; q < kParts; q++) N.gcov[(size_t)q * N.n + k] = make_float2(0.f, 0.f);
}

struct SegOut {
    int4* seg;    // n0, n1, n2, type
    uint2* col;   // left, right RGB (0xBBGGRR)
};

__device__ __forceinline__ uint32_t pixel_rgb(const Geo& G, int i, int j)
{
    const uint32_t c = load_bgr(G.img, G.ws, G.layout, i, j); // b0 | b1 << 8 | b2 << 16
    // reference bytes (b0, b1, b2) = (B, G, R) -> R | G << 8 | B << 16
    return ((c >> 16) & 0xFFu) | (c & 0xFF00u) | ((c & 0xFFu) << 16);
}
__device__ __forceinline__ uint32_t cell_rgb(const Geo& G, int idx) { return pixel_rgb(G, idx % G.w, idx / G.w); }

// segment slots: 3 per edge, then one per node
__global__ void k_rf_segments(Geo G, Scan<int> nid, int4* edges, int E, int Nn, const int* flags, const int2* nbr,
                              const int2* nbr_edge, SegOut S)
{
    follow_last();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < E) {
        int4 ed = edges[t];
        const int u = nid.at(ed.x), v = nid.at(ed.y);
        const uint2 col = make_uint2(cell_rgb(G, ed.z), cell_rgb(G, ed.w));
        const bool pu = flags[u] & 1, pv = flags[v] & 1;
        S.seg[3 * t] = pu ? make_int4(u, v, -1, SEG_PIN_U) : make_int4(-1, -1, -1, SEG_NONE);
        S.seg[3 * t + 1] = make_int4(u, v, -1, SEG_MID);
        S.seg[3 * t + 2] = pv ? make_int4(u, v, -1, SEG_PIN_V) : make_int4(-1, -1, -1, SEG_NONE);
        S.col[3 * t] = S.col[3 * t + 1] = S.col[3 * t + 2] = col;
    } else if (t < E + Nn) {
        const int p = t - E;
        const int s = 3 * E + p;
        if (flags[p] & 1) {
            S.seg[s] = make_int4(-1, -1, -1, SEG_NONE);
            S.col[s] = make_uint2(0, 0);
            return;
        }
        const int a = nbr[p].x, b = nbr[p].y;
        const int e = nbr_edge[p].x; // the edge between a and p
        const int4 ed = edges[e];
        const uint32_t l = cell_rgb(G, ed.z), r = cell_rgb(G, ed.w);
        const bool flip = nid.at(ed.x) != a; // stored as p -> a
        S.seg[s] = make_int4(a, p, b, SEG_CORNER);
        S.col[s] = flip ? make_uint2(r, l) : make_uint2(l, r);
    }
}

// exact segment ends at the start, in 1/(32 s) source pixel
__device__ __forceinline__ void seg_ends(const int4 sg, const int2* q, int scale, long long& ax, long long& ay,
                                         long long& bx, long long& by)
{
    ax = ay = bx = by = 0;
    const int nodes[3] = {sg.x, sg.y, sg.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (nodes[k] < 0) continue;
        const int2 p = q[nodes[k]];
        ax += (long long)seg_wa(sg.w, k) * p.x;
        ay += (long long)seg_wa(sg.w, k) * p.y;
        bx += (long long)seg_wb(sg.w, k) * p.x;
        by += (long long)seg_wb(sg.w, k) * p.y;
    }
    const long long m = 2 * scale; // weights x4, quarter -> 1/(32 s): x 8 s / 4
    ax *= m;
    ay *= m;
    bx *= m;
    by *= m;
}

// A segment and the output samples of its box (with the band), numbered row by
// row: sample Xo sits at 16 (2 Xo + 1). Coordinates relative to the first end
// fit 32 bits (a segment spans a few source pixels of 32 s units).
struct SegBox {
    int x0, y0, nx, ny; // first sample, samples
    int ex, ey, wx, wy; // second end, and the first sample's position, from the first end
    __device__ __forceinline__ int count() const { return nx > 0 && ny > 0 ? nx * ny : 0; }
};

__device__ __forceinline__ long long floor_div_ll(long long a, long long b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

__device__ __forceinline__ SegBox seg_box(const int4 sg, const int2* q, int scale, int ow, int oh)
{
    long long ax, ay, bx, by;
    seg_ends(sg, q, scale, ax, ay, bx, by);
    const long long x0 = max(0LL, -floor_div_ll(-(min(ax, bx) - kBand - 16), 32));
    const long long x1 = min((long long)ow - 1, floor_div_ll(max(ax, bx) + kBand - 16, 32));
    const long long y0 = max(0LL, -floor_div_ll(-(min(ay, by) - kBand - 16), 32));
    const long long y1 = min((long long)oh - 1, floor_div_ll(max(ay, by) + kBand - 16, 32));
    return SegBox{(int)x0, (int)y0, (int)(x1 - x0 + 1), (int)(y1 - y0 + 1), (int)(bx - ax), (int)(by - ay),
                  (int)(16 * (2 * x0 + 1) - ax), (int)(16 * (2 * y0 + 1) - ay)};
}

// Order of the squared distances of the box's samples (i, j), without their
// rounded quotients: in the middle of a segment the squared distance is
// cr^2 / L in whole numbers, L the segment's squared length, at most 512 s^2
// (half a hull edge, or a quarter of two, of 4 sqrt 2 quarter pixels at most).
// Two different ones lie 1 / (512 s^2)^2 apart or more, so that their floors to
// frac_bits = 2 log2(512 s^2) binary digits keep their order and tell them
// apart (as their quotients rounded to double do). At most band^2 < 2^12.
// kFar beyond the band. The digits come 15 at a time from a float quotient,
// which is off by at most one, corrected in whole numbers. (64-bit float
// quotients, on a unit of two lanes a cycle, were most of the two passes' 34 us
// each over a 256x224 frame at x4.)
constexpr unsigned long long kFar = ~0ull;
__host__ __device__ __forceinline__ int frac_bits(int scale)
{
    int b = 0;
    while ((1 << b) < 512 * scale * scale) b++;
    return 2 * b;
}
__device__ __forceinline__ uint32_t divide(uint32_t a, uint32_t L, float inv, uint32_t& rem)
{
    uint32_t q = (uint32_t)__float2uint_rz((float)a * inv);
    int r = (int)(a - q * L);
    if (r < 0) {
        q--;
        r += (int)L;
    } else if (r >= (int)L) {
        q++;
        r -= (int)L;
    }
    rem = (uint32_t)r;
    return q;
}
__device__ __forceinline__ unsigned long long seg_key(const SegBox& B, int i, int j, float inv, int bits)
{
    constexpr int band2 = kBand * kBand;
    const int wx = B.wx + 32 * i, wy = B.wy + 32 * j;
    const int L = B.ex * B.ex + B.ey * B.ey, dot = B.ex * wx + B.ey * wy;
    if (dot <= 0 || dot >= L) {
        const int ux = dot <= 0 ? wx : wx - B.ex, uy = dot <= 0 ? wy : wy - B.ey;
        const int d = ux * ux + uy * uy;
        return d <= band2 ? (unsigned long long)d << bits : kFar;
    }
    const long long cr = (long long)B.ex * wy - (long long)B.ey * wx;
    if (cr * cr > (long long)band2 * L) return kFar;
    uint32_t r;
    unsigned long long key = divide((uint32_t)(cr * cr), (uint32_t)L, inv, r);
    for (int left = bits; left > 0; left -= 15) {
        const int n = min(left, 15);
        key = key << n | divide(r << n, (uint32_t)L, inv, r);
    }
    return key;
}

// The samples of each slot's box, kBoxLanes lanes a slot: fn(slot, box, live,
// output sample, column, row) for every sample, the lanes of the warp together
// (live: the lane has one); a box's samples come in ascending order. (One lane a
// slot, with 64-bit coordinates, spent 39 us on each pass over the boxes of a
// 256x224 frame at x4; eight lanes take 15 to assign and 12 to fill.)
constexpr int kBoxLanes = 8;
template <typename Fn>
__device__ __forceinline__ void box_samples(const SegBox& B, int ow, Fn fn)
{
    const int n = B.count(), gl = threadIdx.x & (kBoxLanes - 1);
    int most = n;
#pragma unroll
    for (int o = kBoxLanes; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xFFFFFFFFu, most, o));
    int i = gl, j = 0; // column and row of the lane's sample
    for (int k = gl; k - gl < most; k += kBoxLanes, i += kBoxLanes) {
        const bool live = k < n;
        if (live)
            while (i >= B.nx) {
                i -= B.nx;
                j++;
            }
        fn(live, live ? (B.y0 + j) * ow + B.x0 + i : 0, i, j);
    }
}

// the lane's slot and its box (empty for slots without a segment)
__device__ __forceinline__ SegBox slot_box(const int4* seg, int S, const int2* q, int scale, int ow, int oh, int& slot)
{
    slot = (blockIdx.x * blockDim.x + threadIdx.x) / kBoxLanes;
    const int4 sg = slot < S ? seg[slot] : make_int4(-1, -1, -1, SEG_NONE);
    if (sg.w == SEG_NONE) return SegBox{0, 0, 0, 0, 0, 0, 0, 0};
    return seg_box(sg, q, scale, ow, oh);
}

// The slot nearest to each output sample, ties to the lower one. Where distance
// and slot fit one 64-bit key (slot_bits > 0, any frame of up to 2^18 slots at
// any scale), its minimum is all; else the least distance, then the lowest slot
// that has it.
struct Owner {
    unsigned long long* best;
    int* bseg;     // NULL with keys that hold the slot
    int slot_bits;
    __device__ __forceinline__ int operator()(int x) const
    {
        return bseg ? bseg[x] : (int)(best[x] & ((1ull << slot_bits) - 1ull)); // none: no slot's number
    }
};

template <bool SLOT_PASS>
__global__ void k_rf_assign(const int4* seg, int S, const int2* q, int scale, int ow, int oh, Owner own)
{
    follow_last();
    int slot;
    const SegBox B = slot_box(seg, S, q, scale, ow, oh, slot);
    const float inv = 1.f / (float)max(B.ex * B.ex + B.ey * B.ey, 1);
    const int bits = frac_bits(scale);
    box_samples(B, ow, [&](bool live, int x, int i, int j) {
        if (!live) return;
        const unsigned long long key = seg_key(B, i, j, inv, bits);
        if (key == kFar) return;
        if constexpr (SLOT_PASS) {
            if (key == own.best[x]) atomicMin(&own.bseg[x], slot);
        } else {
            atomicMin(&own.best[x], own.slot_bits ? key << own.slot_bits | (unsigned)slot : key);
        }
    });
}

// samples assigned to each slot
__global__ void k_rf_count_samples(const int4* seg, int S, const int2* q, int scale, int ow, int oh, Owner own,
                                   int* seg_count)
{
    follow_last();
    int slot, c = 0;
    const SegBox B = slot_box(seg, S, q, scale, ow, oh, slot);
    box_samples(B, ow, [&](bool live, int x, int, int) { c += live && own(x) == slot; });
#pragma unroll
    for (int o = kBoxLanes / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if (slot < S && (threadIdx.x & (kBoxLanes - 1)) == 0) seg_count[slot] = c;
}

// the nearest-neighbour target under the coverage Gaussian, per sample
// (separable: three column and three row weights), and its position
__global__ void k_rf_targets(Geo G, int scale, float sig, const int* samp, const int* pM, float4* tgt,
                             float2* sxy)
{
    follow_last();
    const int M = *pM, ow = G.w * scale;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < M; m += gridDim.x * blockDim.x) {
        const int yo = samp[m] / ow, xo = samp[m] - yo * ow;
        const float x = ((float)xo + 0.5f) / (float)scale, y = ((float)yo + 0.5f) / (float)scale;
        const int ix = xo / scale, iy = yo / scale;
        const float inv = 1.f / sig;
        float cx[3], cy[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const int ii = ix + d - 1, jj = iy + d - 1;
            cx[d] = (ii >= 0 && ii < G.w) ? normcdff((x - (float)ii) * inv) - normcdff((x - (float)ii - 1.f) * inv) : 0.f;
            cy[d] = (jj >= 0 && jj < G.h) ? normcdff((y - (float)jj) * inv) - normcdff((y - (float)jj - 1.f) * inv) : 0.f;
        }
        float r = 0.f, g = 0.f, b = 0.f;
#pragma unroll
        for (int dj = 0; dj < 3; dj++) {
            const int jj = iy + dj - 1;
            if (jj < 0 || jj >= G.h) continue;
#pragma unroll
            for (int di = 0; di < 3; di++) {
                const int ii = ix + di - 1;
                if (ii < 0 || ii >= G.w) continue;
                const float wgt = cx[di] * cy[dj];
                const uint32_t c = pixel_rgb(G, ii, jj);
                r += wgt * (float)(c & 0xFF);
                g += wgt * (float)((c >> 8) & 0xFF);
                b += wgt * (float)((c >> 16) & 0xFF);
            }
        }
        tgt[m] = make_float4(r, g, b, 0.f);
        sxy[m] = make_float2(x, y);
    }
}

// ------------------------------------------------------------ warm start

constexpr int kWarmTile = 16; // source pixels per tile side

// Tile signature, a warp per tile: the sum over the pixels of the tile and its
// one-pixel ring (those inside the frame) of a 64-bit mix of the pixel's place,
// resolved graph byte and RGB: everything the tile's cells, curve edges and
// targets depend on. Only compared, frame against frame of one size. (A
// byte-by-byte FNV-1a, a lane per tile, was one chain of 1296 products: 57 us.)
__global__ void k_rf_tile_hash(Geo G, int tiles_x, int tiles, uint64_t* hash)
{
    follow_last();
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= tiles) return;
    const int x0 = (t % tiles_x) * kWarmTile - 1, y0 = (t / tiles_x) * kWarmTile - 1;
    constexpr int W = kWarmTile + 2;
    unsigned long long sum = 0;
    for (int k = lane; k < W * W; k += 32) {
        const int x = x0 + k % W, y = y0 + k / W;
        if (x < 0 || y < 0 || x >= G.w || y >= G.h) continue;
        // the finaliser of MurmurHash3 (Appleby, public domain)
        unsigned long long z = (unsigned long long)pixel_rgb(G, x, y) | (unsigned long long)G.g[y * G.w + x] << 24 |
                               (unsigned long long)(k + 1) << 32;
        z ^= z >> 33;
        z *= 0xFF51AFD7ED558CCDull;
        z ^= z >> 33;
        z *= 0xC4CEB9FE1A85EC53ull;
        z ^= z >> 33;
        sum += z;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) hash[t] = sum;
}

__global__ void k_rf_warm_scatter(const int2* q, const float2* pos, int N, int gw, float2* grid, int* stamp, int epoch)
{
    follow_last();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    const int v = (q[k].y + 1) * gw + (q[k].x + 1);
    grid[v] = pos[k];
    stamp[v] = epoch;
}

__global__ void k_rf_warm_gather(const int2* q, const float2* pos0, int N, int w, int h, int gw, int tiles_x,
                                 const uint64_t* hash, const uint64_t* prev_hash, const float2* grid,
                                 const int* stamp, int epoch, float2* out)
{
    follow_last();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= N) return;
    const int2 c = q[k];
    const int px = min(max(c.x >> 2, 0), w - 1), py = min(max(c.y >> 2, 0), h - 1);
    const int t = (py / kWarmTile) * tiles_x + px / kWarmTile;
    const int v = (c.y + 1) * gw + (c.x + 1);
    out[k] = (hash[t] == prev_hash[t] && stamp[v] == epoch) ? grid[v] : pos0[k];
}

__global__ void k_rf_same_tiles(const uint64_t* a, const uint64_t* b, int tiles, int* count)
{
    follow_last();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool same = t < tiles && a[t] == b[t];
    const unsigned m = __ballot_sync(0xFFFFFFFFu, same);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(count, __popc(m));
}

// ------------------------------------------------------- energy and adjoint

// Frame sizes the step kernels read from device memory, so that a captured
// graph of the Adam loop serves every frame of the same buffers.
struct RefineFrame {
    int N;      // nodes
    int L;      // live segments (with samples)
    int ow, oh; // output raster
    int scale;
    int F;      // free nodes
    float inv_samples3; // 1 / (3 ow oh), rounded once on the host
};

// A live segment, packed for one load: its nodes and type, its sample
// range and its colours.
struct LiveSeg {
    int4 nodes;  // n0, n1, n2, type | its part of n0 << 3, of n1 << 6, of n2 << 9
    int4 range;  // first sample, end, left colour, right colour (0xBBGGRR)
};

// A free node and the nodes its curvature gradient reads: its neighbours
// a, b and, where a neighbour is free, that neighbour's neighbours (-1 when
// pinned), packed for one load.
struct FreeNode {
    int4 k_a_b_aa; // node, a, b, a's first neighbour
    int4 ab_ba_bb; // a's second neighbour, b's neighbours, unused
};

struct StepArgs {
    const float2* x;     // positions read
    float2* y;           // positions written (Adam)
    float2* gcov;        // coverage gradient: kParts parts of N nodes, zero where no live segment writes
    float2* gout;        // gradient out (energy/gradient call), or NULL
    const float2* x0;
    const float4* tgt;
    const int* flags;
    const LiveSeg* live;
    const float2* sxy;   // sample positions (source pixels), in segment order
    const FreeNode* fnodes;
    const RefineFrame* fr;
    float2* m;
    float2* v;
    double* energy;      // [3] when not NULL
    float sigma;         // output pixels
    float w_curv, w_dev, w_cov;
    float lr, bc1, bc2;  // Adam step and bias corrections 1 - beta^t
};

constexpr float kBeta1 = 0.9f, kBeta2 = 0.999f, kEps = 1e-8f;
constexpr float kInvSqrt2Pi = 0.3989422804014327f;
// Lanes per segment in the coverage pass: three store a node's part each, and
// with 8 lanes a step of 20 over a 256x224 x4 frame took 6.7 us where 4 took 5.9.
constexpr int kSegLanes = 4;

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__device__ __forceinline__ float group_sum(float v, unsigned mask)
{
#pragma unroll
    for (int o = kSegLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// A live segment's line at positions x, its Chaikin ends recomputed from the
// nodes, and its colours.
struct Edge {
    float2 A, B;
    float cr[3], dl[3], ex, ey, invL;
};
__device__ __forceinline__ Edge live_edge(const LiveSeg& ls, const float2* x)
{
    Edge E;
    const int4 sg = ls.nodes;
    const int nodes[3] = {sg.x, sg.y, sg.z}, type = sg.w & 7;
    E.A = E.B = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (nodes[k] < 0) continue;
        const float2 p = x[nodes[k]];
        const float wa = 0.25f * seg_wa(type, k), wb = 0.25f * seg_wb(type, k);
        E.A.x += wa * p.x;
        E.A.y += wa * p.y;
        E.B.x += wb * p.x;
        E.B.y += wb * p.y;
    }
    const uint32_t left = (uint32_t)ls.range.z, right = (uint32_t)ls.range.w;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        E.cr[c] = (float)((right >> (8 * c)) & 0xFF);
        E.dl[c] = (float)(int)((left >> (8 * c)) & 0xFF) - (float)(int)((right >> (8 * c)) & 0xFF);
    }
    E.ex = E.B.x - E.A.x;
    E.ey = E.B.y - E.A.y;
    E.invL = rsqrtf(E.ex * E.ex + E.ey * E.ey);
    return E;
}

// One sample's soft colour against its target: adds d loss / d ends to g (A.x,
// A.y, B.x, B.y) and returns the squared error.
__device__ __forceinline__ float sample_loss(const Edge& E, float2 X, float4 t, float inv_sig, float cov_norm, float (&g)[4])
{
    const float wx = X.x - E.A.x, wy = X.y - E.A.y;
    const float d = (E.ex * wy - E.ey * wx) * E.invL;
    const float z = d * inv_sig;
    const float Phi = normcdff(z);
    const float r0 = (E.cr[0] + E.dl[0] * Phi - t.x) * (1.f / 255.f);
    const float r1 = (E.cr[1] + E.dl[1] * Phi - t.y) * (1.f / 255.f);
    const float r2 = (E.cr[2] + E.dl[2] * Phi - t.z) * (1.f / 255.f);
    const float phi = expf(-0.5f * z * z) * kInvSqrt2Pi * inv_sig;
    const float dEdd = 2.f * cov_norm * (1.f / 255.f) * (r0 * E.dl[0] + r1 * E.dl[1] + r2 * E.dl[2]) * phi;
    // d d / d e = (wy, -wx) / L - d e / L^2 ; d d / d w = (-ey, ex) / L
    const float dex = wy * E.invL - d * E.ex * E.invL * E.invL, dey = -wx * E.invL - d * E.ey * E.invL * E.invL;
    const float dwx = -E.ey * E.invL, dwy = E.ex * E.invL;
    g[0] += dEdd * (-dex - dwx);
    g[1] += dEdd * (-dey - dwy);
    g[2] += dEdd * dex;
    g[3] += dEdd * dey;
    return r0 * r0 + r1 * r1 + r2 * r2;
}

// Coverage: kSegLanes lanes per live segment, the samples' gradients reduced in
// the group and stored as the segment's parts of its free nodes' gradients.
template <bool ENERGY>
__global__ void __launch_bounds__(256) k_rf_coverage(StepArgs a)
{
    const RefineFrame F = *a.fr;
    const float inv_sig = (float)F.scale / a.sigma;
    const float cov_norm = a.w_cov * F.inv_samples3;
    const int lane = threadIdx.x & 31, gl = lane & (kSegLanes - 1);
    const unsigned gmask = ((1u << kSegLanes) - 1u) << (lane & ~(kSegLanes - 1));
    const int groups = (gridDim.x * blockDim.x) / kSegLanes;
    float eloss = 0.f;
    bool waited = false;
    for (int l = (blockIdx.x * blockDim.x + threadIdx.x) / kSegLanes; l < F.L; l += groups) {
        const LiveSeg ls = a.live[l];
        const int m0 = ls.range.x + gl;
        const bool have = m0 < ls.range.y;
        float2 X = make_float2(0.f, 0.f);
        float4 T = make_float4(0.f, 0.f, 0.f, 0.f);
        if (have) {
            X = a.sxy[m0];
            T = a.tgt[m0];
        }
        const int4 sg = ls.nodes;
        const int my = gl == 0 ? sg.x : (gl == 1 ? sg.y : (gl == 2 ? sg.z : -1));
        const bool push = my >= 0 && !(a.flags[my] & 1);
        if (!waited) follow_last();
        waited = true;
        const Edge E = live_edge(ls, a.x);
        float g[4] = {0.f, 0.f, 0.f, 0.f};
        if (have) eloss += sample_loss(E, X, T, inv_sig, cov_norm, g);
        for (int m = m0 + kSegLanes; m < ls.range.y; m += kSegLanes)
            eloss += sample_loss(E, a.sxy[m], a.tgt[m], inv_sig, cov_norm, g);
#pragma unroll
        for (int k = 0; k < 4; k++) g[k] = group_sum(g[k], gmask);
        if (push) {
            const int type = sg.w & 7, part = sg.w >> (3 + 3 * gl) & 7;
            const float wa = 0.25f * seg_wa(type, gl), wb = 0.25f * seg_wb(type, gl);
            a.gcov[(size_t)part * F.N + my] = make_float2(wa * g[0] + wb * g[2], wa * g[1] + wb * g[3]);
        }
    }
    if (!waited) follow_last(); // a grid that ended without it could overtake the one before
    if constexpr (ENERGY) {
        eloss = warp_sum(eloss);
        if (lane == 0 && eloss != 0.f) atomicAdd(&a.energy[2], (double)eloss * (double)cov_norm);
    }
}

// The curvature stencil of a free node p: its second difference t and the sum g
// of what its own and its free neighbours' second differences give p. nb, qn:
// the neighbours' neighbours (-1 where the neighbour is pinned).
struct Stencil {
    float2 t, g;
};
__device__ __forceinline__ Stencil node_stencil(float2 p, float2 pa, float2 pb, const int (&nb)[4], const float2 (&qn)[4])
{
    const float tx = pa.x - 2.f * p.x + pb.x, ty = pa.y - 2.f * p.y + pb.y;
    float gx = -2.f * tx, gy = -2.f * ty;
    if (nb[0] >= 0) { // a is free: its second difference reads p
        gx += qn[0].x - 2.f * pa.x + qn[1].x;
        gy += qn[0].y - 2.f * pa.y + qn[1].y;
    }
    if (nb[2] >= 0) {
        gx += qn[2].x - 2.f * pb.x + qn[3].x;
        gy += qn[2].y - 2.f * pb.y + qn[3].y;
    }
    return Stencil{make_float2(tx, ty), make_float2(gx, gy)};
}

// The gradient and Adam's moments, with their roundings written out: where a
// gradient should be zero, Adam makes a step of full length of its last bits, so
// another choice of fused operations (the compiler's changed with the code around
// them) moved nodes of some frames by hundredths of a pixel.
__device__ __forceinline__ float node_gradient(float curv, float g, float dev, float d, float cov)
{
    return __fadd_rn(__fmaf_rn(curv, g, __fmul_rn(dev, d)), cov);
}
__device__ __forceinline__ float first_moment(float m, float g) { return __fmaf_rn(1.f - kBeta1, g, __fmul_rn(kBeta1, m)); }
__device__ __forceinline__ float second_moment(float v, float g)
{
    return __fmaf_rn(__fmul_rn(1.f - kBeta2, g), g, __fmul_rn(kBeta2, v));
}

// Sum of a node's parts, rounded as if once: Knuth's two-sum (The Art of Computer
// Programming, volume 2, section 4.2.2) keeps what each addition rounds away.
__device__ __forceinline__ float sum_parts(const float (&part)[kParts])
{
    float s = part[0], lost = 0.f;
#pragma unroll
    for (int q = 1; q < kParts; q++) {
        const float t = __fadd_rn(s, part[q]), b = __fsub_rn(t, s);
        lost = __fadd_rn(lost, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(part[q], b)));
        s = t;
    }
    const float sum = __fadd_rn(s, lost);
    return sum == sum ? sum : s; // an infinite sum loses its difference to itself
}

// One thread per free node: curvature and deviation gradients, the coverage
// gradient's parts that k_rf_coverage left, then an Adam step, or the energy and
// the gradient written out.
template <bool ENERGY>
__global__ void __launch_bounds__(64) k_rf_nodes(StepArgs a)
{
    const RefineFrame F = *a.fr;
    const float curv_k = a.w_curv / (float)max(F.F, 1), dev_k = a.w_dev / (float)max(F.F, 1);
    float ec = 0.f, ed = 0.f;
    bool waited = false;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F.F; f += gridDim.x * blockDim.x) {
        const FreeNode fn = a.fnodes[f];
        const int k = fn.k_a_b_aa.x;
        const float2 p0 = a.x0[k];
        if (!waited) follow_last();
        waited = true;
        const int nb[4] = {fn.k_a_b_aa.w, fn.ab_ba_bb.x, fn.ab_ba_bb.y, fn.ab_ba_bb.z};
        float2 qn[4];
#pragma unroll
        for (int t = 0; t < 4; t++) qn[t] = nb[t] >= 0 ? a.x[nb[t]] : make_float2(0.f, 0.f);
        const float2 p = a.x[k], pa = a.x[fn.k_a_b_aa.y], pb = a.x[fn.k_a_b_aa.z];
        float cx[kParts], cy[kParts];
#pragma unroll
        for (int q = 0; q < kParts; q++) {
            const float2 c = a.gcov[(size_t)q * F.N + k];
            cx[q] = c.x;
            cy[q] = c.y;
        }
        float2 m = make_float2(0.f, 0.f), v = m;
        if constexpr (!ENERGY) {
            m = a.m[f];
            v = a.v[f];
        }
        const Stencil S = node_stencil(p, pa, pb, nb, qn);
        const float dx = p.x - p0.x, dy = p.y - p0.y;
        const float gx = node_gradient(0.25f * curv_k, S.g.x, 2.f * dev_k, dx, sum_parts(cx));
        const float gy = node_gradient(0.25f * curv_k, S.g.y, 2.f * dev_k, dy, sum_parts(cy));
        if constexpr (ENERGY) {
            ec += 0.125f * (S.t.x * S.t.x + S.t.y * S.t.y);
            ed += dx * dx + dy * dy;
            if (a.gout) a.gout[k] = make_float2(gx, gy);
        } else {
            m.x = first_moment(m.x, gx);
            m.y = first_moment(m.y, gy);
            v.x = second_moment(v.x, gx);
            v.y = second_moment(v.y, gy);
            a.m[f] = m;
            a.v[f] = v;
            a.y[k] = make_float2(p.x - a.lr * (m.x / a.bc1) / (sqrtf(v.x / a.bc2) + kEps),
                                 p.y - a.lr * (m.y / a.bc1) / (sqrtf(v.y / a.bc2) + kEps));
        }
    }
    if (!waited) follow_last();
    if constexpr (ENERGY) {
        ec = warp_sum(ec);
        ed = warp_sum(ed);
        if ((threadIdx.x & 31) == 0) {
            if (ec != 0.f) atomicAdd(&a.energy[0], (double)ec * (double)curv_k);
            if (ed != 0.f) atomicAdd(&a.energy[1], (double)ed * (double)dev_k);
        }
    }
}

// Which of a free node's kParts parts a segment (slot, sg) keeps; at: the node's
// place in the segment (0..2), nbr_edge: the nodes' edges.
__device__ __forceinline__ int node_part(const int4 sg, int slot, int at, const int2* nbr_edge)
{
    const int k = at == 0 ? sg.x : (at == 1 ? sg.y : sg.z);
    if (k < 0) return 0;
    if (sg.w == SEG_CORNER && at == 1) return 2;
    // the edge by which the segment reaches the node
    const int e = sg.w != SEG_CORNER ? slot / 3 : (at == 0 ? nbr_edge[sg.y].x : nbr_edge[sg.y].y);
    return (sg.w == SEG_MID ? 0 : 3) + (nbr_edge[k].x == e ? 0 : 1);
}

// The samples of each slot in ascending order (summation order fixed) at its
// offset, the live segments (those with samples) packed, and the offsets.
__global__ void k_rf_fill_samples(const int4* seg, int S, const int2* q, int scale, int ow, int oh, Owner own,
                                  const int* seg_count, Scan<unsigned long long> off, const uint2* col, int* samp,
                                  int* seg_off, const int2* nbr_edge, LiveSeg* live)
{
    follow_last();
    int slot;
    SegBox B = slot_box(seg, S, q, scale, ow, oh, slot);
    const int gl = threadIdx.x & (kBoxLanes - 1), shift = threadIdx.x & 31 & ~(kBoxLanes - 1);
    const unsigned long long o = slot < S ? off.at(slot) : 0ull;
    int at = (int)(unsigned)o;
    const int c = slot < S ? seg_count[slot] : 0;
    if (slot < S && gl == 0) {
        seg_off[slot] = at;
        if (slot == S - 1) seg_off[S] = at + c;
    }
    int4 sg = make_int4(-1, -1, -1, SEG_NONE);
    int parts = 0; // of the three nodes, a lane each
    if (c) {
        sg = seg[slot];
        if (gl < 3) parts = node_part(sg, slot, gl, nbr_edge) << (3 + 3 * gl);
    }
    parts |= __shfl_xor_sync(0xFFFFFFFFu, parts, 1);
    parts |= __shfl_xor_sync(0xFFFFFFFFu, parts, 2);
    if (c && gl == 0) {
        const uint2 lr = col[slot];
        sg.w |= parts;
        live[o >> 32] = LiveSeg{sg, make_int4(at, at + c, (int)lr.x, (int)lr.y)};
    }
    if (!c) B.nx = 0;
    box_samples(B, ow, [&](bool have, int x, int, int) {
        const bool mine = have && own(x) == slot;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, mine) >> shift & ((1u << kBoxLanes) - 1u);
        if (mine) samp[at + __popc(m & ((1u << gl) - 1u))] = x;
        at += __popc(m);
    });
}

// start of an Adam run: both position buffers from src, moments zeroed
__global__ void k_rf_begin(const float2* src, float2* x, float2* y, float2* m, float2* v, int N)
{
    follow_last();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 q = src[i];
        x[i] = q;
        y[i] = q; // pinned nodes never move: both buffers start equal
        m[i] = make_float2(0.f, 0.f);
        v[i] = make_float2(0.f, 0.f);
    }
}

// the free nodes packed with their curvature stencils; and the step kernels'
// frame record (F the free nodes, L the live segments)
__global__ void k_rf_free_nodes(const int* flags, const int2* nbr, Scan<int> pos, int N, FreeNode* out,
                                const unsigned long long* samples_live, int* totals, int ow, int oh, int scale,
                                float inv_samples3, RefineFrame* fr)
{
    follow_last();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) {
        const unsigned long long t = *samples_live;
        totals[2] = (int)(unsigned)t;  // M
        totals[4] = (int)(t >> 32);    // L
        *fr = RefineFrame{N, (int)(t >> 32), ow, oh, scale, *pos.total, inv_samples3};
    }
    if (k >= N || (flags[k] & 1)) return;
    const int2 nb = nbr[k];
    const int2 na = (flags[nb.x] & 1) ? make_int2(-1, -1) : nbr[nb.x];
    const int2 nbb = (flags[nb.y] & 1) ? make_int2(-1, -1) : nbr[nb.y];
    out[pos.at(k)] = FreeNode{make_int4(k, nb.x, nb.y, na.x), make_int4(na.y, nbb.x, nbb.y, 0)};
}

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t cap = 0;
    // grows with a quarter of headroom, so that frames of about the same
    // size reuse the buffer (a free in between would synchronize the device)
    cudaError_t reserve(size_t n)
    {
        if (n <= cap && p) return cudaSuccess;
        dev_free(p);
        p = nullptr;
        cap = 0;
        const size_t want = std::max<size_t>(n + n / 4, 1);
        cudaError_t e = dev_alloc(&p, want * sizeof(T));
        if (e == cudaSuccess) cap = want;
        return e;
    }
    void release()
    {
        dev_free(p);
        p = nullptr;
        cap = 0;
    }
};

}  // namespace

}  // namespace depix

using namespace depix;

struct depix_refiner {
    int device = 0;
    size_t max_pixels = 0;
    int sms = 0;
    const uint64_t* lut = nullptr;
    // frame
    int w = 0, h = 0, scale = 0, ow = 0, oh = 0;
    int E = 0, N = 0, F = 0, S = 0, M = 0; // F, M and L: -1 until read back (fetch_counts)
    int max_split = 0; // split curve edges a cell can own at most (its hull box's lattice steps)
    float sigma = 0.5f; // coverage sigma of the targets (output pixels)
    DevBuf<uint32_t> vgrid;
    DevBuf<uint32_t> box;
    DevBuf<uint8_t> own_graph, own_snap; // resolved graph when the caller gives none
    DevBuf<uint64_t> tile_hash;
    DevBuf<float2> warm_grid;
    DevBuf<int> warm_stamp;
    int tiles_x = 0, tiles = 0, warm_epoch = 0;
    DevBuf<int> cell_count, cell_off, cell_tiles, nid, nid_tiles, free_pos, free_tiles, scalars;
    DevBuf<uint16_t> edge_slots;
    DevBuf<unsigned long long> samp_off, samp_tiles, samp_total;
    DevBuf<int> tickets; // of the four scans
    DevBuf<int2> nb_v, nb_e;
    DevBuf<int4> edges;
    DevBuf<int2> node_q, node_nbr, node_nbr_edge;
    DevBuf<int> node_flags;
    DevBuf<float2> pos0, pos_a, pos_b, gcov, adam_m, adam_v;
    DevBuf<int4> seg;
    DevBuf<uint2> seg_col;
    DevBuf<unsigned long long> best;
    DevBuf<int> bseg, seg_count, seg_off, samp;
    DevBuf<float4> tgt;
    DevBuf<double> energy;
    DevBuf<LiveSeg> live;
    DevBuf<FreeNode> fnodes;
    DevBuf<float2> sxy;
    DevBuf<RefineFrame> frame;
    int L = 0;
    int* h_scalars = nullptr; // pinned
    cudaEvent_t counted = nullptr; // E and N are on the host
    double* h_energy = nullptr;
    bool ready = false;
    // the Adam loop as a graph, replayed while its parameters and buffers stay
    cudaStream_t capture_stream = nullptr;
    cudaGraphExec_t loop = nullptr;
    StepArgs loop_args{};
    int loop_steps = -1;
    int loop_cov_blocks = 0, loop_node_blocks = 0;
    long long captures = 0; // of the loop
};

namespace {

depix_status rf_fail(cudaError_t e, const char* where)
{
    set_last_error(std::string(where) + ": " + cudaGetErrorString(e));
    return DEPIX_ERR_CUDA;
}

#define DEPIX_TRY_RF(call)                                              \
    do {                                                                \
        depix_status st_ = (call);                                      \
        if (st_ != DEPIX_OK) return st_;                                \
    } while (0)

#define RF_CK(call)                                                     \
    do {                                                                \
        cudaError_t e_ = (call);                                        \
        if (e_ != cudaSuccess) return rf_fail(e_, #call);               \
    } while (0)

int blocks_for(long long n, int t = 256) { return (int)std::max<long long>(1, (n + t - 1) / t); }

// scan totals in slots [slot, slot + n), read back to the host (synchronous)
depix_status read_totals(depix_refiner* r, int slot, int n, int* out, cudaStream_t s)
{
    RF_CK(cudaMemcpyAsync(r->h_scalars + slot, r->scalars.p + slot, n * sizeof(int), cudaMemcpyDeviceToHost, s));
    RF_CK(cudaStreamSynchronize(s));
    for (int k = 0; k < n; k++) out[k] = r->h_scalars[slot + k];
    return DEPIX_OK;
}

// M, F and L of the set-up frame (scan totals left on the device by the
// setup), read back when a caller asks for them
depix_status fetch_counts(depix_refiner* r)
{
    if (r->M >= 0) return DEPIX_OK;
    RF_CK(cudaDeviceSynchronize());
    RF_CK(cudaMemcpy(r->h_scalars + 2, r->scalars.p + 2, 3 * sizeof(int), cudaMemcpyDeviceToHost));
    r->M = r->h_scalars[2];
    r->F = r->h_scalars[3];
    r->L = r->h_scalars[4];
    return DEPIX_OK;
}

depix_status check_refiner(depix_refiner* r)
{
    if (!r) {
        set_last_error("NULL refiner");
        return DEPIX_ERR_INVALID_ARG;
    }
    if (!r->ready) {
        set_last_error("refiner has no frame: call depix_refine_setup first");
        return DEPIX_ERR_INVALID_ARG;
    }
    return DEPIX_OK;
}

StepArgs step_args(depix_refiner* r, const depix_refine_params* p)
{
    StepArgs a{};
    a.gcov = r->gcov.p;
    a.x0 = r->pos0.p;
    a.tgt = r->tgt.p;
    a.flags = r->node_flags.p;
    a.live = r->live.p;
    a.sxy = r->sxy.p;
    a.fnodes = r->fnodes.p;
    a.fr = r->frame.p;
    a.m = r->adam_m.p;
    a.v = r->adam_v.p;
    a.sigma = r->sigma;
    a.w_curv = p->w_curvature;
    a.w_dev = p->w_deviation;
    a.w_cov = p->w_coverage;
    a.lr = p->lr;
    return a;
}

depix_status check_rparams(const depix_refine_params* p)
{
    if (!p || !(p->sigma > 0.f) || !(p->lr >= 0.f) || p->steps < 0 || !(p->w_curvature >= 0.f) ||
        !(p->w_deviation >= 0.f) || !(p->w_coverage >= 0.f)) {
        set_last_error("refine params: sigma > 0, lr, weights >= 0, steps >= 0");
        return DEPIX_ERR_INVALID_ARG;
    }
    return DEPIX_OK;
}

depix_status check_sigma(const depix_refiner* r, const depix_refine_params* p)
{
    if (p->sigma != r->sigma) {
        set_last_error("coverage sigma differs from the one the targets were set up with");
        return DEPIX_ERR_INVALID_ARG;
    }
    return DEPIX_OK;
}

// Blocks of a step's two passes for the set-up frame: a group of lanes for every
// live segment and a thread for every free node (F <= N), at most 8 blocks of 256
// threads per SM. One block too few costs every step a second trip (a 256x224
// frame with 324 blocks of live segments: 5.3 us with 320, 4.1 with 352 to 608,
// 4.4 with 1216). The live segments are counted on the device only; they are the
// edges' middles, the nodes' corners and the pinned pieces, in all but noise less
// than 1.2 times the edges and nodes (1.03 in plain frames, 2.0 in noise of random
// colours).
int blocks_needed(long long threads, int block, int most)
{
    return (int)std::min<long long>(std::max<long long>(1, (threads + block - 1) / block), most);
}
int most_cov(const depix_refiner* r) { return r->sms * 8; }
int most_node(const depix_refiner* r) { return r->sms * 32; }
int cov_needed(const depix_refiner* r)
{
    return blocks_needed(((long long)r->E + r->N) * 5 / 4 * kSegLanes, 256, most_cov(r));
}
int node_needed(const depix_refiner* r) { return blocks_needed(r->N, 64, most_node(r)); }

// A captured loop's grid: the need rounded up to a power of two or one and a half
// times one. The kernels stride over the sizes they read on the device, so that
// the loop serves every frame that needs no more, down to a quarter of it
// (loop_fits): frames whose counts move to and fro replay the one captured for
// the largest. (A capture with 20 steps costs 113 us, twice the blocks of a frame
// a tenth of a microsecond a step.)
int grid_for(int need, int most)
{
    int p = 1;
    while (p < need) p <<= 1;
    return std::min(p / 4 * 3 >= need ? p / 4 * 3 : p, most);
}
int cov_blocks(const depix_refiner* r) { return grid_for(cov_needed(r), most_cov(r)); }
int node_blocks(const depix_refiner* r) { return grid_for(node_needed(r), most_node(r)); }
bool loop_fits(int blocks, int need, int grid) { return blocks >= need && blocks <= 4 * grid; }

bool same_loop(const StepArgs& a, const StepArgs& b)
{
    return a.gcov == b.gcov && a.x0 == b.x0 && a.tgt == b.tgt && a.flags == b.flags && a.live == b.live &&
           a.sxy == b.sxy && a.fnodes == b.fnodes && a.fr == b.fr && a.m == b.m && a.v == b.v && a.sigma == b.sigma && a.w_curv == b.w_curv &&
           a.w_dev == b.w_dev && a.w_cov == b.w_cov && a.lr == b.lr;
}

// launches the Adam steps from pos_a (result in pos_a after an even number
// of steps, pos_b after an odd one). A step is two short kernels, bound by the
// latency of their launches and loads (one of a 256x224 frame touches 4 MB in
// L2): 20 steps of it take 135 us when each waits for the other before its first
// load, 98 with early starts (64x64 112 and 82, 1500x1000 1726 and 1655). (One
// kernel that gathers a node's gradient over the five segments that read it,
// evaluating each 2.7 times, took 7.2 us a step where the two took 5.9.)
cudaError_t launch_steps(depix_refiner* r, const StepArgs& base, int steps, cudaStream_t s)
{
    StepArgs a = base;
    float2* x = r->pos_a.p;
    float2* y = r->pos_b.p;
    double b1 = 1.0, b2 = 1.0;
    cudaError_t e = cudaSuccess;
    for (int t = 1; t <= steps && e == cudaSuccess; t++) {
        b1 *= (double)kBeta1;
        b2 *= (double)kBeta2;
        a.x = x;
        a.y = y;
        a.bc1 = (float)(1.0 - b1);
        a.bc2 = (float)(1.0 - b2);
        e = launch_early(true, k_rf_coverage<false>, cov_blocks(r), 256, 0, s, a);
        if (e == cudaSuccess) e = launch_early(true, k_rf_nodes<false>, node_blocks(r), 64, 0, s, a);
        std::swap(x, y);
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
}

// energy (and gradient when gout) at positions x, without an update
depix_status eval(depix_refiner* r, const depix_refine_params* p, const float2* x, float2* gout, double out[4],
                  cudaStream_t s)
{
    StepArgs a = step_args(r, p);
    a.x = x;
    a.gout = gout;
    a.energy = r->energy.p;
    RF_CK(cudaMemsetAsync(r->energy.p, 0, 3 * sizeof(double), s));
    if (gout) RF_CK(cudaMemsetAsync(gout, 0, (size_t)r->N * sizeof(float2), s)); // pinned nodes stay zero
    RF_CK(launch_early(true, k_rf_coverage<true>, cov_blocks(r), 256, 0, s, a));
    RF_CK(launch_early(true, k_rf_nodes<true>, node_blocks(r), 64, 0, s, a));
    RF_CK(cudaMemcpyAsync(r->h_energy, r->energy.p, 3 * sizeof(double), cudaMemcpyDeviceToHost, s));
    RF_CK(cudaStreamSynchronize(s));
    out[0] = r->h_energy[0];
    out[1] = r->h_energy[1];
    out[2] = r->h_energy[2];
    out[3] = out[0] + out[1] + out[2];
    return DEPIX_OK;
}

}  // namespace

extern "C" {

void depix_refine_default_params(depix_refine_params* p)
{
    if (!p) return;
    p->w_curvature = 1.0f;
    p->w_deviation = 0.25f;
    p->w_coverage = 1.0f;
    p->sigma = 0.5f;
    p->lr = 0.05f;
    p->steps = 200;
}

depix_status depix_refiner_create(depix_refiner** out, size_t max_pixels)
{
    if (!out) {
        set_last_error("NULL refiner pointer");
        return DEPIX_ERR_INVALID_ARG;
    }
    *out = nullptr;
    if (max_pixels < 1) {
        set_last_error("capacity must be >= 1");
        return DEPIX_ERR_INVALID_ARG;
    }
    depix_status st = depix_init_device();
    if (st != DEPIX_OK) return st;
    depix_refiner* r = new (std::nothrow) depix_refiner();
    if (!r) return DEPIX_ERR_ALLOC;
    r->max_pixels = max_pixels;
    cudaError_t e = cudaGetDevice(&r->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&r->sms, cudaDevAttrMultiProcessorCount, r->device);
    if (e == cudaSuccess) e = hull_table_address(&r->lut);
    if (e == cudaSuccess) e = r->box.reserve(4096);
    if (e == cudaSuccess) {
        k_rf_boxes<<<16, 256>>>(r->lut, r->box.p);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
    }
    if (e == cudaSuccess) {
        // A cell's split curve edges lie on its convex hull, at most one per
        // quarter-unit lattice step: at most 2 (width + height) of the hull's
        // box, over all patterns.
        std::vector<uint32_t> box(4096);
        e = cudaMemcpy(box.data(), r->box.p, 4096 * sizeof(uint32_t), cudaMemcpyDeviceToHost);
        for (uint32_t b : box) {
            if (b == 0xFFu) continue;
            const int x0 = (int)(b & 0xFF), x1 = (int)((b >> 8) & 0xFF), y0 = (int)((b >> 16) & 0xFF), y1 = (int)(b >> 24);
            r->max_split = std::max(r->max_split, 2 * ((x1 - x0) + (y1 - y0)));
        }
        r->max_split = std::max(r->max_split, 1);
    }
    if (e == cudaSuccess) e = r->scalars.reserve(8);
    if (e == cudaSuccess) e = r->samp_total.reserve(1);
    if (e == cudaSuccess) e = r->tickets.reserve(4);
    if (e == cudaSuccess) e = cudaMemset(r->tickets.p, 0, 4 * sizeof(int));
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&r->counted, cudaEventDisableTiming);
    if (e == cudaSuccess) e = r->energy.reserve(3);
    if (e == cudaSuccess) e = cudaHostAlloc(&r->h_scalars, 8 * sizeof(int), cudaHostAllocDefault);
    if (e == cudaSuccess) e = cudaHostAlloc(&r->h_energy, 4 * sizeof(double), cudaHostAllocDefault);
    if (e == cudaSuccess) e = r->frame.reserve(1);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&r->capture_stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        cudaGetLastError();
        depix_refiner_destroy(r);
        set_last_error(std::string("refiner set-up: ") + cudaGetErrorString(e));
        return DEPIX_ERR_ALLOC;
    }
    *out = r;
    return DEPIX_OK;
}

depix_status depix_refiner_destroy(depix_refiner* r)
{
    if (!r) return DEPIX_OK;
    r->vgrid.release();
    r->box.release();
    r->own_graph.release(); r->own_snap.release(); r->tile_hash.release(); r->warm_grid.release();
    r->warm_stamp.release();
    r->cell_count.release(); r->cell_off.release(); r->cell_tiles.release(); r->nid.release(); r->nid_tiles.release();
    r->free_pos.release(); r->free_tiles.release(); r->scalars.release(); r->edge_slots.release();
    r->samp_off.release(); r->samp_tiles.release(); r->samp_total.release(); r->tickets.release();
    r->nb_v.release(); r->nb_e.release(); r->edges.release();
    r->node_q.release(); r->node_nbr.release(); r->node_nbr_edge.release(); r->node_flags.release();
    r->pos0.release(); r->pos_a.release(); r->pos_b.release(); r->gcov.release();
    r->adam_m.release(); r->adam_v.release();
    r->seg.release(); r->seg_col.release(); r->best.release(); r->bseg.release();
    r->seg_count.release(); r->seg_off.release(); r->samp.release(); r->tgt.release();
    r->energy.release();
    r->live.release(); r->frame.release(); r->fnodes.release(); r->sxy.release();
    if (r->counted) cudaEventDestroy(r->counted);
    if (r->loop) cudaGraphExecDestroy(r->loop);
    if (r->capture_stream) cudaStreamDestroy(r->capture_stream);
    cudaFreeHost(r->h_scalars);
    cudaFreeHost(r->h_energy);
    delete r;
    return DEPIX_OK;
}

depix_status depix_refine_setup(depix_refiner* r, const uint8_t* d_img, int w, int h, int widthstep,
                                depix_layout layout, const uint8_t* d_graph, const depix_params* p,
                                const depix_refine_params* rp, depix_stream s_)
{
    DEPIX_TRY_RF(check_rparams(rp));
    if (!r || !d_img || !p || w < 1 || h < 1) {
        set_last_error("refine setup: NULL argument or size below 1");
        return DEPIX_ERR_INVALID_ARG;
    }
    if ((size_t)w * h > r->max_pixels) {
        set_last_error("frame larger than the refiner capacity");
        return DEPIX_ERR_TOO_LARGE;
    }
    if (p->scale < 1 || p->scale > kMaxRefineScale) {
        set_last_error("refine scale must be in 1..12");
        return DEPIX_ERR_INVALID_ARG;
    }
    if (p->vote != 0 && p->vote != 1) {
        set_last_error("vote must be 0 or 1");
        return DEPIX_ERR_INVALID_ARG;
    }
    if (layout == DEPIX_LAYOUT_RGBA ? (widthstep < 4 * w || (widthstep & 3)) : (layout != DEPIX_LAYOUT_BGR || widthstep < 3 * w)) {
        set_last_error("refine setup: bad layout or widthstep");
        return DEPIX_ERR_INVALID_ARG;
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(s_);
    r->ready = false;
    const int n = w * h, gw = 4 * w + 3, gh = 4 * h + 3, nv = gw * gh;
    if (!d_graph) {
        // the frame's resolved graph: similarity + trivial, then heuristics
        RF_CK(r->own_graph.reserve(n));
        RF_CK(r->own_snap.reserve(n));
        const FrameBatch fb{d_img, 0, r->own_snap.p, 0, w, h, widthstep, (int)layout};
        RF_CK(launch_graph(fb, 1, pack_thresholds(p->tr_y, p->tr_u, p->tr_v, p->yuv), true, s));
        RF_CK(launch_heuristics(GraphBatch{r->own_snap.p, r->own_graph.p, 0, w, h, p->vote}, 1, nullptr, s));
        d_graph = r->own_graph.p;
    }
    Geo G{d_img, widthstep, (int)layout, d_graph, w, h, gw, gh, r->lut, r->box.p,
          pack_thresholds(p->tr_y, p->tr_u, p->tr_v, p->yuv)};
    const int ow = w * p->scale, oh = h * p->scale, no_px = ow * oh;
    RF_CK(r->vgrid.reserve(nv));
    RF_CK(r->cell_count.reserve(n));
    RF_CK(r->cell_off.reserve(n));
    RF_CK(r->cell_tiles.reserve(n / kScanTile + 1));
    RF_CK(r->edge_slots.reserve((size_t)n * r->max_split));
    RF_CK(r->nid.reserve(nv));
    RF_CK(r->nid_tiles.reserve(nv / kScanTile + 1));
    RF_CK(r->nb_v.reserve(nv));
    RF_CK(r->nb_e.reserve(nv));
    RF_CK(r->best.reserve(no_px));
    r->tiles_x = (w + kWarmTile - 1) / kWarmTile;
    r->tiles = r->tiles_x * ((h + kWarmTile - 1) / kWarmTile);
    RF_CK(r->tile_hash.reserve(r->tiles));
    const Scan<int> cells{r->cell_off.p, r->cell_tiles.p, r->scalars.p + 0, r->tickets.p + 0};
    const Scan<int> nid{r->nid.p, r->nid_tiles.p, r->scalars.p + 1, r->tickets.p + 1};
    RF_CK(cudaMemsetAsync(r->vgrid.p, 0, (size_t)nv * sizeof(uint32_t), s));
    // the topology is some twenty short kernels, each started while the one
    // before it ends (us one after the other and so: 64x64 117 and 86, 256x224 142
    // and 112, 640x480 436 and 402, 1500x1000 1717 and 1679)
    RF_CK(launch_early(true, k_rf_mark_vertices, blocks_for(n), 256, 0, s, G, r->vgrid.p));
    RF_CK(launch_early(true, k_rf_count_edges, blocks_for(n, kEdgeCells), kEdgeThreads, 0, s, G, r->vgrid.p,
                       r->max_split, r->cell_count.p, r->edge_slots.p));
    RF_CK(cudaGetLastError());
    RF_CK(exclusive_scan(CellCount{r->cell_count.p}, n, cells, s));
    // edges reserved for the most a frame can have, so that E and N come
    // back together: the one read back of the setup (they size the node and
    // segment arrays; the later counts stay on the device)
    RF_CK(r->edges.reserve((size_t)n * r->max_split));
    RF_CK(launch_early(true, k_rf_emit_edges, blocks_for(n, 128), 128, 0, s, G, r->vgrid.p, r->max_split,
                       r->cell_count.p, cells, r->edge_slots.p, r->edges.p, r->nb_v.p, r->nb_e.p));
    RF_CK(cudaGetLastError());
    RF_CK(exclusive_scan(NodeFlag{r->vgrid.p}, nv, nid, s));
    RF_CK(cudaMemcpyAsync(r->h_scalars, r->scalars.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    RF_CK(cudaEventRecord(r->counted, s));
    // what needs neither runs while the host waits for them
    RF_CK(cudaMemsetAsync(r->best.p, 0xFF, (size_t)no_px * sizeof(unsigned long long), s));
    RF_CK(launch_early(true, k_rf_tile_hash, blocks_for(32LL * r->tiles), 256, 0, s, G, r->tiles_x, r->tiles,
                       r->tile_hash.p));
    RF_CK(cudaGetLastError());
    RF_CK(cudaEventSynchronize(r->counted));
    const int E = r->h_scalars[0], N = r->h_scalars[1];
    RF_CK(r->node_q.reserve(N));
    RF_CK(r->node_flags.reserve(N));
    RF_CK(r->node_nbr.reserve(N));
    RF_CK(r->node_nbr_edge.reserve(N));
    RF_CK(r->pos0.reserve(N));
    RF_CK(r->pos_a.reserve(N));
    RF_CK(r->pos_b.reserve(N));
    RF_CK(r->gcov.reserve((size_t)kParts * N));
    RF_CK(r->adam_m.reserve(N));
    RF_CK(r->adam_v.reserve(N));
    const int S = 3 * E + N;
    RF_CK(r->seg.reserve(S));
    RF_CK(r->seg_col.reserve(S));
    RF_CK(r->seg_count.reserve((size_t)S + 1));
    RF_CK(r->seg_off.reserve((size_t)S + 1));
    RF_CK(r->samp_off.reserve((size_t)S + 1));
    RF_CK(r->samp_tiles.reserve((size_t)S / kScanTile + 1));
    RF_CK(r->free_pos.reserve(N));
    RF_CK(r->free_tiles.reserve((size_t)N / kScanTile + 1));
    RF_CK(r->fnodes.reserve(N));
    RF_CK(r->live.reserve(S));
    // samples (M on the device): at most one per output pixel
    RF_CK(r->samp.reserve(no_px));
    RF_CK(r->tgt.reserve(no_px));
    RF_CK(r->sxy.reserve(no_px));
    NodeOut no{r->node_q.p, r->node_flags.p, r->node_nbr.p, r->node_nbr_edge.p, r->pos0.p, r->gcov.p, N};
    RF_CK(launch_early(true, k_rf_make_nodes, blocks_for(nv), 256, 0, s, G, r->vgrid.p, nid, r->nb_v.p, r->nb_e.p,
                       no));
    RF_CK(launch_early(true, k_rf_segments, blocks_for((long long)E + N), 256, 0, s, G, nid, r->edges.p, E, N,
                       r->node_flags.p, r->node_nbr.p, r->node_nbr_edge.p, SegOut{r->seg.p, r->seg_col.p}));
    RF_CK(cudaGetLastError());
    // sample assignment
    const Scan<unsigned long long> soff{r->samp_off.p, r->samp_tiles.p, r->samp_total.p, r->tickets.p + 2};
    const int box_blocks = blocks_for((long long)S * kBoxLanes);
    Owner own{r->best.p, nullptr, 0};
    int bits = 1;
    while (((long long)1 << bits) <= S) bits++;
    if (12 + frac_bits(p->scale) + bits <= 64) {
        own.slot_bits = bits;
    } else {
        RF_CK(r->bseg.reserve(no_px));
        RF_CK(cudaMemsetAsync(r->bseg.p, 0x7F, (size_t)no_px * sizeof(int), s)); // above every slot
    }
    RF_CK(launch_early(true, k_rf_assign<false>, box_blocks, 256, 0, s, r->seg.p, S, r->node_q.p, p->scale, ow, oh,
                       own));
    if (!own.slot_bits) {
        own.bseg = r->bseg.p;
        RF_CK(launch_early(true, k_rf_assign<true>, box_blocks, 256, 0, s, r->seg.p, S, r->node_q.p, p->scale, ow, oh,
                           own));
    }
    RF_CK(launch_early(true, k_rf_count_samples, box_blocks, 256, 0, s, r->seg.p, S, r->node_q.p, p->scale, ow, oh,
                       own, r->seg_count.p));
    RF_CK(cudaGetLastError());
    RF_CK(exclusive_scan(SampleCount{r->seg_count.p}, S, soff, s));
    RF_CK(launch_early(true, k_rf_fill_samples, box_blocks, 256, 0, s, r->seg.p, S, r->node_q.p, p->scale, ow, oh,
                       own, r->seg_count.p, soff, r->seg_col.p, r->samp.p, r->seg_off.p, r->node_nbr_edge.p,
                       r->live.p));
    // free nodes and their curvature stencils, and the frame record
    const Scan<int> free_pos{r->free_pos.p, r->free_tiles.p, r->scalars.p + 3, r->tickets.p + 3};
    RF_CK(exclusive_scan(FreeFlag{r->node_flags.p}, N, free_pos, s));
    RF_CK(launch_early(true, k_rf_free_nodes, blocks_for(N), 256, 0, s, r->node_flags.p, r->node_nbr.p, free_pos, N,
                       r->fnodes.p, r->samp_total.p, r->scalars.p, ow, oh, p->scale,
                       (float)(1.0 / (3.0 * (double)ow * (double)oh)), r->frame.p));
    RF_CK(launch_early(true, k_rf_targets, std::min(blocks_for(no_px), r->sms * 8), 256, 0, s, G, p->scale,
                       rp->sigma / (float)p->scale, r->samp.p, r->scalars.p + 2, r->tgt.p, r->sxy.p));
    RF_CK(cudaGetLastError());
    r->w = w;
    r->h = h;
    r->scale = p->scale;
    r->ow = ow;
    r->oh = oh;
    r->E = E;
    r->N = N;
    r->S = S;
    r->F = r->M = r->L = -1; // on the device until fetch_counts
    r->sigma = rp->sigma;
    r->ready = true; // the rest is ordered on s: later calls on s see the frame, others wait on an event of s
    return DEPIX_OK;
}

depix_status depix_refine_counts(depix_refiner* r, long long counts[5])
{
    DEPIX_TRY_RF(check_refiner(r));
    if (!counts) {
        set_last_error("NULL counts");
        return DEPIX_ERR_INVALID_ARG;
    }
    DEPIX_TRY_RF(fetch_counts(r));
    counts[0] = r->N;
    counts[1] = r->F;
    counts[2] = r->E;
    counts[3] = r->S;
    counts[4] = r->M;
    return DEPIX_OK;
}

depix_status depix_refine_export(depix_refiner* r, int32_t* node_q, int32_t* node_flags, int32_t* node_nbr,
                                 int32_t* edges, int32_t* segs, uint32_t* seg_colors, int32_t* samples)
{
    DEPIX_TRY_RF(check_refiner(r));
    DEPIX_TRY_RF(fetch_counts(r));
    if (node_q) RF_CK(cudaMemcpy(node_q, r->node_q.p, (size_t)r->N * sizeof(int2), cudaMemcpyDeviceToHost));
    if (node_flags) RF_CK(cudaMemcpy(node_flags, r->node_flags.p, (size_t)r->N * sizeof(int), cudaMemcpyDeviceToHost));
    if (node_nbr) RF_CK(cudaMemcpy(node_nbr, r->node_nbr.p, (size_t)r->N * sizeof(int2), cudaMemcpyDeviceToHost));
    if (edges) {
        // vertex indices -> node ids on the host copy
        std::vector<int4> ev(r->E);
        std::vector<int> nid((size_t)(4 * r->w + 3) * (4 * r->h + 3)), tiles(nid.size() / kScanTile + 1);
        RF_CK(cudaMemcpy(ev.data(), r->edges.p, (size_t)r->E * sizeof(int4), cudaMemcpyDeviceToHost));
        RF_CK(cudaMemcpy(nid.data(), r->nid.p, nid.size() * sizeof(int), cudaMemcpyDeviceToHost));
        RF_CK(cudaMemcpy(tiles.data(), r->nid_tiles.p, tiles.size() * sizeof(int), cudaMemcpyDeviceToHost));
        for (size_t v = 0; v < nid.size(); v++) nid[v] += tiles[v / kScanTile];
        for (int e = 0; e < r->E; e++) {
            edges[4 * e] = nid[ev[e].x];
            edges[4 * e + 1] = nid[ev[e].y];
            edges[4 * e + 2] = ev[e].z;
            edges[4 * e + 3] = ev[e].w;
        }
    }
    if (segs) RF_CK(cudaMemcpy(segs, r->seg.p, (size_t)r->S * sizeof(int4), cudaMemcpyDeviceToHost));
    if (seg_colors) RF_CK(cudaMemcpy(seg_colors, r->seg_col.p, (size_t)r->S * sizeof(uint2), cudaMemcpyDeviceToHost));
    if (samples) {
        std::vector<int> off((size_t)r->S + 1), smp(r->M);
        RF_CK(cudaMemcpy(off.data(), r->seg_off.p, off.size() * sizeof(int), cudaMemcpyDeviceToHost));
        RF_CK(cudaMemcpy(smp.data(), r->samp.p, smp.size() * sizeof(int), cudaMemcpyDeviceToHost));
        for (int sg = 0; sg < r->S; sg++)
            for (int m = off[sg]; m < off[sg + 1]; m++) {
                samples[2 * m] = smp[m];
                samples[2 * m + 1] = sg;
            }
    }
    return DEPIX_OK;
}

depix_status depix_refine_initial(depix_refiner* r, float* d_pos, depix_stream s)
{
    DEPIX_TRY_RF(check_refiner(r));
    if (!d_pos) {
        set_last_error("NULL positions");
        return DEPIX_ERR_INVALID_ARG;
    }
    RF_CK(cudaMemcpyAsync(d_pos, r->pos0.p, (size_t)r->N * sizeof(float2), cudaMemcpyDeviceToDevice,
                          reinterpret_cast<cudaStream_t>(s)));
    return DEPIX_OK;
}

depix_status depix_refine_warm_start(depix_refiner* r, const depix_refiner* prev, const float* d_prev_pos,
                                     float* d_pos, int* reused_tiles, depix_stream s_)
{
    DEPIX_TRY_RF(check_refiner(r));
    if (!prev || !prev->ready || !d_prev_pos || !d_pos) {
        set_last_error("warm start: previous refiner without a frame, or NULL positions");
        return DEPIX_ERR_INVALID_ARG;
    }
    if (prev->w != r->w || prev->h != r->h) {
        set_last_error("warm start: the previous frame has another size");
        return DEPIX_ERR_INVALID_ARG;
    }
    cudaStream_t s = reinterpret_cast<cudaStream_t>(s_);
    const int gw = 4 * r->w + 3, nv = gw * (4 * r->h + 3);
    if (r->warm_grid.cap < (size_t)nv || !r->warm_grid.p) {
        RF_CK(r->warm_grid.reserve(nv));
        RF_CK(r->warm_stamp.reserve(nv));
        RF_CK(cudaMemsetAsync(r->warm_stamp.p, 0, (size_t)nv * sizeof(int), s));
        r->warm_epoch = 0;
    }
    const int epoch = ++r->warm_epoch;
    RF_CK(launch_early(true, k_rf_warm_scatter, blocks_for(prev->N), 256, 0, s, prev->node_q.p,
                       reinterpret_cast<const float2*>(d_prev_pos), prev->N, gw, r->warm_grid.p, r->warm_stamp.p, epoch));
    RF_CK(launch_early(true, k_rf_warm_gather, blocks_for(r->N), 256, 0, s, r->node_q.p, r->pos0.p, r->N, r->w, r->h,
                       gw, r->tiles_x, r->tile_hash.p, prev->tile_hash.p, r->warm_grid.p, r->warm_stamp.p, epoch,
                       reinterpret_cast<float2*>(d_pos)));
    RF_CK(cudaGetLastError());
    if (reused_tiles) {
        RF_CK(cudaMemsetAsync(r->scalars.p + 5, 0, sizeof(int), s));
        RF_CK(launch_early(true, k_rf_same_tiles, blocks_for(r->tiles), 256, 0, s, r->tile_hash.p, prev->tile_hash.p,
                           r->tiles, r->scalars.p + 5));
        RF_CK(cudaGetLastError());
        DEPIX_TRY_RF(read_totals(r, 5, 1, reused_tiles, s));
    }
    return DEPIX_OK;
}

depix_status depix_debug_refine_captures(const depix_refiner* r, long long* count)
{
    if (!r || !count) {
        set_last_error("NULL refiner or count");
        return DEPIX_ERR_INVALID_ARG;
    }
    *count = r->captures;
    return DEPIX_OK;
}

depix_status depix_refine_energy_grad(depix_refiner* r, const depix_refine_params* p, const float* d_pos,
                                      float* d_grad, double energy[4], depix_stream s)
{
    DEPIX_TRY_RF(check_refiner(r));
    DEPIX_TRY_RF(check_rparams(p));
    DEPIX_TRY_RF(check_sigma(r, p));
    if (!d_pos || !energy) {
        set_last_error("NULL positions or energy");
        return DEPIX_ERR_INVALID_ARG;
    }
    return eval(r, p, reinterpret_cast<const float2*>(d_pos), reinterpret_cast<float2*>(d_grad), energy,
                reinterpret_cast<cudaStream_t>(s));
}

depix_status depix_refine_run(depix_refiner* r, const depix_refine_params* p, float* d_pos, double before[4],
                              double after[4], depix_stream s_)
{
    DEPIX_TRY_RF(check_refiner(r));
    DEPIX_TRY_RF(check_rparams(p));
    DEPIX_TRY_RF(check_sigma(r, p));
    cudaStream_t s = reinterpret_cast<cudaStream_t>(s_);
    const size_t bytes = (size_t)r->N * sizeof(float2);
    float2* x = r->pos_a.p;
    float2* y = r->pos_b.p;
    RF_CK(launch_early(true, k_rf_begin, std::min(blocks_for(r->N), r->sms * 4), 256, 0, s,
                       d_pos ? reinterpret_cast<const float2*>(d_pos) : r->pos0.p, x, y, r->adam_m.p, r->adam_v.p, r->N));
    RF_CK(cudaGetLastError());
    if (before) DEPIX_TRY_RF(eval(r, p, x, nullptr, before, s));
    const StepArgs a = step_args(r, p);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    RF_CK(cudaStreamIsCapturing(s, &cs));
    if (p->steps > 0 && cs == cudaStreamCaptureStatusNone) {
        if (!r->loop || r->loop_steps != p->steps || !same_loop(a, r->loop_args) ||
            r->loop_args.x != r->pos_a.p || r->loop_args.y != r->pos_b.p ||
            !loop_fits(r->loop_cov_blocks, cov_needed(r), cov_blocks(r)) ||
            !loop_fits(r->loop_node_blocks, node_needed(r), node_blocks(r))) {
            if (r->loop) cudaGraphExecDestroy(r->loop);
            r->loop = nullptr;
            RF_CK(cudaStreamBeginCapture(r->capture_stream, cudaStreamCaptureModeThreadLocal));
            cudaError_t e = launch_steps(r, a, p->steps, r->capture_stream);
            cudaGraph_t g = nullptr;
            const cudaError_t e2 = cudaStreamEndCapture(r->capture_stream, &g);
            if (e == cudaSuccess) e = e2;
            if (e == cudaSuccess) e = cudaGraphInstantiate(&r->loop, g, 0);
            if (g) cudaGraphDestroy(g);
            if (e != cudaSuccess) {
                r->loop = nullptr;
                return rf_fail(e, "refine loop capture");
            }
            r->captures++;
            r->loop_args = a;
            r->loop_args.x = r->pos_a.p;
            r->loop_args.y = r->pos_b.p;
            r->loop_steps = p->steps;
            r->loop_cov_blocks = cov_blocks(r);
            r->loop_node_blocks = node_blocks(r);
        }
        RF_CK(cudaGraphLaunch(r->loop, s));
    } else {
        RF_CK(launch_steps(r, a, p->steps, s));
    }
    if (p->steps & 1) x = y;
    if (after) DEPIX_TRY_RF(eval(r, p, x, nullptr, after, s));
    if (d_pos) RF_CK(cudaMemcpyAsync(d_pos, x, bytes, cudaMemcpyDeviceToDevice, s));
    return DEPIX_OK;
}

}  // extern "C"
