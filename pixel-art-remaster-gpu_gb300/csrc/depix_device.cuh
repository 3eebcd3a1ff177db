// depix_device.cuh -- device-side building blocks shared by the kernels.
//
// Geometry is carried in exact integers: every coordinate the reference
// produces is a multiple of 1/64 of a cell (hull points are multiples of
// 1/4, one corner-cutting round and the neighbour midpoints add three more
// halvings), and its float and double arithmetic on such values is exact. So
// the hull, subdivision and ear-clip decisions below, made on integers in
// 1/64-cell units, are the reference's decisions bit for bit.
#pragma once

#include <cstdint>
#include <cuda.h> // CUtensorMap (the type only; the encoder comes through the runtime's driver entry point)
#include <cuda_runtime.h>

#include "../../include/depix.h"

namespace depix {

constexpr int kCell = 45;    // slots per cell in the VBO layout (kernel.cu:8)
constexpr int kMaxHull = 8;  // largest reshaped-cell hull over all 4096 patterns
constexpr int kMaxPoly = 16; // one subdivision round at most doubles the hull
constexpr int kUnit = 64;    // geometry units per cell

// neighbour offset of node bit e (graph_functions.cu:162-235), j upward
__host__ __device__ __forceinline__ int dir_di(int e) { return ((0x9224 >> (2 * e)) & 3) - 1; }
__host__ __device__ __forceinline__ int dir_dj(int e) { return ((0x016A >> (2 * e)) & 3) - 1; }
__host__ __device__ __forceinline__ int bitof(unsigned v, int k) { return (int)((v >> k) & 1u); }

// bits of a node whose neighbour lies inside the image
__device__ __forceinline__ unsigned inside_mask(int x, int y, int w, int h)
{
    unsigned m = 0xFFu;
    if (x == 0) m &= ~0x29u;     // 0, 3, 5
    if (x == w - 1) m &= ~0x94u; // 2, 4, 7
    if (y == 0) m &= ~0xE0u;     // 5, 6, 7
    if (y == h - 1) m &= ~0x07u; // 0, 1, 2
    return m;
}

// Bytes (x .. x + 3, y) of a w x h byte image, zero outside: two aligned words
// shifted together where both lie in the image's memory (rows of odd widths
// start anywhere), else byte by byte. (A byte a load: 877 frames of 33x108 at
// x10 654 us, 622 with it in the heuristics and the raster; 32 of 159x143 at x3
// 63.2 and 62.0.)
__device__ __forceinline__ uint32_t row_bytes4(const uint8_t* g, int w, int h, int x, int y)
{
    if (y < 0 || y >= h || x <= -4 || x >= w) return 0;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(g), a = lo + (size_t)y * w + (ptrdiff_t)x, a0 = a & ~(uintptr_t)3;
    uint32_t v = 0;
    if (a0 >= lo && a0 + 8 <= lo + (size_t)w * h) {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(a0);
        v = __funnelshift_r(p[0], p[1], 8 * (unsigned)(a & 3));
        if (x < 0) v &= ~0u << (-8 * x);
        if (x + 4 > w) v &= ~0u >> (8 * (x + 4 - w));
    } else {
        for (int q = 0; q < 4; q++)
            if (x + q >= 0 && x + q < w) v |= (uint32_t)g[(size_t)y * w + x + q] << (8 * q);
    }
    return v;
}

// inside_mask of the four nodes (x .. x + 3, y), a byte each
__device__ __forceinline__ uint32_t inside_mask4(int x, int y, int w, int h)
{
    uint32_t m = ~0u;
    if (y == 0) m &= ~0xE0E0E0E0u;
    if (y == h - 1) m &= ~0x07070707u;
    if (x <= 0 && x > -4) m &= ~(0x29u << (-8 * x));
    if (x < w && x + 4 >= w) m &= ~(0x94u << (8 * (w - 1 - x)));
    return m;
}

// load(k) for k = threadIdx.x, + blockDim.x, ... below n, U of them in flight
// before their store(k, value)
template <int U, typename Load, typename Store>
__device__ __forceinline__ void for_each_batched(int n, Load load, Store store)
{
    for (int k0 = threadIdx.x; k0 < n; k0 += U * blockDim.x) {
        uint32_t v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k0 + u * (int)blockDim.x < n) v[u] = load(k0 + u * (int)blockDim.x);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k0 + u * (int)blockDim.x < n) store(k0 + u * (int)blockDim.x, v[u]);
    }
}

// ------------------------------------------------------------------ colour

// Packed Y/U/V word of one pixel from its bytes in the reference's memory
// order (b0 plays "r", b2 plays "b": RGBtoYUV + DATAtoINT,
// graph_functions.cu:80-131). y is the truncated double 0.299 r + 0.587 g +
// 0.114 b, evaluated as one of the reference's two builds evaluates it
// (depix_params.yuv):
//  - DEPIX_YUV_CUDA: its CUDA build (nvcc contracts the sum into fused
//    multiply-adds): fma(0.114, b, fma(0.299, r, 0.587 g));
//  - DEPIX_YUV_HOST: its host build, IEEE with no contraction:
//    (0.299 r + 0.587 g) + 0.114 b.
// Off exact multiples of 1/1000 the sum is at least 0.001 away from an
// integer, and either evaluation truncates to the integer quotient of
// 299 r + 587 g + 114 b by 1000; only a zero remainder needs the double
// evaluation, where the two builds differ for 2490 of the 2^24 colours.
__device__ __forceinline__ uint32_t yuv_word(int r, int g, int b, int mode)
{
    int s = 299 * r + 587 * g + 114 * b;
    int y = s / 1000;
    if (s - y * 1000 == 0) {
        double t;
        if (mode == DEPIX_YUV_HOST) {
            t = __dadd_rn(__dmul_rn(0.299, (double)r), __dmul_rn(0.587, (double)g));
            t = __dadd_rn(t, __dmul_rn(0.114, (double)b));
        } else {
            t = __fma_rn(0.114, (double)b, __fma_rn(0.299, (double)r, __dmul_rn(0.587, (double)g)));
        }
        y = __double2int_rz(t);
    }
    int u = __float2int_rz(__fmul_rn((float)(b - y), 0.492f));
    int v = __float2int_rz(__fmul_rn((float)(r - y), 0.877f));
    return (uint32_t)(y * 65536 + u * 256 + v);
}

// Thresholds packed like a word (a field threshold above 255 can never be
// exceeded), with the y arithmetic (depix_params.yuv) in bits 24-31: the
// similarity test ignores that byte, so the kernels that build words carry
// the mode in the thresholds they already take.
__host__ __device__ __forceinline__ uint32_t pack_thresholds(int ty, int tu, int tv, int yuv)
{
    auto c = [](int t) { return (uint32_t)(t < 0 ? 0 : (t > 255 ? 255 : t)); };
    return ((uint32_t)(yuv & 0xFF) << 24) | (c(ty) << 16) | (c(tu) << 8) | c(tv);
}

__host__ __device__ __forceinline__ int yuv_mode_of(uint32_t thr) { return (int)(thr >> 24); }

// similarity of two words: every masked field within its threshold
// (graph_functions.cu:291-293)
__device__ __forceinline__ bool similar(uint32_t a, uint32_t b, uint32_t thr)
{
    return (__vcmpleu4(__vabsdiffu4(a, b), thr) & 0x00FFFFFFu) == 0x00FFFFFFu;
}

// Reference-layout bytes of one pixel (b0, b1, b2) packed little-endian.
__device__ __forceinline__ uint32_t load_bgr(const uint8_t* img, int ws, int layout, int i, int j)
{
    if (layout == DEPIX_LAYOUT_RGBA) {
        uint32_t p = reinterpret_cast<const uint32_t*>(img + (size_t)j * ws)[i];
        // RGBA -> B,G,R
        return ((p >> 16) & 0xFFu) | (p & 0xFF00u) | ((p & 0xFFu) << 16);
    }
    const uint8_t* q = img + (size_t)j * ws + 3 * i;
    return (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16);
}

// word of packed bytes c = b0 | b1 << 8 | b2 << 16 under the y arithmetic
// carried in the packed thresholds thr
__device__ __forceinline__ uint32_t word_of_bgr(uint32_t c, uint32_t thr)
{
    return yuv_word((int)(c & 0xFF), (int)((c >> 8) & 0xFF), (int)((c >> 16) & 0xFF), yuv_mode_of(thr));
}

// Byte at linear offset `off` of the reference's BGR image (rows `vws` bytes,
// 3*w used, zero padding), zero outside the image. For RGBA input the
// reference image is the 4-byte-aligned BGR image it would have loaded.
__device__ __forceinline__ int ref_byte(const uint8_t* img, int w, int h, int ws, int layout, long long off)
{
    if (layout == DEPIX_LAYOUT_BGR) {
        if (off < 0 || off >= (long long)h * ws) return 0;
        return img[off];
    }
    int vws = (3 * w + 3) & ~3;
    if (off < 0 || off >= (long long)h * vws) return 0;
    int row = (int)(off / vws), col = (int)(off % vws);
    if (col >= 3 * w) return 0;
    int px = col / 3, ch = col % 3; // ch 0 = B, 1 = G, 2 = R
    return img[(size_t)row * ws + 4 * px + (2 - ch)];
}

__device__ __forceinline__ int ref_stride(int w, int ws, int layout)
{
    return layout == DEPIX_LAYOUT_BGR ? ws : ((3 * w + 3) & ~3);
}

// The three bytes at a linear offset (isColorEqual compares them,
// subdivision_functions.cu:157-167).
__device__ __forceinline__ uint32_t ref_color(const uint8_t* img, int w, int h, int ws, int layout, long long off)
{
    if (layout == DEPIX_LAYOUT_BGR && off >= 0 && off + 2 < (long long)h * ws) {
        const uint8_t* q = img + off;
        return (uint32_t)q[0] | (uint32_t)q[1] << 8 | (uint32_t)q[2] << 16;
    }
    return (uint32_t)ref_byte(img, w, h, ws, layout, off) | (uint32_t)ref_byte(img, w, h, ws, layout, off + 1) << 8 |
           (uint32_t)ref_byte(img, w, h, ws, layout, off + 2) << 16;
}

// T-junction test at vertex (cx, cy) of cell (i, j) (checkTJunction,
// subdivision_functions.cu:170-242): its bounds test (written with the width
// in place of the stride) answers true for any vertex; past it only the four
// corners can answer true. Reads the image through linear offsets.
static __device__ __noinline__ bool t_junction_global(const uint8_t* img, int w, int h, int ws, int layout, int i, int j,
                                               int cx, int cy)
{
    long long st = ref_stride(w, ws, layout);
    long long index = (long long)j * st + (long long)i * 3;
    if ((index - st - 1) < 0 || (index + w + 1) > ((long long)h * st - 1)) return true;
    if ((cx != 0 && cx != kUnit) || (cy != 0 && cy != kUnit)) return false;
    // the neighbours beside, across and above or below the corner
    const long long dx = cx == 0 ? -3 : 3, dy = cy == 0 ? -st : st;
    const uint32_t across = ref_color(img, w, h, ws, layout, index + dy + dx);
    const uint32_t beside = ref_color(img, w, h, ws, layout, index + dx);
    return (beside != across) | (across != ref_color(img, w, h, ws, layout, index + dy));
}

// ------------------------------------------------------- cell pattern tables

// Pattern of a cell: node byte (bits 0-7), left neighbour bit 2 (8) and
// bit 7 (9), right neighbour bit 0 (10) and bit 5 (11): all that decides its
// reshaped polygon (createCellFromPattern, diagram_functions.cu:320-520).
__device__ __forceinline__ int cell_pattern(unsigned node, unsigned left, unsigned right)
{
    return (int)(node & 0xFF) | (bitof(left, 2) << 8) | (bitof(left, 7) << 9) | (bitof(right, 0) << 10) |
           (bitof(right, 5) << 11);
}

// A cell polygon in 1/64-cell units. Every vertex lies in [-0.75, 1.75] of
// its cell (hull points in [-0.25, 1.25]; subdivision midpoints pair an own
// point with a neighbour's), i.e. in [-48, 112]: int8 storage keeps the
// per-thread arrays small.
struct Poly {
    int n;
    int8_t x[kMaxPoly];
    int8_t y[kMaxPoly];
};

// Decodes a hull table entry (built once per device in depix_geom.cu):
// vertex count in bits 0-3, then 8 vertices of 6 bits (x+1 | (y+1) << 3,
// quarter units).
__device__ __forceinline__ void hull_from_lut(uint64_t e, Poly& p)
{
    p.n = (int)(e & 0xF);
#pragma unroll
    for (int t = 0; t < kMaxHull; t++) {
        unsigned v = (unsigned)(e >> (4 + 6 * t)) & 63u;
        p.x[t] = (int8_t)(((int)(v & 7) - 1) * (kUnit / 4));
        p.y[t] = (int8_t)(((int)(v >> 3) - 1) * (kUnit / 4));
    }
}

// ------------------------------------------------------------- subdivision

__device__ __forceinline__ int pmod(int i, int n) { return (n + (i % n)) % n; }

// Neighbour direction an edge is shared with, or -1 (isLinkedEdge,
// subdivision_functions.cu:245-424). In integer units the float slope test
// "== +-1" is dy == +-dx with dx != 0, and the 0.5 tests compare with 32.
__device__ __forceinline__ int edge_link(const Poly& c, unsigned node, int idx)
{
    int b = pmod(idx + 1, c.n);
    int ax = c.x[idx], ay = c.y[idx], bx = c.x[b], by = c.y[b];
    int dx = bx - ax, dy = by - ay, my2 = ay + by;
    const int half = kUnit / 2;
    if (ay == by && ay > half && bitof(node, 1)) return 1;
    if (ax == bx && ax > half && bitof(node, 4)) return 4;
    if (ay == by && ay < half && bitof(node, 6)) return 6;
    if (ax == bx && ax < half && bitof(node, 3)) return 3;
    bool s1 = dx != 0 && dy == dx, sm1 = dx != 0 && dy == -dx;
    if (s1 && my2 > kUnit && bitof(node, 0)) return 0;
    if (sm1 && my2 > kUnit && bitof(node, 2)) return 2;
    if (s1 && my2 < kUnit && bitof(node, 7)) return 7;
    if (sm1 && my2 < kUnit && bitof(node, 5)) return 5;
    return -1;
}

// corner-cutting points on edge i -> i+1 (getQ_i / getR_i,
// subdivision_functions.cu:42-122): 3/4-1/4 when the edge is at most one cell
// long, else 7/8-1/8.
__device__ __forceinline__ void qr_point(const Poly& c, int i, bool want_r, int& ox, int& oy)
{
    int a = i % c.n;
    if (a < 0) a += c.n;
    int b = (i + 1) % c.n;
    int px = c.x[a], py = c.y[a], nx = c.x[b], ny = c.y[b];
    int l2 = (nx - px) * (nx - px) + (ny - py) * (ny - py);
    if (l2 <= kUnit * kUnit) {
        if (want_r) { ox = (px + 3 * nx) / 4; oy = (py + 3 * ny) / 4; }
        else { ox = (3 * px + nx) / 4; oy = (3 * py + ny) / 4; }
    } else {
        if (want_r) { ox = (px + 7 * nx) / 8; oy = (py + 7 * ny) / 8; }
        else { ox = (7 * px + nx) / 8; oy = (7 * py + ny) / 8; }
    }
}

// Q (or R) point of a linked neighbour's hull around the vertex matching
// (px, py), mapped back to this cell (get{Q,R}_i_from_linked_cell,
// subdivision_functions.cu:125-154; getPointIndex falls back to index 0).
__device__ __forceinline__ void linked_point(const Poly& nb, int link, int px, int py, bool want_r, int& ox,
                                             int& oy)
{
    int tx = px - kUnit * dir_di(link), ty = py - kUnit * dir_dj(link);
    int op = 0;
    for (int t = 0; t < nb.n; t++)
        if (nb.x[t] == tx && nb.y[t] == ty) { op = t; break; }
    qr_point(nb, want_r ? op - 1 : op, want_r, ox, oy);
    ox += kUnit * dir_di(link);
    oy += kUnit * dir_dj(link);
}

// One corner-cutting round of a cell (subdivision, subdivision_functions.cu:564-669).
// NbHull(link, Poly&) fetches the hull of the neighbour in direction link;
// TJ(cx, cy) is the T-junction test at a cell corner.
template <typename NbHull, typename TJ>
__device__ void subdivide_cell(const Poly& c, unsigned node, NbHull nb_hull, TJ tj, Poly& out)
{
    int link[kMaxHull];
    for (int e = 0; e < c.n; e++) link[e] = edge_link(c, node, e);
    int m = 0;
    Poly nb;
    for (int v = 0; v < c.n; v++) {
        int lp = link[pmod(v - 1, c.n)];
        bool cur = link[v] >= 0, prev = lp >= 0;
        int px = c.x[v], py = c.y[v];
        if (!cur && !prev) {
            // the test's image-bounds check answers "keep" for any vertex of
            // the cells it covers, before it looks at corners
            if (tj(px, py)) {
                out.x[m] = (int8_t)px; out.y[m] = (int8_t)py; m++;
            } else {
                int rx, ry, qx, qy;
                qr_point(c, v - 1, true, rx, ry);
                qr_point(c, v, false, qx, qy);
                out.x[m] = (int8_t)rx; out.y[m] = (int8_t)ry; m++;
                out.x[m] = (int8_t)qx; out.y[m] = (int8_t)qy; m++;
            }
        } else if (!cur && prev) {
            int qx, qy, ax, ay;
            qr_point(c, v, false, qx, qy);
            nb_hull(lp, nb);
            linked_point(nb, lp, px, py, true, ax, ay);
            out.x[m] = (int8_t)((qx + ax) / 2); out.y[m] = (int8_t)((qy + ay) / 2); m++;
            out.x[m] = (int8_t)qx; out.y[m] = (int8_t)qy; m++;
        } else if (cur && !prev) {
            int rx, ry, ax, ay;
            nb_hull(link[v], nb);
            linked_point(nb, link[v], px, py, false, ax, ay);
            qr_point(c, v - 1, true, rx, ry);
            out.x[m] = (int8_t)rx; out.y[m] = (int8_t)ry; m++;
            out.x[m] = (int8_t)((rx + ax) / 2); out.y[m] = (int8_t)((ry + ay) / 2); m++;
        } else {
            out.x[m] = (int8_t)px; out.y[m] = (int8_t)py; m++;
        }
    }
    out.n = m;
}

// ----------------------------------------------------------- ear clipping

__device__ __forceinline__ bool inside_tri(int Ax, int Ay, int Bx, int By, int Cx, int Cy, int Px, int Py)
{
    int a = (Cx - Bx) * (Py - By) - (Cy - By) * (Px - Bx);
    int c = (Bx - Ax) * (Py - Ay) - (By - Ay) * (Px - Ax);
    int b = (Ax - Cx) * (Py - Cy) - (Ay - Cy) * (Px - Cx);
    return a >= 0 && b >= 0 && c >= 0;
}

// Ear clipping (process / snip / area, triangulate_functions.cu:6-217) in
// integer units: the reference's EPSILON test on an exact product of
// 1/64-multiples is "cross <= 0". Writes corner indices, returns the triangle
// count; ok = false when the reference's loop guard gives up.
__device__ __forceinline__ int ear_clip(const Poly& c, uint8_t* tri, bool& ok)
{
    ok = true;
    int n = c.n;
    if (n < 3) { ok = false; return 0; }
    int area = 0;
    for (int p = n - 1, q = 0; q < n; p = q++) area += c.x[p] * c.y[q] - c.x[q] * c.y[p];
    uint8_t V[kMaxPoly];
    for (int v = 0; v < n; v++) V[v] = (uint8_t)(area > 0 ? v : (n - 1) - v);
    int nv = n, nt = 0, count = 2 * nv;
    for (int v = nv - 1; nv > 2;) {
        if (0 >= (count--)) { ok = false; return nt; }
        int u = v;
        if (nv <= u) u = 0;
        v = u + 1;
        if (nv <= v) v = 0;
        int w = v + 1;
        if (nv <= w) w = 0;
        int Ax = c.x[V[u]], Ay = c.y[V[u]], Bx = c.x[V[v]], By = c.y[V[v]], Cx = c.x[V[w]], Cy = c.y[V[w]];
        bool ear = ((Bx - Ax) * (Cy - Ay) - (By - Ay) * (Cx - Ax)) > 0;
        if (ear) {
            // a point outside the triangle's bounding box cannot be inside or on it
            const int x0 = min(Ax, min(Bx, Cx)), x1 = max(Ax, max(Bx, Cx));
            const int y0 = min(Ay, min(By, Cy)), y1 = max(Ay, max(By, Cy));
            for (int p = 0; p < nv; p++) {
                if (p == u || p == v || p == w) continue;
                const int Px = c.x[V[p]], Py = c.y[V[p]];
                if (Px < x0 || Px > x1 || Py < y0 || Py > y1) continue;
                if (inside_tri(Ax, Ay, Bx, By, Cx, Cy, Px, Py)) { ear = false; break; }
            }
        }
        if (ear) {
            tri[3 * nt] = (uint8_t)V[u];
            tri[3 * nt + 1] = (uint8_t)V[v];
            tri[3 * nt + 2] = (uint8_t)V[w];
            nt++;
            for (int s = v, t = v + 1; t < nv; s++, t++) V[s] = V[t];
            nv--;
            count = 2 * nv;
        }
    }
    return nt;
}

// ------------------------------------------------------------------ raster

// Sample coverage of one triangle under the top-left rule, all in integer
// units of 1/256 output pixel relative to a common origin. The triangle is
// taken counter-clockwise (y up); zero area covers nothing.
__device__ __forceinline__ bool covers(int ax, int ay, int bx, int by, int cx, int cy, int sx, int sy)
{
    int area = (bx - ax) * (cy - ay) - (by - ay) * (cx - ax);
    if (area == 0) return false;
    if (area < 0) {
        int tx = bx, ty = by;
        bx = cx; by = cy; cx = tx; cy = ty;
    }
    int ex, ey, f;
    ex = bx - ax; ey = by - ay; f = ex * (sy - ay) - ey * (sx - ax);
    if (!(f > 0 || (f == 0 && (ey < 0 || (ey == 0 && ex < 0))))) return false;
    ex = cx - bx; ey = cy - by; f = ex * (sy - by) - ey * (sx - bx);
    if (!(f > 0 || (f == 0 && (ey < 0 || (ey == 0 && ex < 0))))) return false;
    ex = ax - cx; ey = ay - cy; f = ex * (sy - cy) - ey * (sx - cx);
    if (!(f > 0 || (f == 0 && (ey < 0 || (ey == 0 && ex < 0))))) return false;
    return true;
}

// Roots of up to four consecutive labels q[0..n): one 16-byte load where
// aligned, the finds interleaved, so that their loads are in flight together
// (one find per pixel is bound by load latency; settling groups of one label
// by one find measured slower, 217 against 194 us for 1024 frames with the
// merge: the warp then runs both ways one after the other; two or four groups of
// four a thread 177 and 282 against 176: fewer warps). Groups in which nothing
// changes are not written, the others by one 16-byte store where aligned (a
// store per label: 184 us).
__device__ __forceinline__ void flatten4(int32_t* L, int32_t* q, int n)
{
    int x[4], p[4], first[4];
    const bool whole = n == 4 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
    if (whole) {
        const int4 v = *reinterpret_cast<const int4*>(q);
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = q[i < n ? i : 0];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        first[i] = x[i];
        p[i] = L[x[i]];
    }
    for (;;) {
        bool more = false;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (p[i] != x[i]) {
                x[i] = p[i];
                p[i] = L[x[i]];
                more = true;
            }
        if (!more) break;
    }
    if (!((first[0] ^ x[0]) | (first[1] ^ x[1]) | (first[2] ^ x[2]) | (first[3] ^ x[3]))) return;
    if (whole) {
        *reinterpret_cast<int4*>(q) = make_int4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i < n && first[i] != x[i]) q[i] = x[i];
    }
}

// flatten4 over a tile of TW x TH labels
template <int TW, int TH>
__device__ __forceinline__ void flatten_tile(int32_t* L, int w, int h, int x0, int y0)
{
    for (int k = threadIdx.x; k < TW / 4 * TH; k += blockDim.x) {
        const int x = x0 + 4 * (k % (TW / 4)), y = y0 + k / (TW / 4);
        if (x < w && y < h) flatten4(L, L + (size_t)y * w + x, min(4, w - x));
    }
}

}  // namespace depix

namespace depix {

// ------------------------------------------------- hull table entries

// hull vertex t of a pattern-table entry, in 1/64 cell
__host__ __device__ __forceinline__ int hx(uint64_t e, int t) { return ((int)((e >> (4 + 6 * t)) & 7u) - 1) * (kUnit / 4); }
__host__ __device__ __forceinline__ int hy(uint64_t e, int t) { return ((int)((e >> (7 + 6 * t)) & 7u) - 1) * (kUnit / 4); }

// edge_link (isLinkedEdge) on a hull entry
__host__ __device__ __forceinline__ int hull_edge_link(uint64_t e, int n, unsigned node, int idx)
{
    int b = idx + 1 == n ? 0 : idx + 1;
    int ax = hx(e, idx), ay = hy(e, idx), bx = hx(e, b), by = hy(e, b);
    int dx = bx - ax, dy = by - ay, my2 = ay + by;
    const int half = kUnit / 2;
    if (ay == by && ay > half && bitof(node, 1)) return 1;
    if (ax == bx && ax > half && bitof(node, 4)) return 4;
    if (ay == by && ay < half && bitof(node, 6)) return 6;
    if (ax == bx && ax < half && bitof(node, 3)) return 3;
    bool s1 = dx != 0 && dy == dx, sm1 = dx != 0 && dy == -dx;
    if (s1 && my2 > kUnit && bitof(node, 0)) return 0;
    if (sm1 && my2 > kUnit && bitof(node, 2)) return 2;
    if (s1 && my2 < kUnit && bitof(node, 7)) return 7;
    if (sm1 && my2 < kUnit && bitof(node, 5)) return 5;
    return -1;
}

// getQ_i / getR_i on a hull entry (index i taken modulo n, as the reference)
__host__ __device__ __forceinline__ void hull_qr(uint64_t e, int n, int i, bool want_r, int& ox, int& oy)
{
    int a = i % n;
    if (a < 0) a += n;
    int b = (i + 1) % n;
    int px = hx(e, a), py = hy(e, a), nx = hx(e, b), ny = hy(e, b);
    int l2 = (nx - px) * (nx - px) + (ny - py) * (ny - py);
    int wp, wn, d;
    if (l2 <= kUnit * kUnit) {
        wp = want_r ? 1 : 3;
        wn = want_r ? 3 : 1;
        d = 4;
    } else {
        wp = want_r ? 1 : 7;
        wn = want_r ? 7 : 1;
        d = 8;
    }
    ox = (wp * px + wn * nx) / d;
    oy = (wp * py + wn * ny) / d;
}

// ------------------------------------------------- TMA tile loads (sm_90+)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Waits for the phase with the given parity to complete, at most max_iter
// polls; false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int max_iter)
{
    for (int i = 0; i < max_iter; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Polls a block allows a TMA tile load before it gives up (about a second on
// GB300 at most; a load completes in microseconds).
constexpr int kTmaPolls = 1 << 22;

// Waits for the tile load completing on bar. When the wait gives up, it sets
// the stage's sticky fault flag and then waits again, bounded the same way,
// for the load it issued, so that a load still in flight does not land in
// shared memory after the block has left; the block then leaves its tile
// unwritten. False when the first wait gave up.
__device__ __forceinline__ bool tma_wait_or_flag(uint64_t* bar, int* fault, int polls = kTmaPolls)
{
    if (mbar_wait_bounded(bar, 0, polls)) return true;
    atomicExch(fault, 1);
    mbar_wait_bounded(bar, 0, polls);
    return false;
}

// One 3-D tile of a tensor map into shared memory, completing on bar. The
// innermost coordinate times the element size must be a multiple of 16
// bytes (the caller guarantees it); out-of-range elements read as zero.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

}  // namespace depix

namespace depix {

// A kernel launched by launch_early may start while the one before it on the
// stream still runs: it waits for its end, with all that it wrote, before its
// first access to memory (buffers that the one before may have written are then
// read with plain loads, not through the non-coherent path), and only then lets
// the next one start, so that no more than two kernels of a stream overlap.
__device__ __forceinline__ void early_start() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_for_last() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void follow_last()
{
    wait_for_last();
    early_start();
}

// Persistent work loop: the block pulls `gran` tile indices at a time from
// *counter until `total` is reached and runs body(t) on each; a barrier
// separates tiles (the bodies reuse shared memory). No block waits on
// another: a block stops when the counter passes the end.
template <typename Body>
__device__ __forceinline__ void queue_loop(int* counter, int total, int gran, Body body)
{
    __shared__ int s_first;
    for (;;) {
        if (threadIdx.x == 0) s_first = atomicAdd(counter, gran);
        __syncthreads();
        const int t0 = s_first;
        __syncthreads();
        if (t0 >= total) break;
        const int t1 = min(t0 + gran, total);
        for (int t = t0; t < t1; t++) {
            body(t);
            __syncthreads();
        }
    }
}

// The same with each warp pulling its own tiles (bodies that need no
// barrier: one warp per tile).
template <typename Body>
__device__ __forceinline__ void warp_queue_loop(int* counter, int total, int gran, Body body)
{
    const int lane = threadIdx.x & 31;
    for (;;) {
        int t0 = 0;
        if (lane == 0) t0 = atomicAdd(counter, gran);
        t0 = __shfl_sync(0xFFFFFFFFu, t0, 0);
        if (t0 >= total) break;
        const int t1 = min(t0 + gran, total);
        for (int t = t0; t < t1; t++) body(t);
    }
}

// the frame f with base[f] <= t < base[f + 1]
__device__ __forceinline__ int queue_frame(const uint32_t* base, int n, uint32_t t)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

}  // namespace depix
