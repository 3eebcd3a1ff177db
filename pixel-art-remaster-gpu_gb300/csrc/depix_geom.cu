// depix_geom.cu -- reshaped cells, subdivision, triangulation, VBO output
// and the headless rasterizer.
//
// A cell's hull depends only on 12 bits of the resolved graph (its node byte
// and two bits of each row neighbour), so the hull and its ear clip are
// computed once per device for all 4096 patterns by k_init_tables and looked
// up afterwards. Corner cutting and the ear clip of the cut polygon depend on
// neighbours and on the image, and are computed per cell.
#include <array>
#include <cstring>
#include <map>
#include <memory>
#include <new>
#include <type_traits>
#include <vector>

#include "depix_internal.h"

namespace depix {

__device__ uint64_t g_hull_lut[4096];
__device__ uint64_t g_tri_lut[4096];

// ---- cut polygons by pieces
//
// One corner-cutting round changes a hull edge by edge, so the boundary of a
// cut polygon is made of pieces (subdivision, subdivision_functions.cu:564-669):
//  - what the cell's own pattern decides: border edges from Q_v to R_v+1, cut
//    corners R_v -> Q_v, linked edges between two linked ones;
//  - per linked edge with a border edge at one end or both: the path over the
//    midpoint(s) with the linked neighbour's R or Q, which the edge's geometry
//    and the neighbour's pattern decide;
//  - per corner that the T-junction test keeps: the triangle R, P, Q.
// Coverage by crossing number is the XOR of the pieces' coverages, so a cut
// cell's mask is a few table entries XORed (k_build_scale_masks), with no
// polygon built. Over all 4096 patterns there are 16 geometries of such
// linked edges, at most 4 of them in a pattern, 7924 pairs of an edge's own
// cut ends and a neighbour's points, and 68 corner triangles.
constexpr int kGeoms = 16, kMaxPaths = 8192, kMaxCorners = 128;
struct CutPath { // an open path of n points in 1/64 cell
    int8_t n, x[4], y[4];
};
struct CutCorner { // hull vertex P between two border edges, R before and Q after it
    int8_t px, py, rx, ry, qx, qy;
};
struct CutTables {
    // per pattern its linked edges with a border edge beside them: first path
    // of the edge's own class (bits 0-15), geometry (16-19), link (20-22),
    // present (23)
    uint4 edges[4096];
    uint64_t verts[4096];   // per hull vertex between border edges (byte v): its corner class, else 0xFF
    uint32_t corners[4096]; // the same for the vertices at the cell's corners (0,0), (1,0), (1,1), (0,1)
    uint8_t nb_class[kGeoms * 4096]; // per geometry and neighbour pattern: the neighbour's class
    CutPath paths[kMaxPaths];        // [own class first path + neighbour's class]
    CutCorner tris[kMaxCorners];
};
__device__ __align__(16) CutTables g_cut;

// ------------------------------------------------------ pattern tables

struct QP {
    int x, y; // quarter units
};

// Cell points in emission order, directions 0,1,2,4,7,6,5,3
// (createCellFromPattern, diagram_functions.cu:320-520). The misses of bits 4
// and 6 emit (0.75,0.75) and (0.25,0.75) as the reference does.
__device__ int cell_points(unsigned nd, unsigned left, unsigned right, QP* p)
{
    int n = 0;
    auto put = [&](int x, int y) { p[n].x = x; p[n].y = y; n++; };
    // corner direction d between sides a (first) and b (second): both sides
    // present -> two points; one side -> the point on the other side's axis
    if (bitof(nd, 0)) {
        if (bitof(nd, 1) && !bitof(nd, 3)) put(-1, 3);
        else if (bitof(nd, 3) && !bitof(nd, 1)) put(1, 5);
        else { put(-1, 3); put(1, 5); }
    } else if (bitof(left, 2)) put(1, 3);
    else put(0, 4);
    if (bitof(nd, 1)) { put(0, 4); put(4, 4); }
    else put(2, 3);
    if (bitof(nd, 2)) {
        if (bitof(nd, 1) && !bitof(nd, 4)) put(5, 3);
        else if (bitof(nd, 4) && !bitof(nd, 1)) put(3, 5);
        else { put(3, 5); put(5, 3); }
    } else if (bitof(right, 0)) put(3, 3);
    else put(4, 4);
    if (bitof(nd, 4)) { put(4, 4); put(4, 0); }
    else put(3, 3);
    if (bitof(nd, 7)) {
        if (bitof(nd, 4) && !bitof(nd, 6)) put(3, -1);
        else if (bitof(nd, 6) && !bitof(nd, 4)) put(5, 1);
        else { put(5, 1); put(3, -1); }
    } else if (bitof(right, 5)) put(3, 1);
    else put(4, 0);
    if (bitof(nd, 6)) { put(4, 0); put(0, 0); }
    else put(1, 3);
    if (bitof(nd, 5)) {
        if (bitof(nd, 3) && !bitof(nd, 6)) put(1, -1);
        else if (bitof(nd, 6) && !bitof(nd, 3)) put(-1, 1);
        else { put(1, -1); put(-1, 1); }
    } else if (bitof(left, 7)) put(1, 1);
    else put(0, 0);
    if (bitof(nd, 3)) { put(0, 0); put(0, 4); }
    else put(1, 2);
    return n;
}

__device__ __forceinline__ void qswap(QP& a, QP& b)
{
    QP t = a;
    a = b;
    b = t;
}

// The reference's point ordering (sort + sort_y, diagram_functions.cu:37-129):
// gather all points with the smallest remaining x to the front, then bring
// the smallest y of that group to its front. Ties beyond two points stay in
// scan order, as in the reference.
__device__ void lex_order(QP* P, int n)
{
    int done = 0;
    while (done < n) {
        int lo = 1 << 20, tie = 0, idx[kMaxPoly];
        for (int i = done; i < n; i++) {
            if (P[i].x < lo) { lo = P[i].x; tie = 0; idx[0] = i; }
            else if (P[i].x == lo) idx[++tie] = i;
        }
        for (int t = 0; t <= tie; t++) qswap(P[done + t], P[idx[t]]);
        if (tie > 0) {
            int ly = 1 << 20, yt = 0, yidx[kMaxPoly];
            for (int i = done; i <= done + tie; i++) {
                if (P[i].y < ly) { ly = P[i].y; yt = 0; yidx[0] = i; }
                else if (P[i].y == ly) yidx[++yt] = i;
            }
            for (int t = 0; t <= yt; t++) qswap(P[done + t], P[yidx[t]]);
        }
        done += tie + 1;
    }
}

__device__ __forceinline__ int qcross(QP o, QP a, QP b) { return (a.x - o.x) * (b.y - o.y) - (a.y - o.y) * (b.x - o.x); }

// Monotone chain (convex_hull, diagram_functions.cu:239-316); returns the
// vertex count, H[0..count-1] counter-clockwise from the first sorted point.
__device__ int monotone_hull(QP* P, int n, QP* H)
{
    lex_order(P, n);
    int k = 0;
    for (int i = 0; i < n; i++) {
        while (k >= 2 && qcross(H[k - 2], H[k - 1], P[i]) <= 0) k--;
        H[k++] = P[i];
    }
    for (int i = n - 2, t = k + 1; i >= 0; i--) {
        while (k >= t && qcross(H[k - 2], H[k - 1], P[i]) <= 0) k--;
        H[k++] = P[i];
    }
    return k - 1;
}

__global__ void k_init_tables()
{
    int pat = blockIdx.x * blockDim.x + threadIdx.x;
    if (pat >= 4096) return;
    unsigned node = pat & 0xFF;
    unsigned left = ((unsigned)bitof(pat, 8) << 2) | ((unsigned)bitof(pat, 9) << 7);
    unsigned right = (unsigned)bitof(pat, 10) | ((unsigned)bitof(pat, 11) << 5);
    QP P[kMaxPoly], H[2 * kMaxPoly];
    int np = cell_points(node, left, right, P);
    int k = monotone_hull(P, np, H);
    uint64_t e = (uint64_t)k;
    for (int t = 0; t < k && t < kMaxHull; t++)
        e |= (uint64_t)((H[t].x + 1) | ((H[t].y + 1) << 3)) << (4 + 6 * t);
    g_hull_lut[pat] = e;
    Poly c;
    hull_from_lut(e, c);
    uint8_t tri[3 * kMaxPoly];
    bool ok;
    int nt = ear_clip(c, tri, ok);
    uint64_t te = 0;
    for (int q = 0; q < 3 * nt; q++) te |= (uint64_t)tri[q] << (3 * q);
    g_tri_lut[pat] = te;
}

// The tables of g_cut from the hull table; false when a class count does not
// fit (it cannot: the patterns are fixed).
static bool build_cut_tables(const uint64_t* hull, CutTables& T)
{
    using Key = std::array<int, 9>;
    std::map<std::array<int, 5>, int> geoms; // link, P_v, P_v+1
    std::map<int, std::map<std::array<int, 4>, int>> nb; // per geometry: (Q at P_v, R at P_v+1) -> class
    std::map<Key, int> own;                  // geometry, R_v, Q_v+1 where cut -> first path
    std::map<std::array<int, 6>, int> tris;
    int npaths = 0;
    memset(&T, 0, sizeof(T));
    for (int pat = 0; pat < 4096; pat++) {
        const uint64_t e = hull[pat];
        const int n = (int)(e & 0xF);
        int link[kMaxHull];
        for (int v = 0; v < n; v++) link[v] = hull_edge_link(e, n, (unsigned)pat & 0xFFu, v);
        T.verts[pat] = ~0ull;
        T.corners[pat] = ~0u;
        uint32_t ed[4] = {0, 0, 0, 0};
        int ne = 0;
        for (int v = 0; v < n; v++) {
            const int v1 = v + 1 == n ? 0 : v + 1;
            const bool prev = link[v == 0 ? n - 1 : v - 1] >= 0, cur = link[v] >= 0;
            const int px = hx(e, v), py = hy(e, v), p1x = hx(e, v1), p1y = hy(e, v1);
            int rx, ry, qx, qy;
            hull_qr(e, n, v - 1, true, rx, ry);
            if (!cur && !prev) {
                hull_qr(e, n, v, false, qx, qy);
                const auto it = tris.emplace(std::array<int, 6>{px, py, rx, ry, qx, qy}, (int)tris.size()).first;
                if (it->second >= kMaxCorners) return false;
                T.tris[it->second] = CutCorner{(int8_t)px, (int8_t)py, (int8_t)rx, (int8_t)ry, (int8_t)qx, (int8_t)qy};
                const uint64_t id = (uint64_t)it->second;
                T.verts[pat] = (T.verts[pat] & ~(0xFFull << (8 * v))) | id << (8 * v);
                if ((px == 0 || px == kUnit) && (py == 0 || py == kUnit)) {
                    const int c = py == 0 ? (px == 0 ? 0 : 1) : (px == 0 ? 3 : 2);
                    T.corners[pat] = (T.corners[pat] & ~(0xFFu << (8 * c))) | (uint32_t)id << (8 * c);
                }
            }
            const bool cut0 = !prev, cut1 = link[v1] < 0; // R_v -> M_v, M_v+1 -> Q_v+1
            if (!cur || (!cut0 && !cut1)) continue;
            const int L = link[v];
            hull_qr(e, n, v1, false, qx, qy);
            const int g = geoms.emplace(std::array<int, 5>{L, px, py, p1x, p1y}, (int)geoms.size()).first->second;
            if (g >= kGeoms || ne == 4) return false;
            auto& cls = nb[g];
            if (cls.empty()) {
                for (int np = 0; np < 4096; np++) {
                    const uint64_t he = hull[np];
                    const int hn = (int)(he & 0xF);
                    // the neighbour's vertex at this position, else its vertex 0 (getPointIndex)
                    auto at = [&](int x, int y) {
                        for (int t = 0; t < hn; t++)
                            if (hx(he, t) == x - kUnit * dir_di(L) && hy(he, t) == y - kUnit * dir_dj(L)) return t;
                        return 0;
                    };
                    int ax, ay, bx, by;
                    hull_qr(he, hn, at(px, py), false, ax, ay);
                    hull_qr(he, hn, at(p1x, p1y) - 1, true, bx, by);
                    const int id = cls.emplace(std::array<int, 4>{ax + kUnit * dir_di(L), ay + kUnit * dir_dj(L),
                                                                  bx + kUnit * dir_di(L), by + kUnit * dir_dj(L)},
                                               (int)cls.size()).first->second;
                    if (id > 255) return false;
                    T.nb_class[g * 4096 + np] = (uint8_t)id;
                }
            }
            const Key key{g, cut0, cut0 ? rx : 0, cut0 ? ry : 0, cut1, cut1 ? qx : 0, cut1 ? qy : 0, 0, 0};
            const auto it = own.emplace(key, npaths).first;
            if (it->second == npaths) {
                if (npaths + (int)cls.size() > kMaxPaths) return false;
                for (const auto& c : cls) {
                    CutPath& p = T.paths[npaths + c.second];
                    auto put = [&](int x, int y) {
                        p.x[p.n] = (int8_t)x;
                        p.y[p.n++] = (int8_t)y;
                    };
                    if (cut0) {
                        put(rx, ry);
                        put((rx + c.first[0]) / 2, (ry + c.first[1]) / 2);
                    } else {
                        put(px, py);
                    }
                    if (cut1) {
                        put((qx + c.first[2]) / 2, (qy + c.first[3]) / 2);
                        put(qx, qy);
                    } else {
                        put(p1x, p1y);
                    }
                }
                npaths += (int)cls.size();
            }
            ed[ne++] = (uint32_t)it->second | (uint32_t)g << 16 | (uint32_t)L << 20 | 1u << 23;
        }
        T.edges[pat] = make_uint4(ed[0], ed[1], ed[2], ed[3]);
    }
    return true;
}

cudaError_t init_tables(cudaStream_t s)
try {
    std::vector<uint64_t> hull(4096);
    std::unique_ptr<CutTables> T(new CutTables);
    k_init_tables<<<16, 256, 0, s>>>();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyFromSymbolAsync(hull.data(), g_hull_lut, sizeof(g_hull_lut), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    if (!build_cut_tables(hull.data(), *T)) return cudaErrorUnknown;
    e = cudaMemcpyToSymbolAsync(g_cut, T.get(), sizeof(CutTables), 0, cudaMemcpyHostToDevice, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
} catch (const std::bad_alloc&) {
    return cudaErrorMemoryAllocation;
}

cudaError_t hull_table_address(const uint64_t** out)
{
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_hull_lut);
    *out = static_cast<const uint64_t*>(p);
    return e;
}

cudaError_t copy_tables(uint64_t* hull, uint64_t* tri)
{
    cudaError_t e = cudaMemcpyFromSymbol(hull, g_hull_lut, sizeof(g_hull_lut));
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(tri, g_tri_lut, sizeof(g_tri_lut));
    return e;
}

// ------------------------------------------- 45-slot stage entry points

__device__ __forceinline__ unsigned linear_at(const uint8_t* g, int n, int idx)
{
    return (idx < 0 || idx >= n) ? 0u : (unsigned)g[idx];
}

// cells_Kernel (kernel.cu:192-213): row neighbours read linearly
__global__ void k_cells(const uint8_t* g, int w, int h, float2* diagram, int* ec)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x, n = w * h;
    if (idx >= n) return;
    int pat = cell_pattern(g[idx], linear_at(g, n, idx - 1), linear_at(g, n, idx + 1));
    Poly c;
    hull_from_lut(__ldg(&g_hull_lut[pat]), c);
    float2* cell = diagram + (size_t)idx * kCell;
    const float inv = 1.0f / kUnit;
    for (int t = 0; t < kCell; t++) {
        float2 v = make_float2(0.f, 0.f);
        if (t <= c.n) {
            int q = t < c.n ? t : 0;
            v = make_float2((float)c.x[q] * inv, (float)c.y[q] * inv);
        }
        cell[t] = v;
    }
    ec[idx] = c.n;
}

__device__ __forceinline__ bool poly_from_slots(const float2* cell, int n, int cap, Poly& p)
{
    if (n < 3 || n > cap) return false;
    p.n = n;
    for (int t = 0; t < n; t++) {
        float2 v = cell[t];
        p.x[t] = (int8_t)__float2int_rn(v.x * (float)kUnit);
        p.y[t] = (int8_t)__float2int_rn(v.y * (float)kUnit);
    }
    return true;
}

// subdivision_Kernel (kernel.cu:216-261): reads the snapshot, skips byte 90
__global__ void k_subdivide(const uint8_t* img, int w, int h, int ws, int layout, const uint8_t* g,
                            const float2* snap, const int* ec_snap, float2* diagram, int* ec)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= w * h) return;
    unsigned node = g[idx];
    if (node == 90) return;
    int i = idx % w, j = idx / w;
    Poly c, out;
    if (!poly_from_slots(snap + (size_t)idx * kCell, ec_snap[idx], kMaxHull, c)) return;
    auto nb_hull = [&](int link, Poly& p) {
        // linear neighbour index as the reference computes it; a bit that
        // points past either end of the frame finds no cell
        int nb = idx + dir_dj(link) * w + dir_di(link);
        if (nb < 0 || nb >= w * h || !poly_from_slots(snap + (size_t)nb * kCell, ec_snap[nb], kMaxHull, p)) {
            p.n = 1;
            p.x[0] = p.y[0] = 0;
        }
    };
    auto tj = [&](int px, int py) { return t_junction_global(img, w, h, ws, layout, i, j, px, py); };
    subdivide_cell(c, node, nb_hull, tj, out);
    float2* cell = diagram + (size_t)idx * kCell;
    const float inv = 1.0f / kUnit;
    for (int t = 0; t < out.n; t++) cell[t] = make_float2((float)out.x[t] * inv, (float)out.y[t] * inv);
    ec[idx] = out.n;
}

// triangulate_Kernel (kernel.cu:264-282): triangle corners + (i, j) in the
// first 3*count slots; the remaining slots get (-100, -100)
__global__ void k_triangulate(float2* diagram, const int* ec, int w, int h)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= w * h) return;
    int i = idx % w, j = idx / w;
    float2* cell = diagram + (size_t)idx * kCell;
    Poly c;
    int nt = 0;
    uint8_t tri[3 * kMaxPoly];
    if (poly_from_slots(cell, ec[idx], kMaxPoly, c)) {
        bool ok;
        nt = ear_clip(c, tri, ok);
    }
    const float inv = 1.0f / kUnit;
    for (int t = 0; t < kCell; t++) {
        float2 v = make_float2(-100.f, -100.f);
        if (t < 3 * nt) v = make_float2((float)c.x[tri[t]] * inv + (float)i, (float)c.y[tri[t]] * inv + (float)j);
        cell[t] = v;
    }
}

// position_kernel + color_kernel (kernel.cu:67-137)
__global__ void k_emit(const uint8_t* img, int w, int h, int ws, int layout, const float2* diagram, const int* ec,
                       float2* pos, uchar4* col)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= w * h) return;
    int i = idx % w, j = idx / w;
    int lim = (ec[idx] - 2) * 3;
    size_t base = (size_t)idx * kCell;
    if (pos)
        for (int t = 0; t < kCell; t++) pos[base + t] = t < lim ? diagram[base + t] : make_float2(-100.f, -100.f);
    if (col) {
        uint32_t c = load_bgr(img, ws, layout, i, j);
        uchar4 v = make_uchar4((c >> 16) & 0xFF, (c >> 8) & 0xFF, c & 0xFF, 255);
        for (int t = 0; t < kCell; t++) col[base + t] = v;
    }
}

// ------------------------------------------------------ a frame's VBO whole
//
// What the stage kernels above do one after the other over a frame (cells,
// snapshot, subdivision, triangulation, emission), in one pass: a block takes
// kVboCells cells, keeps their polygons and triangles in shared memory and
// writes the three buffers a slot per lane, in order. The stages moved the
// 45-slot buffers seven times, a cell's 360 bytes by one lane, and clipped ears
// with the polygon in local memory: 15 + 8 (snapshot) + 39 + 44 + 31 us of a
// 256x224 frame, where this takes 25 (10 without subdivision, about the 52 MB
// written; the rest is the latency of the longest ear clips).
//
// A cell whose edges are all linked (or with no subdivision every cell) keeps
// its hull, whose triangles are in the table; the others, about one in five, go
// to a list. Eight lanes cut a cell, a hull vertex each (a hull has at most
// eight); then a lane clips its ears, the lanes of a warp side by side (28 us
// with the list dealt out to all warps; 33 us at 32 cells a block, 30 at 128).
constexpr int kVboCells = 64, kVboThreads = 128;

struct VboShared {
    char2 xy[kVboCells][kMaxPoly + 2]; // nine words, for lanes that read a cell each
    uint64_t hull[kVboCells];
    uint8_t tri[kVboCells][3 * kMaxPoly + 4];
    int origin[kVboCells][2];
    uint32_t color[kVboCells];
    uint8_t node[kVboCells], n[kVboCells], nt[kVboCells], list[kVboCells];
    int listed;
};

// hull entry of cell idx, neighbours read linearly; a single point at the
// origin outside the frame
__device__ __forceinline__ uint64_t linear_hull(const uint8_t* g, int n, int idx)
{
    if (idx < 0 || idx >= n) return 1 | 1 << 4 | 1 << 7;
    return __ldg(&g_hull_lut[cell_pattern(g[idx], linear_at(g, n, idx - 1), linear_at(g, n, idx + 1))]);
}

// Q (or R) of the linked neighbour's hull nb around vertex (px, py)
// (get{Q,R}_i_from_linked_cell), in this cell's coordinates
__device__ __forceinline__ int2 hull_linked_qr(uint64_t nb, int link, int px, int py, bool want_r)
{
    const int n = (int)(nb & 15), bx = kUnit * dir_di(link), by = kUnit * dir_dj(link);
    int at = 0;
    for (int t = n - 1; t >= 0; t--)
        if (hx(nb, t) == px - bx && hy(nb, t) == py - by) at = t;
    int2 o;
    hull_qr(nb, n, want_r ? at - 1 : at, want_r, o.x, o.y);
    return make_int2(o.x + bx, o.y + by);
}

// ear_clip on a polygon in shared memory, without the places it tests in vain:
// it clips the first ear after the place it stands at, an ear being a convex
// corner with no other vertex in or on its triangle. Vertices are their places
// in its list, which runs counter-clockwise; corners that are not convex are
// kept in a mask, of which a clip changes two. (Eight lanes a cell that test
// place after place, or that keep the vertices in each corner's triangle, take
// 37 and 36 us for the whole kernel on a 256x224 frame, where a lane a cell
// takes 25: they issue several times as many instructions.)
__device__ __forceinline__ int clip_ears(const char2* xy, int n, uint8_t* tri)
{
    if (n < 3) return 0;
    int area = 0;
    for (int q = 0; q < n; q++) {
        const char2 p = xy[q > 0 ? q - 1 : n - 1], r = xy[q];
        area += p.x * r.y - r.x * p.y;
    }
    const bool turned = area <= 0;
    auto at = [&](int k) { return turned ? n - 1 - k : k; };
    unsigned alive = (1u << n) - 1u;
    auto next = [](unsigned set, int k) { // of a set that is not empty: its first place from k on, around
        const unsigned up = set >> k << k;
        return __ffs(up != 0 ? up : set) - 1;
    };
    auto before = [&](int k) {
        const unsigned down = alive & ((1u << k) - 1u);
        return 31 - __clz(down != 0 ? down : alive);
    };
    auto convex = [](char2 A, char2 B, char2 C) {
        return (B.x - A.x) * (C.y - A.y) - (B.y - A.y) * (C.x - A.x) > 0;
    };
    unsigned corners = 0; // the convex ones
    char2 A = xy[at(n - 1)], B = xy[at(0)];
    for (int q = 0; q < n; q++) {
        const char2 C = xy[at(q + 1 < n ? q + 1 : 0)];
        if (convex(A, B, C)) corners |= 1u << q;
        A = B;
        B = C;
    }
    int nt = 0, from = 0;
    unsigned left = corners; // not tested since the last clip
    for (int nv = n; nv > 2 && left != 0;) {
        const int b = next(left, from), u = before(b), d = next(alive, b + 1);
        const char2 U = xy[at(u)], V = xy[at(b)], D = xy[at(d)];
        bool ear = true;
        for (unsigned o = alive & ~(1u << u | 1u << b | 1u << d); o != 0 && ear; o &= o - 1) {
            const char2 P = xy[at(__ffs(o) - 1)];
            ear = !inside_tri(U.x, U.y, V.x, V.y, D.x, D.y, P.x, P.y);
        }
        if (!ear) {
            left &= ~(1u << b);
            from = b + 1;
            continue;
        }
        tri[3 * nt] = (uint8_t)at(u);
        tri[3 * nt + 1] = (uint8_t)at(b);
        tri[3 * nt + 2] = (uint8_t)at(d);
        nt++;
        nv--;
        alive &= ~(1u << b);
        const int uu = before(u), dd = next(alive, d + 1);
        corners &= ~(1u << u | 1u << b | 1u << d);
        if (convex(xy[at(uu)], U, D)) corners |= 1u << u;
        if (convex(U, D, xy[at(dd)])) corners |= 1u << d;
        left = corners;
        from = dd;
    }
    return nt;
}

__global__ void __launch_bounds__(kVboThreads) k_vbo(const uint8_t* img, int w, int h, int ws, int layout,
                                                     const uint8_t* g, int subdivide, float2* diagram, int* ec,
                                                     float2* pos, uchar4* col)
{
    follow_last();
    __shared__ VboShared S;
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const int frame = w * h, first = blockIdx.x * kVboCells, cells = min(kVboCells, frame - first);
    if (threadIdx.x == 0) S.listed = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < cells; c += kVboThreads) {
        const int idx = first + c, j = idx / w, i = idx - j * w;
        const unsigned node = g[idx];
        const int pat = cell_pattern(node, linear_at(g, frame, idx - 1), linear_at(g, frame, idx + 1));
        const uint64_t e = __ldg(&g_hull_lut[pat]);
        const int n = (int)(e & 15);
        // all edges linked: no vertex between border edges, no linked edge beside one
        const bool whole = __ldg(&g_cut.verts[pat]) == ~0ull && (__ldg(&g_cut.edges[pat].x) >> 23 & 1) == 0;
        if (!subdivide || node == 90 || whole) {
            const uint64_t te = __ldg(&g_tri_lut[pat]);
            int nt = 0;
            for (; nt < n - 2 && ((te >> (9 * nt)) & 511u) != 0; nt++)
#pragma unroll
                for (int k = 0; k < 3; k++) S.tri[c][3 * nt + k] = (uint8_t)((te >> (9 * nt + 3 * k)) & 7u);
            for (int v = 0; v < n; v++) S.xy[c][v] = make_char2((signed char)hx(e, v), (signed char)hy(e, v));
            S.n[c] = (uint8_t)n;
            S.nt[c] = (uint8_t)nt;
        } else {
            S.list[atomicAdd(&S.listed, 1)] = (uint8_t)c;
            S.hull[c] = e;
            S.node[c] = (uint8_t)node;
        }
        S.origin[c][0] = i;
        S.origin[c][1] = j;
        if (col) {
            const uint32_t p = load_bgr(img, ws, layout, i, j);
            S.color[c] = (p >> 16 & 0xFFu) | (p & 0xFF00u) | (p & 0xFFu) << 16 | 0xFF000000u;
        }
    }
    __syncthreads();

    const int lane = threadIdx.x & 31, base = lane & 24, v = lane & 7, listed = S.listed;
    for (int q0 = 4 * (threadIdx.x >> 5); q0 < listed; q0 += kVboThreads / 8) {
        const bool live = q0 + (base >> 3) < listed;
        const int c = S.list[live ? q0 + (base >> 3) : q0], idx = first + c;
        const unsigned node = S.node[c];
        const uint64_t e = live ? S.hull[c] : 0;
        const int n = (int)(e & 15);
        const int link = v < n ? hull_edge_link(e, n, node, v) : -1;
        const int before = __shfl_sync(kAll, link, base + (v > 0 ? v - 1 : max(n - 1, 0)));
        // the vertex stays, or a point on each side of it takes its place
        int x0 = hx(e, v), y0 = hy(e, v), x1 = 0, y1 = 0;
        bool two = false;
        if (v < n && (link < 0 || before < 0)) {
            const int px = x0, py = y0, i = S.origin[c][0], j = S.origin[c][1];
            if (link >= 0 || before >= 0 || !t_junction_global(img, w, h, ws, layout, i, j, px, py)) {
                two = true;
                int2 r, t;
                hull_qr(e, n, v - 1, true, r.x, r.y);
                hull_qr(e, n, v, false, t.x, t.y);
                if (link >= 0 || before >= 0) {
                    const int l = max(link, before);
                    const uint64_t nb = linear_hull(g, frame, idx + dir_dj(l) * w + dir_di(l));
                    const int2 a = hull_linked_qr(nb, l, px, py, before >= 0);
                    if (before >= 0) r = make_int2((t.x + a.x) / 2, (t.y + a.y) / 2);
                    else t = make_int2((r.x + a.x) / 2, (r.y + a.y) / 2);
                }
                x0 = r.x, y0 = r.y, x1 = t.x, y1 = t.y;
            }
        }
        const unsigned twos = __ballot_sync(kAll, two) >> base & 0xFFu;
        const int m = n + __popc(twos), at = v + __popc(twos & ((1u << v) - 1u));
        if (v < n) {
            S.xy[c][at] = make_char2((signed char)x0, (signed char)y0);
            if (two) S.xy[c][at + 1] = make_char2((signed char)x1, (signed char)y1);
        }
        if (live && v == 0) S.n[c] = (uint8_t)m;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < listed; q += kVboThreads) {
        const int c = S.list[q];
        S.nt[c] = (uint8_t)clip_ears(S.xy[c], S.n[c], S.tri[c]);
    }
    __syncthreads();

    for (int c = threadIdx.x; c < cells; c += kVboThreads) ec[first + c] = S.n[c];
    const size_t base_slot = (size_t)first * kCell;
    for (int k = threadIdx.x; k < cells * kCell; k += kVboThreads) {
        const int c = k / kCell, t = k - c * kCell;
        float2 o = make_float2(-100.f, -100.f);
        if (t < 3 * S.nt[c]) {
            const char2 p = S.xy[c][S.tri[c][t]];
            o = make_float2((float)p.x * (1.0f / kUnit) + (float)S.origin[c][0],
                            (float)p.y * (1.0f / kUnit) + (float)S.origin[c][1]);
        }
        diagram[base_slot + k] = o;
        if (pos) pos[base_slot + k] = o;
        if (col) reinterpret_cast<uint32_t*>(col)[base_slot + k] = S.color[c];
    }
}

static dim3 grid1(int n, int b) { return dim3((n + b - 1) / b); }

cudaError_t launch_cells(const uint8_t* g, int w, int h, float* diagram, int* ec, cudaStream_t s)
{
    k_cells<<<grid1(w * h, 128), 128, 0, s>>>(g, w, h, reinterpret_cast<float2*>(diagram), ec);
    return cudaGetLastError();
}

cudaError_t launch_subdivide(const uint8_t* img, int w, int h, int ws, int layout, const uint8_t* g,
                             const float* snap, const int* ec_snap, float* diagram, int* ec, cudaStream_t s)
{
    k_subdivide<<<grid1(w * h, 128), 128, 0, s>>>(img, w, h, ws, layout, g, reinterpret_cast<const float2*>(snap),
                                                   ec_snap, reinterpret_cast<float2*>(diagram), ec);
    return cudaGetLastError();
}

cudaError_t launch_triangulate(float* diagram, const int* ec, int w, int h, cudaStream_t s)
{
    k_triangulate<<<grid1(w * h, 128), 128, 0, s>>>(reinterpret_cast<float2*>(diagram), ec, w, h);
    return cudaGetLastError();
}

cudaError_t launch_emit(const uint8_t* img, int w, int h, int ws, int layout, const float* diagram, const int* ec,
                        float* pos, uint8_t* col, cudaStream_t s)
{
    k_emit<<<grid1(w * h, 128), 128, 0, s>>>(img, w, h, ws, layout, reinterpret_cast<const float2*>(diagram), ec,
                                             reinterpret_cast<float2*>(pos), reinterpret_cast<uchar4*>(col));
    return cudaGetLastError();
}

cudaError_t launch_vbo(const uint8_t* img, int w, int h, int ws, int layout, const uint8_t* g, bool subdivide,
                       float* diagram, int* ec, float* pos, uint8_t* col, cudaStream_t s)
{
    return launch_early(early_stages((long long)w * h), k_vbo, grid1(w * h, kVboCells), kVboThreads, 0, s, img, w, h, ws, layout, g, subdivide ? 1 : 0,
                        reinterpret_cast<float2*>(diagram), ec, reinterpret_cast<float2*>(pos),
                        reinterpret_cast<uchar4*>(col));
}

// ------------------------------------------------------------------ raster
//
// One CTA per tile of kRTW x kRTH cells. Phase A stages the resolved graph
// (halo 3: a ring cell's linked neighbours need their own row neighbours) and
// the pixels (halo 2: corner tests of ring cells) in shared memory. Phase B
// builds the triangles of the tile's cells and of the ring around it (ring
// cells reach 0.25 cell into the tile). Phase C shades every output pixel of
// the tile as a gather: of the 3x3 cells around its sample, the one latest in
// VBO order (highest row, then highest column) whose triangles cover the
// sample gives the colour; rows of 4 pixels go out as one 16-byte store.

constexpr int kRTW = 32, kRTH = 8;
constexpr int kGW = kRTW + 2, kGH = kRTH + 2, kGN = kGW * kGH;
constexpr int kBW = kRTW + 6, kBH = kRTH + 6;
constexpr int kCW = kRTW + 4, kCH = kRTH + 4;
constexpr int kMaxTri = kMaxPoly - 2;

struct RasterShared {
    uint8_t graph[kBH][kBW];
    uint32_t pix[kCH][kCW];
    int8_t vx[kGN][kMaxPoly];
    int8_t vy[kGN][kMaxPoly];
    uint8_t tri[kGN][3 * kMaxTri];
    uint8_t nt[kGN];
    int8_t bb[kGN][4];
};


template <int LAYOUT>
__device__ void raster_tile(RasterShared& S, const uint8_t* img, int ws, const uint8_t* g, uint8_t* out, int w,
                            int h, int scale, bool subdivide, int x0, int y0)
{
    // ---- phase A
    for (int k = threadIdx.x; k < kBW * kBH; k += blockDim.x) {
        int gx = x0 - 3 + k % kBW, gy = y0 - 3 + k / kBW;
        unsigned v = 0;
        if (gx >= 0 && gy >= 0 && gx < w && gy < h) v = __ldg(g + (size_t)gy * w + gx) & inside_mask(gx, gy, w, h);
        S.graph[k / kBW][k % kBW] = (uint8_t)v;
    }
    for (int k = threadIdx.x; k < kCW * kCH; k += blockDim.x) {
        int gx = x0 - 2 + k % kCW, gy = y0 - 2 + k / kCW;
        uint32_t v = 0;
        if (gx >= 0 && gy >= 0 && gx < w && gy < h) v = load_bgr(img, ws, LAYOUT, gx, gy);
        S.pix[k / kCW][k % kCW] = v;
    }
    __syncthreads();

    // ---- phase B
    for (int k = threadIdx.x; k < kGN; k += blockDim.x) {
        int lx = k % kGW, ly = k / kGW;
        int ci = x0 - 1 + lx, cj = y0 - 1 + ly;
        if (ci < 0 || cj < 0 || ci >= w || cj >= h) {
            S.nt[k] = 0;
            continue;
        }
        const int bx = lx + 2, by = ly + 2;
        unsigned node = S.graph[by][bx];
        int pat = cell_pattern(node, S.graph[by][bx - 1], S.graph[by][bx + 1]);
        Poly c;
        hull_from_lut(__ldg(&g_hull_lut[pat]), c);
        int nt;
        if (subdivide && node != 90) {
            auto nb_hull = [&](int link, Poly& p) {
                int nx = bx + dir_di(link), ny = by + dir_dj(link);
                int np = cell_pattern(S.graph[ny][nx], S.graph[ny][nx - 1], S.graph[ny][nx + 1]);
                hull_from_lut(__ldg(&g_hull_lut[np]), p);
            };
            auto tj = [&](int px, int py) -> bool {
                long long st = LAYOUT == DEPIX_LAYOUT_BGR ? ws : ((3 * w + 3) & ~3);
                long long index = (long long)cj * st + (long long)ci * 3;
                if ((index - st - 1) < 0 || (index + w + 1) > ((long long)h * st - 1)) return true;
                if (ci == 0 || ci == w - 1 || cj >= h - 1)
                    return t_junction_global(img, w, h, ws, LAYOUT, ci, cj, px, py);
                const int qx = lx + 1, qy = ly + 1; // this pixel in S.pix
                auto C = [&](int dx, int dy) { return S.pix[qy + dy][qx + dx]; };
                if (px == 0 && py == 0) return C(-1, 0) != C(-1, -1) || C(-1, -1) != C(0, -1);
                if (px == kUnit && py == 0) return C(1, 0) != C(1, -1) || C(1, -1) != C(0, -1);
                if (px == kUnit && py == kUnit) return C(0, 1) != C(1, 1) || C(1, 1) != C(1, 0);
                if (px == 0 && py == kUnit) return C(-1, 1) != C(0, 1) || C(0, 1) != C(-1, 0);
                return false;
            };
            Poly sp;
            subdivide_cell(c, node, nb_hull, tj, sp);
            bool ok;
            nt = ear_clip(sp, S.tri[k], ok);
            c = sp;
        } else {
            uint64_t te = __ldg(&g_tri_lut[pat]);
            nt = c.n - 2;
            for (int q = 0; q < 3 * nt; q++) S.tri[k][q] = (uint8_t)((te >> (3 * q)) & 7u);
        }
        int mnx = 127, mny = 127, mxx = -128, mxy = -128;
        for (int t = 0; t < c.n; t++) {
            S.vx[k][t] = c.x[t];
            S.vy[k][t] = c.y[t];
            mnx = min(mnx, c.x[t]); mxx = max(mxx, c.x[t]);
            mny = min(mny, c.y[t]); mxy = max(mxy, c.y[t]);
        }
        S.nt[k] = (uint8_t)nt;
        S.bb[k][0] = (int8_t)mnx; S.bb[k][1] = (int8_t)mny;
        S.bb[k][2] = (int8_t)mxx; S.bb[k][3] = (int8_t)mxy;
    }
    __syncthreads();

    // ---- phase C
    const int s = scale, u = 4 * s;
    const int ow = w * s, oh = h * s;
    const int OW = kRTW * s, OH = kRTH * s;
    const int X0 = x0 * s, Y0 = y0 * s;
    const bool vec = (ow % 4) == 0 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
    for (int q = threadIdx.x; q < (OW / 4) * OH; q += blockDim.x) {
        int r = q / (OW / 4), c4 = 4 * (q % (OW / 4));
        int Y = Y0 + r;
        if (Y >= oh) continue;
        int cj = Y / s;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            int X = X0 + c4 + e;
            uint32_t color = 0xFF000000u;
            if (X < ow) {
                int ci = X / s;
                int SX = 256 * X + 128, SY = 256 * Y + 128;
                bool hit = false;
                for (int dj = 1; dj >= -1 && !hit; dj--)
                    for (int di = 1; di >= -1 && !hit; di--) {
                        int lx = ci + di - (x0 - 1), ly = cj + dj - (y0 - 1);
                        int k = ly * kGW + lx;
                        int nt = S.nt[k];
                        if (nt == 0) continue;
                        int rx = SX - (ci + di) * 256 * s, ry = SY - (cj + dj) * 256 * s;
                        if (rx < S.bb[k][0] * u || rx > S.bb[k][2] * u || ry < S.bb[k][1] * u || ry > S.bb[k][3] * u)
                            continue;
                        for (int t = 0; t < nt; t++) {
                            int a = S.tri[k][3 * t], b = S.tri[k][3 * t + 1], cc = S.tri[k][3 * t + 2];
                            if (covers(S.vx[k][a] * u, S.vy[k][a] * u, S.vx[k][b] * u, S.vy[k][b] * u,
                                       S.vx[k][cc] * u, S.vy[k][cc] * u, rx, ry)) {
                                uint32_t p = S.pix[ly + 1][lx + 1]; // ring cell -> pixel tile
                                color = ((p >> 16) & 0xFFu) | (p & 0xFF00u) | ((p & 0xFFu) << 16) | 0xFF000000u;
                                hit = true;
                                break;
                            }
                        }
                    }
            }
            v[e] = color;
        }
        size_t o = ((size_t)Y * ow + (size_t)(X0 + c4)) * 4;
        if (vec && X0 + c4 + 3 < ow) {
            __stcs(reinterpret_cast<uint4*>(out + o), make_uint4(v[0], v[1], v[2], v[3]));
        } else {
            for (int e = 0; e < 4; e++)
                if (X0 + c4 + e < ow) reinterpret_cast<uint32_t*>(out + o)[e] = v[e];
        }
    }
}

template <int LAYOUT>
__global__ void __launch_bounds__(256) k_raster(RasterBatch b)
{
    __shared__ RasterShared S;
    size_t z = blockIdx.z;
    raster_tile<LAYOUT>(S, b.img + b.img_stride * z, b.ws, b.graph + b.graph_stride * z, b.out + b.out_stride * z,
                        b.w, b.h, b.scale, b.subdivide != 0, blockIdx.x * kRTW, blockIdx.y * kRTH);
}

cudaError_t launch_raster(const RasterBatch& b, int nframes, cudaStream_t s)
{
    dim3 grid((b.w + kRTW - 1) / kRTW, (b.h + kRTH - 1) / kRTH, nframes);
    if (b.layout == DEPIX_LAYOUT_RGBA)
        k_raster<DEPIX_LAYOUT_RGBA><<<grid, 256, 0, s>>>(b);
    else
        k_raster<DEPIX_LAYOUT_BGR><<<grid, 256, 0, s>>>(b);
    return cudaGetLastError();
}


// ------------------------------------------------------------ mask raster
//
// The gather above tests triangles per output pixel. This raster instead
// reduces every cell to a coverage bitmask over the samples its polygon can
// reach and resolves each output block with bit operations:
//
//  - a cell polygon lies inside [-0.75, 1.75]^2 of its own cell: hull points
//    lie in [-0.25, 1.25], subdivision adds midpoints of an own point and a
//    neighbour's point (neighbour hull shifted by one cell);
//  - footprint: output samples (X+0.5)/s in that box, offsets m = X - i*s in
//    [mlo, mlo + F), F <= 30 for s <= 12;
//  - plain cells take their mask from a per-scale table over the 4096 hull
//    patterns, subdivided cells XOR theirs from table entries (CutTables);
//  - an output block (the s x s samples of one cell) takes, per sample, the
//    latest covering cell in VBO order among the 3x3 cells around it.
//
// Mask layouts (mask_layout): up to scale 4 and at 8 a mask is nine parts, one
// per cell of the 3x3 around it (the cell itself is part 4), each part the s*s
// samples of that cell in s rows of s bits, so that a block reads one part of
// each of its nine candidates and resolves all its samples (at 8 two rows of
// them) at once. A part is 16 bits up to scale 4, 64 bits at 8. At 5 to 7 and
// above 8 a mask is one word per footprint row and a word on the parts that it
// touches: parts would need up to 144 bits each, twice the shared memory of the
// rows, and at 5 to 7 a block's rows of 5 to 7 pixels do not make whole 16-byte
// stores, where the rows of 32 blocks do.
//
// What bounds it: a 32x32 tile's phases (tile load, plain cells, cut cells,
// fills, shared blocks) take 22, 22, 28, 20 and 8 % of a block's time, each a
// short chain of shared-memory accesses; cut cells wait on table loads. 1024
// frames of 256x224 at x4: 2605 us when a cell per distinct neighbourhood
// built its polygon from dependent table lookups and masked it by crossing
// number (hash tables found the distinct ones), 885 us now (4.6 TB/s of
// input and output, 0.67 of the measured copy rate; 968 with the labels' roots).
// 16 frames of 640x480 at x8: 597 us before, 289 us now (4.4 TB/s).

struct MaskGeom {
    int s;
    int mlo, F; // footprint of any cell polygon
};

__host__ __device__ __forceinline__ MaskGeom mask_geom(int s)
{
    MaskGeom g;
    g.s = s;
    g.mlo = -((3 * s + 2) / 4);
    g.F = (7 * s - 2) / 4 - g.mlo + 1;
    return g;
}

enum MaskLayout { ML_U16, ML_U64, ML_ROWS };
__host__ __device__ constexpr MaskLayout mask_layout(int s) { return s <= 4 ? ML_U16 : (s == 8 ? ML_U64 : ML_ROWS); }
// words of a mask, of a table entry (mask, then 16 flag bits: above part 8
// for ML_U16, in a word of their own else) and between masks in shared memory
// (odd, so that a warp's cells fall into different banks)
__host__ __device__ __forceinline__ int mask_words(int s)
{
    return s <= 4 ? 5 : (s == 8 ? 18 : mask_geom(s).F);
}
__host__ __device__ __forceinline__ int entry_words(int s) { return s <= 4 ? 8 : (s == 8 ? 20 : ((mask_geom(s).F + 4) & ~3)); }
__host__ __device__ __forceinline__ int mask_stride(int s) { return mask_words(s) | 1; }

// a scale's table: plain hulls, cut cells' own pieces (per pattern), paths
// over a linked neighbour, corner triangles
constexpr int kPlainEntry = 0, kCutEntry = 4096, kPathEntry = 8192, kCornerEntry = kPathEntry + kMaxPaths;
constexpr int kScaleEntries = kCornerEntry + kMaxCorners;
size_t scale_mask_words(int s) { return (size_t)kScaleEntries * entry_words(s); }

// Sets the footprint samples (offsets mlo.. in both axes, F of them) that the
// triangle covers under the top-left rule. Vertices in 1/256 output pixel
// relative to the cell origin.
__device__ __forceinline__ void tri_mask(int ax, int ay, int bx, int by, int cx, int cy, int mlo, int F, uint32_t* rows)
{
    int area = (bx - ax) * (cy - ay) - (by - ay) * (cx - ax);
    if (area == 0) return;
    if (area < 0) {
        int tx = bx, ty = by;
        bx = cx; by = cy; cx = tx; cy = ty;
    }
    // E(p) = A px + B py + C; covered iff E >= bias on all three edges, where
    // bias 0 on a top or left edge (dy < 0, or dy == 0 and dx < 0 with
    // dx = B, dy = -A) and 1 elsewhere: E > 0, or E == 0 on a top/left edge
    const int A0 = ay - by, B0 = bx - ax, C0 = -(A0 * ax + B0 * ay);
    const int A1 = by - cy, B1 = cx - bx, C1 = -(A1 * bx + B1 * by);
    const int A2 = cy - ay, B2 = ax - cx, C2 = -(A2 * cx + B2 * cy);
    const int b0 = (A0 > 0 || (A0 == 0 && B0 < 0)) ? 0 : 1;
    const int b1 = (A1 > 0 || (A1 == 0 && B1 < 0)) ? 0 : 1;
    const int b2 = (A2 > 0 || (A2 == 0 && B2 < 0)) ? 0 : 1;
    const int minx = min(ax, min(bx, cx)), maxx = max(ax, max(bx, cx));
    const int miny = min(ay, min(by, cy)), maxy = max(ay, max(by, cy));
    // sample offsets whose position 256 m + 128 lies inside the bounding box
    // (>> on a signed int is a floor division by 256)
    const int m0 = max(mlo, -((128 - minx) >> 8)), m1 = min(mlo + F - 1, (maxx - 128) >> 8);
    const int n0 = max(mlo, -((128 - miny) >> 8)), n1 = min(mlo + F - 1, (maxy - 128) >> 8);
    for (int n = n0; n <= n1; n++) {
        int py = 256 * n + 128;
        int e0 = B0 * py + C0, e1 = B1 * py + C1, e2 = B2 * py + C2;
        uint32_t bits = 0;
        for (int m = m0; m <= m1; m++) {
            int px = 256 * m + 128;
            if (A0 * px + e0 >= b0 && A1 * px + e1 >= b1 && A2 * px + e2 >= b2) bits |= 1u << (m - mlo);
        }
        if (bits) rows[n - mlo] |= bits;
    }
}

// Crossing-number coverage of one directed edge (1/64 cell): on every sample
// row it crosses, the samples left of the crossing toggle. The sample point
// is shifted by (+e, -e^2), so that the XOR over a simple polygon's edges is
// what the top-left rule gives for any exact triangulation of it.
__device__ void edge_mask(int x0, int y0, int x1, int y1, const MaskGeom& G, uint32_t* rows)
{
    const int u = 4 * G.s;
    int lx = x0 * u, ly = y0 * u, hxx = x1 * u, hyy = y1 * u;
    if (ly == hyy) return;
    if (ly > hyy) {
        int t = lx; lx = hxx; hxx = t;
        t = ly; ly = hyy; hyy = t;
    }
    // rows whose sample height py = 256 row + 128 has ly < py <= hyy
    const int r0 = max(((ly - 128) >> 8) + 1, G.mlo), r1 = min((hyy - 128) >> 8, G.mlo + G.F - 1);
    const int D = hyy - ly, den = 256 * D;
    for (int row = r0; row <= r1; row++) {
        // samples left of the crossing: 256 m + 128 < x_cross  <=>  m < num / den
        const int num = lx * D + (256 * row + 128 - ly) * (hxx - lx) - 128 * D;
        int q = num / den;
        if (num % den > 0) q++; // ceil; the division truncates toward zero
        const int k = q - G.mlo;
        rows[row - G.mlo] ^= k <= 0 ? 0u : (k >= 32 ? 0xFFFFFFFFu : ((1u << k) - 1u));
    }
}

// An edge's part in the test that the polygon is star-shaped about the cell
// centre (every edge turns strictly counter-clockwise around it and the
// polygon winds around it once; it is then simple, the reference's ear clip
// never gives up on it and tiles it exactly): 64 when the edge does not turn
// counter-clockwise, 1 when it passes angle 0. Sums to 1 over the edges of a
// star-shaped polygon.
__device__ __forceinline__ int edge_flags(int x0, int y0, int x1, int y1)
{
    const int ax = x0 - kUnit / 2, ay = y0 - kUnit / 2, bx = x1 - kUnit / 2, by = y1 - kUnit / 2;
    const bool up0 = ay > 0 || (ay == 0 && ax > 0), up1 = by > 0 || (by == 0 && bx > 0);
    return (ax * by - ay * bx > 0 ? 0 : 64) + (!up0 && up1 ? 1 : 0);
}

// footprint rows to a mask in the scale's layout
__device__ __forceinline__ void pack_mask(const MaskGeom& G, const uint32_t* rows, uint32_t* dst)
{
    const int s = G.s;
    if (mask_layout(s) == ML_ROWS) {
        for (int r = 0; r < G.F; r++) dst[r] = rows[r];
        return;
    }
    const uint32_t blockbits = (1u << s) - 1u;
    uint64_t part[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int rr = 0; rr < G.F; rr++) {
        const int m = rr + G.mlo, dj = m < 0 ? -1 : (m >= s ? 1 : 0);
        const uint64_t x = (uint64_t)rows[rr] << (s + G.mlo);
        for (int di = -1; di <= 1; di++)
            part[(dj + 1) * 3 + di + 1] |= ((x >> ((di + 1) * s)) & blockbits) << ((m - dj * s) * s);
    }
    if (mask_layout(s) == ML_U16) {
        for (int p = 0; p < 4; p++) dst[p] = (uint32_t)part[2 * p] | (uint32_t)part[2 * p + 1] << 16;
        dst[4] = (uint32_t)part[8];
    } else {
        for (int p = 0; p < 9; p++) {
            dst[2 * p] = (uint32_t)part[p];
            dst[2 * p + 1] = (uint32_t)(part[p] >> 32);
        }
    }
}

__global__ void k_build_scale_masks(int s, uint32_t* lut)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= kScaleEntries) return;
    const MaskGeom G = mask_geom(s);
    uint32_t rows[32];
    for (int r = 0; r < 32; r++) rows[r] = 0;
    int flags = 0;
    auto edge = [&](int x0, int y0, int x1, int y1) {
        edge_mask(x0, y0, x1, y1, G, rows);
        flags += edge_flags(x0, y0, x1, y1);
    };
    if (id < kCutEntry) {
        Poly c;
        hull_from_lut(g_hull_lut[id], c);
        const uint64_t te = g_tri_lut[id];
        const int u = 4 * s;
        for (int t = 0; t < c.n - 2; t++) {
            int a = (int)((te >> (9 * t)) & 7), b = (int)((te >> (9 * t + 3)) & 7), d = (int)((te >> (9 * t + 6)) & 7);
            tri_mask(c.x[a] * u, c.y[a] * u, c.x[b] * u, c.y[b] * u, c.x[d] * u, c.y[d] * u, G.mlo, G.F, rows);
        }
    } else if (id < kPathEntry) {
        const int pat = id - kCutEntry;
        const uint64_t e = g_hull_lut[pat];
        const int n = (int)(e & 0xF);
        for (int v = 0; v < n; v++) {
            const int v1 = v + 1 == n ? 0 : v + 1;
            const bool prev = hull_edge_link(e, n, (unsigned)pat & 0xFFu, v == 0 ? n - 1 : v - 1) >= 0;
            const bool cur = hull_edge_link(e, n, (unsigned)pat & 0xFFu, v) >= 0;
            const bool next = hull_edge_link(e, n, (unsigned)pat & 0xFFu, v1) >= 0;
            int qx, qy, rx, ry, r1x, r1y;
            hull_qr(e, n, v, false, qx, qy);
            hull_qr(e, n, v - 1, true, rx, ry);
            hull_qr(e, n, v, true, r1x, r1y); // R before vertex v + 1
            if (!cur && !prev) edge(rx, ry, qx, qy);
            if (!cur) edge(qx, qy, r1x, r1y);
            else if (prev && next) edge(hx(e, v), hy(e, v), hx(e, v1), hy(e, v1));
        }
    } else if (id < kCornerEntry) {
        const CutPath& p = g_cut.paths[id - kPathEntry];
        for (int k = 0; k + 1 < p.n; k++) edge(p.x[k], p.y[k], p.x[k + 1], p.y[k + 1]);
    } else {
        // a kept corner: R -> P -> Q in place of R -> Q
        const CutCorner& t = g_cut.tris[id - kCornerEntry];
        edge(t.rx, t.ry, t.px, t.py);
        edge(t.px, t.py, t.qx, t.qy);
        edge_mask(t.rx, t.ry, t.qx, t.qy, G, rows);
        flags -= edge_flags(t.rx, t.ry, t.qx, t.qy);
    }
    for (int r = 0; r < G.F; r++) rows[r] &= (1u << G.F) - 1u; // F <= 30
    uint32_t* dst = lut + (size_t)id * entry_words(s);
    for (int k = 0; k < entry_words(s); k++) dst[k] = 0;
    pack_mask(G, rows, dst);
    const uint32_t f = (uint32_t)flags & 0xFFFFu;
    if (mask_layout(s) == ML_U16) dst[4] |= f << 16;
    else dst[mask_words(s)] = f;
}

cudaError_t build_scale_masks(int s, uint32_t* lut, cudaStream_t st)
{
    k_build_scale_masks<<<(kScaleEntries + 127) / 128, 128, 0, st>>>(s, lut);
    return cudaGetLastError();
}

// set when a bounded wait for a TMA tile load gave up (the block then left
// its tile unwritten); read and cleared by depix_take_device_faults
__device__ int g_raster_fault;

// Compile-time scale of a raster kernel: 1..4 and 8 themselves, 0 the scales
// 5 to 7, -1 the scales above 8.
__host__ __device__ constexpr int raster_mode(int s) { return (s <= 4 || s == 8) ? s : (s < 8 ? 0 : -1); }
__host__ __device__ constexpr MaskLayout mode_layout(int S) { return S <= 0 ? ML_ROWS : mask_layout(S); }

// Threads of a raster block, and the blocks per SM that its registers leave
// room for: 48 registers and five blocks up to x4, whose masks take 23 KB of a
// 32x32 tile (1024 frames of 256x224 at x4: 128 threads and six blocks 965 us,
// 256 and four 956, 256 and five 886); above, the masks allow three.
constexpr int kRT = 256;
constexpr int raster_blocks(int S) { return S > 0 && S <= 4 ? 5 : 3; }

template <int S, int TW, int TH>
struct MaskTile {
    static constexpr int GW = TW + 2, GH = TH + 2, GN = GW * GH; // cells with their ring
    static constexpr int BW = TW + 6, BH = TH + 6;               // graph, halo 3
    static constexpr int CW = TW + 4, CH = TH + 4;               // pixels, halo 2
    // pixels (RGBA words; the alpha byte may hold anything) with halo 2,
    // stored from two columns further left (x0 - 4) so that a TMA box can
    // start on a 16-byte boundary: pixel (lx, ly) of the halo-2 window is
    // pix[ly][lx + 2]
    __align__(128) uint32_t pix[CH][CW + 4];
    uint64_t bar;      // completion of the TMA loads
    int tma_ok;
    // graph bytes with halo 3, stored from 13 columns further left (x0 - 16)
    // so that a TMA box starts on a 16-byte boundary: graph byte (bx, by) of
    // the halo-3 window is graph[by][bx + kGOff]
    static constexpr int kGOff = 13, GRW = TW + 32;
    __align__(128) uint8_t graph[BH][GRW];
    // sample groups of a block that are resolved at once (at most 16 samples):
    // the whole block up to x4, two of its rows at x8
    static constexpr int NG = S == 8 ? 4 : 1;
    static constexpr uint32_t kFull = S == 4 || S == 8 ? 0xFFFFu : (S > 0 && S < 4 ? (1u << (S * S & 15)) - 1u : 0u);
    static constexpr int NL = GN > TW * TH * NG ? GN : TW * TH * NG;
    uint16_t list[NL]; // subdivided cells of the tile, then the sample groups that need owner resolution
    int count;         // cells in list
    int slow;          // groups in list
};

// RGBA word of one pixel with alpha 255
template <int LAYOUT>
__device__ __forceinline__ uint32_t load_rgba(const uint8_t* img, int ws, int i, int j)
{
    if (LAYOUT == DEPIX_LAYOUT_RGBA) return reinterpret_cast<const uint32_t*>(img + (size_t)j * ws)[i];
    const uint32_t p = load_bgr(img, ws, LAYOUT, i, j);
    return ((p >> 16) & 0xFFu) | (p & 0xFF00u) | ((p & 0xFFu) << 16);
}

// a slot in a shared list for every lane with pred, one atomic per warp (all
// lanes call it)
__device__ __forceinline__ int list_slot(int* counter, bool pred)
{
    const unsigned m = __ballot_sync(0xFFFFFFFFu, pred);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (m && lane == __ffs(m) - 1) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, m ? __ffs(m) - 1 : 0);
    return base + __popc(m & ((1u << lane) - 1u));
}

// Mask of a cut polygon that is not star-shaped about its cell centre: built
// and ear-clipped as the reference does, triangle by triangle. g: the cell's
// graph byte in the tile window (rows of `pitch` bytes); keep: bit c the
// corner test at corner c (as CutTables::corners), bit 4 every vertex kept.
__device__ __noinline__ void ear_clip_cell_mask(const uint8_t* g, int pitch, unsigned keep, int s, uint32_t* dst,
                                                uint16_t* info)
{
    const MaskGeom G = mask_geom(s);
    auto pattern = [&](const uint8_t* q) { return cell_pattern(q[0], q[-1], q[1]); };
    Poly c, p;
    hull_from_lut(__ldg(&g_hull_lut[pattern(g)]), c);
    subdivide_cell(
        c, g[0], [&](int L, Poly& nb) { hull_from_lut(__ldg(&g_hull_lut[pattern(g + dir_dj(L) * pitch + dir_di(L))]), nb); },
        [&](int px, int py) -> bool {
            if (keep & 16u) return true;
            if (px == 0 && py == 0) return keep & 1u;
            if (px == kUnit && py == 0) return keep & 2u;
            if (px == kUnit && py == kUnit) return keep & 4u;
            if (px == 0 && py == kUnit) return keep & 8u;
            return false;
        },
        p);
    uint8_t tri[3 * kMaxPoly];
    bool ok;
    const int nt = ear_clip(p, tri, ok), u = 4 * s;
    uint32_t rows[32];
    for (int r = 0; r < 32; r++) rows[r] = 0;
    for (int t = 0; t < nt; t++) {
        const int a = tri[3 * t], b = tri[3 * t + 1], d = tri[3 * t + 2];
        tri_mask(p.x[a] * u, p.y[a] * u, p.x[b] * u, p.y[b] * u, p.x[d] * u, p.y[d] * u, G.mlo, G.F, rows);
    }
    pack_mask(G, rows, dst);
    if (mask_layout(s) == ML_ROWS) {
        const uint32_t blockbits = (1u << s) - 1u;
        unsigned touched = 512u;
        for (int r = 0; r < G.F; r++) {
            const int m = r + G.mlo, dj = m < 0 ? 0 : (m >= s ? 2 : 1);
            const uint64_t x = (uint64_t)rows[r] << (s + G.mlo);
            for (int di = 0; di < 3; di++)
                if ((x >> (di * s)) & blockbits) touched |= 1u << (dj * 3 + di);
            if (dj == 1 && ((rows[r] >> -G.mlo) & blockbits) != blockbits) touched &= ~512u;
        }
        *info = (uint16_t)touched;
    }
}

// XOR of table entries in registers
template <MaskLayout ML>
struct MaskAcc {
    static constexpr int W = ML == ML_U16 ? 5 : 18;
    uint32_t w[W];
    unsigned flags;
    uint32_t* dst;
    __device__ __forceinline__ MaskAcc(uint32_t* d, const MaskGeom&, uint16_t*) : flags(0), dst(d)
    {
#pragma unroll
        for (int k = 0; k < W; k++) w[k] = 0;
    }
    __device__ __forceinline__ void add(const uint32_t* e)
    {
        const uint4* q = reinterpret_cast<const uint4*>(e);
        if constexpr (ML == ML_U16) {
            const uint4 a = __ldg(q);
            const uint32_t b = __ldg(e + 4);
            w[0] ^= a.x; w[1] ^= a.y; w[2] ^= a.z; w[3] ^= a.w;
            w[4] ^= b & 0xFFFFu;
            flags += b >> 16;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint4 a = __ldg(q + k);
                w[4 * k] ^= a.x; w[4 * k + 1] ^= a.y; w[4 * k + 2] ^= a.z; w[4 * k + 3] ^= a.w;
            }
            const uint4 a = __ldg(q + 4);
            w[16] ^= a.x; w[17] ^= a.y;
            flags += a.z;
        }
    }
    __device__ __forceinline__ void store() const
    {
#pragma unroll
        for (int k = 0; k < W; k++) dst[k] = w[k];
    }
};
// rows: store() also notes the parts that the mask touches (bits 0-8) and
// whether it covers its own block (bit 9). A cell linked on its four sides only
// is its own square (kSquare) and has no mask, which spares the stores of up to
// 31 rows (100 frames of 152x102 without subdivision: x5 85 us with them, x12
// 206; 79 and 194 without).
constexpr unsigned kSquare = 1024;
template <int MODE>
struct MaskAccRows {
    static constexpr int NQ = MODE == 0 ? 5 : 8; // row quads: F + 1 is at most 18 up to x7, 31 up to x12
    uint32_t w[4 * NQ];
    uint32_t* dst;
    uint16_t* info;
    MaskGeom G;
    unsigned flags;
    __device__ __forceinline__ MaskAccRows(uint32_t* d, const MaskGeom& G_, uint16_t* i) : dst(d), info(i), G(G_), flags(0)
    {
#pragma unroll
        for (int k = 0; k < 4 * NQ; k++) w[k] = 0;
    }
    __device__ __forceinline__ void add(const uint32_t* e)
    {
#pragma unroll
        for (int k = 0; k < NQ; k++)
            if (4 * k < G.F) {
                const uint4 a = __ldg(reinterpret_cast<const uint4*>(e) + k);
                w[4 * k] ^= a.x; w[4 * k + 1] ^= a.y; w[4 * k + 2] ^= a.z; w[4 * k + 3] ^= a.w;
            }
        flags += __ldg(e + G.F);
    }
    __device__ __forceinline__ void store() const
    {
        const uint32_t blockbits = (1u << G.s) - 1u;
        uint32_t lo = 0, mid = 0, hi = 0, all = blockbits;
#pragma unroll
        for (int r = 0; r < 4 * NQ; r++) {
            const int m = r + G.mlo;
            if (r >= G.F) break;
            dst[r] = w[r];
            if (m < 0) lo |= w[r];
            else if (m >= G.s) hi |= w[r];
            else {
                mid |= w[r];
                all &= w[r] >> -G.mlo;
            }
        }
        *info = (uint16_t)(mask_columns(G, lo) | mask_columns(G, mid) << 3 | mask_columns(G, hi) << 6 |
                           (all == blockbits ? 512u : 0u));
    }
    // bit di + 1 set when a footprint row's bits reach the block column di
    static __device__ __forceinline__ unsigned mask_columns(const MaskGeom& G, uint32_t row)
    {
        const uint64_t x = (uint64_t)row << (G.s + G.mlo);
        const uint32_t blockbits = (1u << G.s) - 1u;
        return ((x & blockbits) ? 1u : 0u) | ((x >> G.s & blockbits) ? 2u : 0u) | ((x >> (2 * G.s)) ? 4u : 0u);
    }
};

// Mask of a subdivided cell as the XOR of its pieces. pat, g: its pattern and
// its graph byte in the tile window (rows of `pitch` bytes); keep_of(corner
// classes) the corners (bits 0-3, as CutTables::corners) that the T-junction
// test keeps, bit 4 when it keeps every vertex.
template <typename Acc, typename Keep>
__device__ __forceinline__ void cut_cell_mask(Acc& acc, int pat, const uint8_t* g, int pitch, const uint32_t* lut,
                                              int ES, Keep keep_of)
{
    const uint4 ed = __ldg(&g_cut.edges[pat]);
    const uint32_t corners = __ldg(&g_cut.corners[pat]);
    acc.add(lut + (size_t)(kCutEntry + pat) * ES);
    // the edges' loads in two rounds, each round's in flight together
    const uint32_t e4[4] = {ed.x, ed.y, ed.z, ed.w};
    int cls[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        cls[t] = 0;
        if (e4[t]) {
            const int L = (int)(e4[t] >> 20) & 7;
            const uint8_t* nb = g + dir_dj(L) * pitch + dir_di(L);
            cls[t] = __ldg(&g_cut.nb_class[((e4[t] >> 16) & 15u) * 4096 + cell_pattern(nb[0], nb[-1], nb[1])]);
        }
    }
#pragma unroll
    for (int t = 0; t < 4; t++)
        if (e4[t]) acc.add(lut + (size_t)(kPathEntry + (int)(e4[t] & 0xFFFFu) + cls[t]) * ES);
    const unsigned keep = keep_of(corners);
    if (keep & 16u) {
        const uint64_t verts = __ldg(&g_cut.verts[pat]);
#pragma unroll 1
        for (int v = 0; v < 8; v++) {
            const int id = (int)(verts >> (8 * v)) & 0xFF;
            if (id != 0xFF) acc.add(lut + (size_t)(kCornerEntry + id) * ES);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int id = (int)(corners >> (8 * c)) & 0xFF;
            if (((keep >> c) & 1u) && id != 0xFF) acc.add(lut + (size_t)(kCornerEntry + id) * ES);
        }
    }
}

// The four corner tests (checkTJunction, subdivision_functions.cu:170-242) of
// a cell off the image's edge, px its pixel in the tile (rows of PW words):
// bit c set when the corner's neighbour colours differ.
__device__ __forceinline__ unsigned corner_tests(const uint32_t* px, int PW)
{
    auto ne = [&](int a, int b) -> unsigned { return ((px[a] ^ px[b]) & 0x00FFFFFFu) != 0; };
    return (ne(-1, -PW - 1) | ne(-PW - 1, -PW)) | (ne(1, -PW + 1) | ne(-PW + 1, -PW)) << 1 |
           (ne(PW, PW + 1) | ne(PW + 1, 1)) << 2 | (ne(PW - 1, PW) | ne(PW, -1)) << 3;
}

// Colour (B | G << 8 | R << 16) that the reference's linear addressing reads
// at the pixel (i, j) one column outside the image (i = -1 or w) or above it:
// bytes of the rows before and after, of a row's padding (for RGBA input that
// of the 4-byte aligned BGR rows the reference would have loaded: zeros), or
// zero outside the buffer.
template <int LAYOUT>
__device__ uint32_t wrapped_colour(const uint8_t* img, int ws, int w, int h, int i, int j)
{
    if (LAYOUT == DEPIX_LAYOUT_BGR) {
        uint32_t c = 0;
        const long long off = (long long)j * ws + 3LL * i, end = (long long)h * ws;
        for (int b = 0; b < 3; b++)
            if (off + b >= 0 && off + b < end) c |= (uint32_t)img[off + b] << (8 * b);
        return c;
    }
    const int pad = 8 * (((3 * w + 3) & ~3) - 3 * w); // bits of padding after a row
    if (i < 0) return j >= 1 && j <= h ? load_bgr(img, ws, LAYOUT, w - 1, j - 1) >> pad : 0u;
    if (i >= w) return j + 1 < h ? (load_bgr(img, ws, LAYOUT, 0, j + 1) << pad) & 0x00FFFFFFu : 0u;
    return 0u; // above the last row
}

// The corner tests of a cell on the image's edge (as corner_tests), bit 4 when
// the reference's bounds test keeps every vertex. Neighbours outside the image
// as its linear addressing reads them, the others from the tile's pixels px
// (rows of PW words).
template <int LAYOUT>
__device__ __noinline__ unsigned edge_corner_tests(const uint32_t* px, int PW, const uint8_t* img, int ws, int w, int h,
                                                   int ci, int cj)
{
    const long long st = LAYOUT == DEPIX_LAYOUT_BGR ? ws : ((3 * w + 3) & ~3);
    const long long index = (long long)cj * st + (long long)ci * 3;
    if ((index - st - 1) < 0 || (index + w + 1) > ((long long)h * st - 1)) return 16u;
    auto at = [&](int dx, int dy) -> uint32_t {
        const int i = ci + dx, j = cj + dy;
        if (i < 0 || i >= w || j >= h) return wrapped_colour<LAYOUT>(img, ws, w, h, i, j);
        const uint32_t c = px[dy * PW + dx];
        return ((c >> 16) & 0xFFu) | (c & 0xFF00u) | ((c & 0xFFu) << 16);
    };
    const uint32_t l = at(-1, 0), r = at(1, 0), d = at(0, -1), u = at(0, 1);
    const uint32_t dl = at(-1, -1), dr = at(1, -1), ul = at(-1, 1), ur = at(1, 1);
    return (unsigned)(l != dl || dl != d) | (unsigned)(r != dr || dr != d) << 1 | (unsigned)(u != ur || ur != r) << 2 |
           (unsigned)(ul != u || u != l) << 3;
}

template <int LAYOUT, int S, int TW, int TH, bool TMA = false>
__device__ void mask_raster_tile(MaskTile<S, TW, TH>& M, uint32_t* masks, const uint8_t* img, int ws, const uint8_t* g,
                                 uint8_t* out, int w, int h, int scale, bool subdivide, const uint32_t* lut, int x0,
                                 int y0, int32_t* labels, const CUtensorMap* pix_map = nullptr, int frame = 0,
                                 const CUtensorMap* graph_map = nullptr)
{
    using T = MaskTile<S, TW, TH>;
    constexpr MaskLayout ML = mode_layout(S);
    using Acc = std::conditional_t<ML == ML_ROWS, MaskAccRows<S>, MaskAcc<ML == ML_ROWS ? ML_U16 : ML>>;
    const int s = S > 0 ? S : scale;
    const MaskGeom G = mask_geom(s);
    const int MS = mask_stride(s), ES = entry_words(s), MW = mask_words(s);
    // rows layout: after the masks the cells' touched parts
    uint16_t* info = reinterpret_cast<uint16_t*>(masks + T::GN * MS);
    constexpr uint32_t kAlpha = 0xFF000000u;
    // ---- phase A
    if constexpr (TMA) {
        // the pixel window (x0 - 4 .. x0 + TW + 4) x (y0 - 2 .. y0 + TH + 2)
        // and, with a graph map, the graph window (x0 - 16 .. x0 + TW + 16) x
        // (y0 - 3 .. y0 + TH + 3) by TMA tile loads on one barrier
        if (threadIdx.x == 0) {
            mbar_init(&M.bar, 1);
            mbar_expect_tx(&M.bar, (uint32_t)(sizeof(M.pix) + (graph_map ? sizeof(M.graph) : 0)));
            tma_load_3d(&M.pix[0][0], pix_map, x0 - 4, y0 - 2, frame, &M.bar);
            if (graph_map) tma_load_3d(&M.graph[0][0], graph_map, x0 - T::kGOff - 3, y0 - 3, frame, &M.bar);
        }
    }
    if (threadIdx.x == 0) {
        M.count = 0;
        M.slow = 0;
    }
    // the roots of the tile's labels, while the loads are under way (1024 frames
    // of 256x224 at x4: 120 us as a kernel of its own, 85 here; 156 when the
    // warps do it at the tile's end; 4096 sprites 33 and 10)
    if (labels) flatten_tile<TW, TH>(labels, w, h, x0, y0);
    if (!(TMA && graph_map)) {
        // the window's words, from the one that holds its first byte
        constexpr int C0 = T::kGOff / 4, NC = (T::kGOff + T::BW + 3) / 4 - C0;
        for_each_batched<2>(
            NC * T::BH,
            [&](int k) {
                const int gx = x0 - 3 - T::kGOff + 4 * (C0 + k % NC), gy = y0 - 3 + k / NC;
                return row_bytes4(g, w, h, gx, gy) & inside_mask4(gx, gy, w, h);
            },
            [&](int k, uint32_t v) { *reinterpret_cast<uint32_t*>(&M.graph[k / NC][4 * (C0 + k % NC)]) = v; });
    }
    if constexpr (TMA) {
        if (threadIdx.x == 0) {
            M.tma_ok = tma_wait_or_flag(&M.bar, &g_raster_fault) ? 1 : 0;
        }
        __syncthreads();
        if (!M.tma_ok) return;
        // graph bytes on the image's edge lose their bits toward outside (the
        // box reads zero beyond the image); only tiles that reach an edge
        if (graph_map && (x0 < 3 || y0 < 3 || x0 + TW + 3 > w || y0 + TH + 3 > h)) {
            for (int k = threadIdx.x; k < T::BW * T::BH; k += blockDim.x) {
                const int gx = x0 - 3 + k % T::BW, gy = y0 - 3 + k / T::BW;
                if (gx >= 0 && gy >= 0 && gx < w && gy < h)
                    M.graph[k / T::BW][k % T::BW + T::kGOff] &= (uint8_t)inside_mask(gx, gy, w, h);
            }
            __syncthreads();
        }
    } else {
        for_each_batched<3>(
            T::CW * T::CH,
            [&](int k) {
                const int gx = x0 - 2 + k % T::CW, gy = y0 - 2 + k / T::CW;
                return gx >= 0 && gy >= 0 && gx < w && gy < h ? load_rgba<LAYOUT>(img, ws, gx, gy) : 0u;
            },
            [&](int k, uint32_t v) { M.pix[k / T::CW][k % T::CW + 2] = v; });
        __syncthreads();
    }

    // ---- phase B: plain cells from the table, subdivided cells to the list
    for (int k0 = 0; k0 < T::GN; k0 += blockDim.x) {
        const int k = k0 + threadIdx.x;
        bool cut = false;
        if (k < T::GN) {
            const int lx = k % T::GW, ly = k / T::GW;
            const int ci = x0 - 1 + lx, cj = y0 - 1 + ly;
            uint32_t* dst = masks + k * MS;
            if (ci < 0 || cj < 0 || ci >= w || cj >= h) {
                if (ML == ML_ROWS) info[k] = 0;
                else
                    for (int r = 0; r < MW; r++) dst[r] = 0;
            } else {
                const uint8_t* gb = &M.graph[ly + 2][lx + 2 + T::kGOff];
                const unsigned node = gb[0];
                cut = subdivide && node != 90;
                if (!cut) {
                    if (node == 90) {
                        // linked on its four sides only: its own square, part 4
                        if constexpr (ML == ML_U16) {
                            dst[0] = dst[1] = dst[3] = dst[4] = 0;
                            dst[2] = T::kFull;
                        } else if constexpr (ML == ML_U64) {
#pragma unroll
                            for (int r = 0; r < 18; r++) dst[r] = r == 8 || r == 9 ? 0xFFFFFFFFu : 0u;
                        } else {
                            info[k] = kSquare | 512 | 16;
                        }
                    } else {
                        Acc acc(dst, G, info + k);
                        acc.add(lut + (size_t)(kPlainEntry + cell_pattern(node, gb[-1], gb[1])) * ES);
                        acc.store();
                    }
                }
            }
        }
        const int slot = list_slot(&M.count, cut);
        if (cut) M.list[slot] = (uint16_t)k;
    }
    __syncthreads();

    // ---- phase B2: subdivided cells, XORed from their pieces
    const int nlist = M.count;
    for (int q = threadIdx.x; q < nlist; q += blockDim.x) {
        const int k = M.list[q], lx = k % T::GW, ly = k / T::GW;
        const int ci = x0 - 1 + lx, cj = y0 - 1 + ly;
        const uint8_t* gb = &M.graph[ly + 2][lx + 2 + T::kGOff];
        const uint32_t* px = &M.pix[ly + 1][lx + 3];
        constexpr int PW = T::CW + 4;
        const int pat = cell_pattern(gb[0], gb[-1], gb[1]);
        const bool edge = ci == 0 || cj == 0 || ci == w - 1 || cj == h - 1;
        unsigned keep = edge ? edge_corner_tests<LAYOUT>(px, PW, img, ws, w, h, ci, cj) : 0u;
        Acc acc(masks + k * MS, G, info + k);
        cut_cell_mask(acc, pat, gb, T::GRW, lut, ES, [&](uint32_t corners) {
            if (!edge && corners != 0xFFFFFFFFu) keep = corner_tests(px, PW);
            return keep;
        });
        if ((acc.flags & 0xFFFFu) == 1u) acc.store();
        else ear_clip_cell_mask(gb, T::GRW, keep, s, masks + k * MS, info + k); // not star-shaped
    }
    __syncthreads();

    // ---- phase C: output blocks (one per tile cell). Candidate q = 0..8 of a
    // block is the cell at (1 - q % 3, 1 - q / 3) from it: VBO order from the
    // latest (row above, right to left) to the earliest; its part over the
    // block is part q of its mask.
    const int ow = w * s;
    const bool vec = (S == 4 || S == 8) && (ow % 4) == 0 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
    if constexpr (ML == ML_ROWS) {
        // A warp takes 32 blocks of the tile (one or two of its rows) and
        // writes the output rows of those that their own cell fills in order,
        // four pixels a lane, so that the stores are contiguous whatever s is;
        // the rows of the other blocks follow, one a thread. (Resolving each
        // row of the 32 blocks in the warp and writing it whole: 132 us for 100
        // frames of 152x102 at x5, 96 us so; parts of 64 bits and one thread a
        // block, which stores every pixel apart: 171.)
        constexpr int CM = S == 0 ? 7 : 12; // most samples of a row
        const uint32_t blockbits = (1u << s) - 1u;
        const unsigned inv = (1u << 20) / (unsigned)s + 1u; // x / s = x inv >> 20 for x up to a tile's rows (12 k)
        const int lane = threadIdx.x & 31;
        const bool quads = (ow % 4) == 0 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
        for (int b0 = threadIdx.x & ~31; b0 < TW * TH; b0 += blockDim.x) {
            const int tx = lane % TW, ty = (b0 + lane) / TW, k = (ty + 1) * T::GW + tx + 1;
            const bool in = x0 + tx < w && y0 + ty < h;
            auto touch = [&](int q) { return (unsigned)info[k + (1 - q / 3) * T::GW + 1 - q % 3] >> q & 1u; };
            const bool fill = (info[k] & 512u) && !(touch(0) | touch(1) | touch(2) | touch(3));
            const uint32_t own = M.pix[ty + 2][tx + 4] | kAlpha;
            const int slot = list_slot(&M.slow, in && !fill);
            if (in && !fill) M.list[slot] = (uint16_t)(b0 + lane);
            const unsigned filled = __ballot_sync(0xFFFFFFFFu, in && fill);
            if (!filled) continue;
            const int per = quads ? 4 : 1;
            for (int i0 = 0; i0 < 32 * s; i0 += 32 * per) {
                const int i = i0 + per * lane;
                const bool live = i < 32 * s;
                // a lane's pixels lie in at most two blocks (s > 4)
                const int ba = live ? (int)(i * inv >> 20) : 0, bb = live ? (int)((i + per - 1) * inv >> 20) : 0;
                const uint32_t ca = __shfl_sync(0xFFFFFFFFu, own, ba), cb = __shfl_sync(0xFFFFFFFFu, own, bb);
                const bool fa = filled >> ba & 1u, fb = filled >> bb & 1u;
                if (!live || !(fa || fb)) continue;
                const int row = TW == 32 ? 0 : (i >= TW * s);
                uint32_t* o = reinterpret_cast<uint32_t*>(out) + (size_t)((y0 + b0 / TW + row) * s) * ow +
                              (x0 * s + i - row * TW * s);
                const int left = bb * s - i; // pixels of the lane in block ba, when the blocks differ
                if (!quads) {
                    for (int r = 0; r < s; r++) o[(size_t)r * ow] = ca;
                } else if (fa && fb) {
                    const uint4 v = ba == bb ? make_uint4(ca, ca, ca, ca)
                                             : make_uint4(ca, left > 1 ? ca : cb, left > 2 ? ca : cb, cb);
                    for (int r = 0; r < s; r++) __stcs(reinterpret_cast<uint4*>(o + (size_t)r * ow), v);
                } else {
                    for (int r = 0; r < s; r++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            if ((ba == bb || c < left) ? fa : fb) o[(size_t)r * ow + c] = (ba == bb || c < left) ? ca : cb;
                }
            }
        }
        __syncthreads();
        const int rows = M.slow * s;
        for (int i = threadIdx.x; i < rows; i += blockDim.x) {
            const int bi = (int)((unsigned)i * inv >> 20), r = i - bi * s, q0 = M.list[bi];
            const int tx = q0 % TW, ty = q0 / TW, k = (ty + 1) * T::GW + tx + 1;
            const uint32_t* px = &M.pix[ty + 2][tx + 4];
            uint32_t col[CM], claimed = 0;
#pragma unroll
            for (int c = 0; c < CM; c++) col[c] = kAlpha; // no owner: the clear colour
            unsigned owners = 0; // candidates that touch the block
#pragma unroll
            for (int q = 0; q < 9; q++)
                owners |= (unsigned)info[k + (1 - q / 3) * T::GW + 1 - q % 3] & 1u << q;
            while (owners && claimed != blockbits) {
                const int q = __ffs(owners) - 1, dj = 1 - q / 3, di = 1 - q % 3;
                owners &= owners - 1;
                const int rr = r - s * dj - G.mlo, sh = s * di + G.mlo; // block column = footprint column + sh
                if (rr < 0 || rr >= G.F) continue;
                uint32_t take = blockbits & ~claimed;
                if (q != 4 || !(info[k] & kSquare)) {
                    const uint64_t m = masks[(k + dj * T::GW + di) * MS + rr];
                    take &= (uint32_t)(sh >= 0 ? m << sh : m >> -sh);
                }
                const uint32_t c0 = px[dj * (T::CW + 4) + di] | kAlpha;
                claimed |= take;
#pragma unroll
                for (int c = 0; c < CM; c++)
                    if (take >> c & 1u) col[c] = c0;
            }
            uint32_t* o = reinterpret_cast<uint32_t*>(out) + (size_t)((y0 + ty) * s + r) * ow + (size_t)(x0 + tx) * s;
            if (S < 0 && quads && s % 4 == 0) {
#pragma unroll
                for (int c = 0; c < CM; c += 4)
                    if (c < s) __stcs(reinterpret_cast<uint4*>(o + c), make_uint4(col[c], col[c + 1], col[c + 2], col[c + 3]));
            } else {
#pragma unroll
                for (int c = 0; c < CM; c++)
                    if (c < s) o[c] = col[c];
            }
        }
        return;
    }
    auto cand = [&](int k, int q) -> const uint32_t* { return masks + (k + (1 - q / 3) * T::GW + 1 - q % 3) * MS; };
    constexpr int NG = T::NG;
    constexpr int GR = S == 8 ? 2 : (S > 0 ? S : 1); // rows of a group
    constexpr uint32_t kFull = T::kFull;
    auto group = [&](int k, int q, int gr) -> uint32_t { // candidate q's part over the group
        const uint16_t* m = reinterpret_cast<const uint16_t*>(cand(k, q));
        return m[S == 8 ? 4 * q + gr : q];
    };
    for (int i = threadIdx.x; i < TW * TH * NG; i += blockDim.x) {
        const int q = i % (TW * TH), gr = i / (TW * TH);
        const int tx = q % TW, ty = q / TW;
        const int ci = x0 + tx, cj = y0 + ty;
        const bool in = ci < w && cj < h;
        const int k = (ty + 1) * T::GW + tx + 1;
        // filled at once: its own cell covers all of it and no later one any
        bool fill = false;
        if (in)
            fill = group(k, 4, gr) == kFull &&
                   (group(k, 0, gr) | group(k, 1, gr) | group(k, 2, gr) | group(k, 3, gr)) == 0;
        const int slot = list_slot(&M.slow, in && !fill);
        if (in && !fill) M.list[slot] = (uint16_t)i; // resolved after the barrier, over a compacted list
        if (!fill) continue;
        const uint32_t col = M.pix[ty + 2][tx + 4] | kAlpha;
        uint8_t* orow = out + (((size_t)cj * s + gr * GR) * ow + (size_t)ci * s) * 4;
#pragma unroll
        for (int r = 0; r < GR; r++) {
            uint32_t* o = reinterpret_cast<uint32_t*>(orow + (size_t)r * ow * 4);
            if (vec) {
#pragma unroll
                for (int c4 = 0; c4 < S; c4 += 4) __stcs(reinterpret_cast<uint4*>(o + c4), make_uint4(col, col, col, col));
            } else {
                for (int c = 0; c < s; c++) o[c] = col;
            }
        }
    }
    __syncthreads();
    const int nslow = M.slow;
    for (int qs = threadIdx.x; qs < nslow; qs += blockDim.x) {
        const int i = M.list[qs], q = i % (TW * TH), gr = i / (TW * TH);
        const int tx = q % TW, ty = q / TW;
        const int ci = x0 + tx, cj = y0 + ty;
        const int k = (ty + 1) * T::GW + tx + 1;
        uint8_t* orow = out + (((size_t)cj * s + gr * GR) * ow + (size_t)ci * s) * 4;
        const uint32_t* px = &M.pix[ty + 2][tx + 4];
        // candidates from the latest on until every sample has its owner
        // (each lane walks its own block's owners, so that a warp's trips
        // are the most owners of a block, not the nine candidates)
        constexpr int NS = S == 8 ? 16 : (S > 0 ? S * S : 1), RL = S;
        uint32_t col[NS], claimed = 0;
        unsigned owners = 0;
#pragma unroll
        for (int q = 0; q < 9; q++) {
            const uint32_t m = group(k, q, gr);
            if (m & ~claimed) owners |= 1u << q;
            claimed |= m;
        }
#pragma unroll
        for (int c = 0; c < NS; c++) col[c] = kAlpha; // no owner: the clear colour
        claimed = 0;
        while (owners) {
            const int q = __ffs(owners) - 1;
            owners &= owners - 1;
            const int dj = 1 - q / 3, di = 1 - q % 3;
            const uint16_t* mp = reinterpret_cast<const uint16_t*>(masks + (k + dj * T::GW + di) * MS);
            const uint32_t m = mp[S == 8 ? 4 * q + gr : q], take = m & ~claimed;
            const uint32_t c0 = px[dj * (T::CW + 4) + di] | kAlpha;
            claimed |= m;
#pragma unroll
            for (int c = 0; c < NS; c++)
                if ((take >> c) & 1u) col[c] = c0;
        }
#pragma unroll
        for (int r = 0; r < GR; r++) {
            uint32_t* o = reinterpret_cast<uint32_t*>(orow + (size_t)r * ow * 4);
            if (vec) {
#pragma unroll
                for (int c4 = 0; c4 + 3 < RL; c4 += 4)
                    __stcs(reinterpret_cast<uint4*>(o + c4), make_uint4(col[r * RL + c4], col[r * RL + c4 + 1],
                                                                        col[r * RL + c4 + 2], col[r * RL + c4 + 3]));
            } else {
#pragma unroll
                for (int c = 0; c < RL; c++) o[c] = col[r * RL + c];
            }
        }
    }
}

template <int LAYOUT, int S, int TH, int NT>
__global__ void __launch_bounds__(NT, raster_blocks(S) * kRT / NT) k_mask_raster(RasterBatch b, const uint32_t* lut)
{
    follow_last();
    __shared__ MaskTile<S, 32, TH> M;
    extern __shared__ uint32_t masks[];
    size_t z = blockIdx.z;
    mask_raster_tile<LAYOUT, S, 32, TH>(M, masks, b.img + b.img_stride * z, b.ws, b.graph + b.graph_stride * z,
                                        b.out + b.out_stride * z, b.w, b.h, b.scale, b.subdivide != 0, lut,
                                        blockIdx.x * 32, blockIdx.y * TH,
                                        b.labels ? b.labels + b.label_stride * z : nullptr);
}

// The equal-size batch raster with its pixel windows loaded by TMA (RGBA
// frames whose base, rows and frame stride are 16-byte aligned).
template <int S, int TH, int NT>
__global__ void __launch_bounds__(NT, raster_blocks(S) * kRT / NT) k_mask_raster_tma(RasterBatch b, const uint32_t* lut,
                                                         const __grid_constant__ CUtensorMap pix_map,
                                                         const __grid_constant__ CUtensorMap graph_map, int with_graph)
{
    follow_last();
    __shared__ MaskTile<S, 32, TH> M;
    extern __shared__ uint32_t masks[];
    size_t z = blockIdx.z;
    mask_raster_tile<DEPIX_LAYOUT_RGBA, S, 32, TH, true>(M, masks, b.img + b.img_stride * z, b.ws,
                                                         b.graph + b.graph_stride * z, b.out + b.out_stride * z, b.w,
                                                         b.h, b.scale, b.subdivide != 0, lut, blockIdx.x * 32,
                                                         blockIdx.y * TH,
                                                         b.labels ? b.labels + b.label_stride * z : nullptr, &pix_map, (int)z,
                                                         with_graph ? &graph_map : nullptr);
}

bool rgba_tensor_map(const uint8_t* img, int w, int h, int ws, size_t frame_stride, int nframes, int box_w, int box_h,
                     CUtensorMap* map);

using TensorMapEncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                          const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                          CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                          CUtensorMapFloatOOBfill);

static TensorMapEncodeTiled tensor_map_encoder();

// A tensor map of RGBA frames as words, (w, h, frames), box (box_w, box_h, 1).
// False when the frames do not meet TMA's rules (16-byte aligned base, row
// and frame strides) or no encoder is available.
bool rgba_tensor_map(const uint8_t* img, int w, int h, int ws, size_t frame_stride, int nframes, int box_w, int box_h,
                     CUtensorMap* map)
{
    if ((reinterpret_cast<uintptr_t>(img) & 15) || (ws & 15) || w < 1 || h < 1) return false;
    const uint64_t fstride = nframes > 1 ? (uint64_t)frame_stride : ((uint64_t)ws * h + 15) & ~15ull;
    if (fstride & 15) return false;
    const TensorMapEncodeTiled enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nframes};
    const cuuint64_t strides[2] = {(cuuint64_t)ws, (cuuint64_t)fstride};
    const cuuint32_t box[3] = {(cuuint32_t)box_w, (cuuint32_t)box_h, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t*>(img), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A tensor map of 8-bit frames (graph bytes), (w, h, frames), box (box_w,
// box_h, 1); false when the buffers do not meet TMA's rules.
bool u8_tensor_map(const uint8_t* base, int w, int h, size_t frame_stride, int nframes, int box_w, int box_h,
                   CUtensorMap* map)
{
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (w & 15) || w < 1 || h < 1) return false;
    const uint64_t fstride = nframes > 1 ? (uint64_t)frame_stride : ((uint64_t)w * h + 15) & ~15ull;
    if (fstride & 15) return false;
    const TensorMapEncodeTiled enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nframes};
    const cuuint64_t strides[2] = {(cuuint64_t)w, (cuuint64_t)fstride};
    const cuuint32_t box[3] = {(cuuint32_t)box_w, (cuuint32_t)box_h, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static TensorMapEncodeTiled tensor_map_encoder()
{
    static TensorMapEncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<TensorMapEncodeTiled>(p);
    }();
    return fn;
}

static bool pixel_tensor_map(const RasterBatch& b, int nframes, int TH, CUtensorMap* map)
{
    if (b.layout != DEPIX_LAYOUT_RGBA) return false;
    return rgba_tensor_map(b.img, b.w, b.h, b.ws, b.img_stride, nframes, 32 + 8, TH + 4, map);
}

// dynamic shared memory: the cells' masks, in the rows layout also what they
// touch
template <int S, int TW, int TH>
static size_t mask_smem(int scale)
{
    constexpr size_t GN = MaskTile<S, TW, TH>::GN;
    size_t words = GN * mask_stride(scale);
    if (mode_layout(S) == ML_ROWS) words += (GN + 1) / 2;
    return words * sizeof(uint32_t);
}

template <int LAYOUT, int S, int TH, int NT>
static cudaError_t launch_mask_raster_nt(const RasterBatch& b, int nframes, const uint32_t* lut, cudaStream_t s)
{
    const bool early = early_stages((long long)b.w * b.h * nframes);
    if constexpr (LAYOUT == DEPIX_LAYOUT_RGBA) {
        CUtensorMap map;
        if (pixel_tensor_map(b, nframes, TH, &map)) {
            size_t smem = mask_smem<S, 32, TH>(b.scale);
            if (smem + sizeof(MaskTile<S, 32, TH>) > 48 * 1024) {
                cudaError_t e = cudaFuncSetAttribute(k_mask_raster_tma<S, TH, NT>,
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                if (e != cudaSuccess) return e;
            }
            // the graph window too, when the graph's width and frame stride allow it
            CUtensorMap gmap;
            const bool with_graph = u8_tensor_map(b.graph, b.w, b.h, b.graph_stride, nframes, 32 + 32, TH + 6, &gmap);
            if (!with_graph) gmap = map; // unused
            dim3 grid((b.w + 32 - 1) / 32, (b.h + TH - 1) / TH, nframes);
            return launch_early(early, k_mask_raster_tma<S, TH, NT>, grid, NT, smem, s, b, lut, map, gmap, with_graph ? 1 : 0);
        }
    }
    size_t smem = mask_smem<S, 32, TH>(b.scale);
    if (smem + sizeof(MaskTile<S, 32, TH>) > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_mask_raster<LAYOUT, S, TH, NT>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    dim3 grid((b.w + 32 - 1) / 32, (b.h + TH - 1) / TH, nframes);
    return launch_early(early, k_mask_raster<LAYOUT, S, TH, NT>, grid, NT, smem, s, b, lut);
}

// With so few tiles that all are resident at once with twice the threads (two
// blocks per SM up to x4, one above), a tile's time is the call's, and the
// threads shorten it: a call with labels at x4 takes 26.7 us instead of 28.7 for
// a 256x224 frame (112 tiles), 34.6 instead of 37.7 for five (280), but 44.2
// instead of 43.2 for six (336); at x8 29.9 instead of 32.9 for one (112), 38.9
// instead of 36.3 for two (224). 1024 threads: no better than 512 for one frame,
// worse from four on.
template <int S>
constexpr int kFewTilesPerSm = raster_blocks(S) / 2;

template <int LAYOUT, int S, int TH>
static cudaError_t launch_mask_raster_t(const RasterBatch& b, int nframes, const uint32_t* lut, cudaStream_t s)
{
    const long long tiles = (long long)((b.w + 31) / 32) * ((b.h + TH - 1) / TH) * nframes;
    return tiles <= (long long)kFewTilesPerSm<S> * sm_count() ? launch_mask_raster_nt<LAYOUT, S, TH, 2 * kRT>(b, nframes, lut, s)
                                 : launch_mask_raster_nt<LAYOUT, S, TH, kRT>(b, nframes, lut, s);
}

// ---- uneven batches: the raster as a persistent kernel over a tile queue

template <int S, int TW, int TH>
__global__ void __launch_bounds__(kRT, raster_blocks(S)) k_raster_queue(QueueBatch q)
{
    __shared__ MaskTile<S, TW, TH> M;
    extern __shared__ uint32_t masks[];
    const QueueHeader* H = q.hdr;
    const int n = H->n;
    constexpr int SH = raster_shape_index(TW, TH);
    const int P = q.rbase + SH;
    queue_loop(q.counters + QC_RASTER + SH, (int)H->total[P], q.gran[QS_RASTER], [&](int t) {
        const uint32_t* base = H->base + P * (n + 1);
        const int f = queue_frame(base, n, (uint32_t)t);
        const QueueFrame fr = H->frames[f];
        const int lt = t - (int)base[f], tx = (fr.w + TW - 1) / TW;
        mask_raster_tile<DEPIX_LAYOUT_RGBA, S, TW, TH>(M, masks, H->img + fr.in_off, 4 * fr.w, q.graph_b + fr.px_off,
                                                       H->out + fr.out_off, fr.w, fr.h, q.scale, H->subdivide != 0,
                                                       q.lut, (lt % tx) * TW, (lt / tx) * TH,
                                                       H->labels ? H->labels + fr.px_off : nullptr);
    });
}

template <int S, int TW, int TH>
static cudaError_t queue_raster_t(const QueueBatch& q, int blocks, cudaStream_t s)
{
    // the shared-memory opt-in is made by raster_queue_occupancy, which the
    // host calls on each device before any launch or stream capture
    const size_t smem = mask_smem<S, TW, TH>(q.scale);
    k_raster_queue<S, TW, TH><<<blocks, kRT, smem, s>>>(q);
    return cudaGetLastError();
}

template <int S, int TW, int TH>
static int raster_queue_occupancy(int scale)
{
    int nb = 0;
    const size_t smem = mask_smem<S, TW, TH>(scale);
    if (smem + sizeof(MaskTile<S, TW, TH>) > 48 * 1024 &&
        cudaFuncSetAttribute(k_raster_queue<S, TW, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
        return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_raster_queue<S, TW, TH>, kRT, smem) != cudaSuccess)
        return 0;
    return nb;
}

// raster tile variants of the queue path: 32x32, 32x16, 16x16 cells
#define DEPIX_RQ_SCALES(FN, TW, TH, ...)                                                                \
    switch (raster_mode(q.scale)) {                                                                     \
    case 1: return FN<1, TW, TH>(__VA_ARGS__);                                                          \
    case 2: return FN<2, TW, TH>(__VA_ARGS__);                                                          \
    case 3: return FN<3, TW, TH>(__VA_ARGS__);                                                          \
    case 4: return FN<4, TW, TH>(__VA_ARGS__);                                                          \
    case 8: return FN<8, TW, TH>(__VA_ARGS__);                                                          \
    case 0: return FN<0, TW, TH>(__VA_ARGS__);                                                          \
    default: return FN<-1, TW, TH>(__VA_ARGS__);                                                        \
    }
#define DEPIX_RQ_DISPATCH(FN, ...)                                                                      \
    do {                                                                                                \
        if (q.rtw == 32 && q.rth == 32) DEPIX_RQ_SCALES(FN, 32, 32, __VA_ARGS__)                        \
        if (q.rtw == 32) DEPIX_RQ_SCALES(FN, 32, 16, __VA_ARGS__)                                       \
        DEPIX_RQ_SCALES(FN, 16, 16, __VA_ARGS__)                                                        \
    } while (0)

cudaError_t queue_raster(const QueueBatch& q, int blocks, cudaStream_t s)
{
    DEPIX_RQ_DISPATCH(queue_raster_t, q, blocks, s);
}

int queue_raster_blocks_per_sm(const QueueBatch& q) { DEPIX_RQ_DISPATCH(raster_queue_occupancy, q.scale); }

// 32x32-cell tiles up to scale 4 (more subdivided cells per block to share
// the work), 32x16 above (the footprint masks grow with the scale)
// A single frame fills a fraction of the SMs, so it takes tiles half as high
// at x4 (twice the blocks, each half as long); batches keep the 32-row tiles.
template <int LAYOUT>
static cudaError_t launch_mask_raster_l(const RasterBatch& b, int nframes, const uint32_t* lut, cudaStream_t s)
{
    switch (raster_mode(b.scale)) {
    case 1: return launch_mask_raster_t<LAYOUT, 1, 32>(b, nframes, lut, s);
    case 2: return launch_mask_raster_t<LAYOUT, 2, 32>(b, nframes, lut, s);
    case 3: return launch_mask_raster_t<LAYOUT, 3, 32>(b, nframes, lut, s);
    case 4:
        return nframes == 1 ? launch_mask_raster_t<LAYOUT, 4, 16>(b, nframes, lut, s)
                            : launch_mask_raster_t<LAYOUT, 4, 32>(b, nframes, lut, s);
    case 8: return launch_mask_raster_t<LAYOUT, 8, 16>(b, nframes, lut, s);
    case 0: return launch_mask_raster_t<LAYOUT, 0, 16>(b, nframes, lut, s);
    default: return launch_mask_raster_t<LAYOUT, -1, 16>(b, nframes, lut, s);
    }
}

cudaError_t launch_mask_raster(const RasterBatch& b, int nframes, const uint32_t* lut, cudaStream_t s)
{
    return b.layout == DEPIX_LAYOUT_RGBA ? launch_mask_raster_l<DEPIX_LAYOUT_RGBA>(b, nframes, lut, s)
                                         : launch_mask_raster_l<DEPIX_LAYOUT_BGR>(b, nframes, lut, s);
}

cudaError_t take_raster_fault(int* out)
{
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_raster_fault, sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_raster_fault, &zero, sizeof(int));
    return e;
}

}  // namespace depix
