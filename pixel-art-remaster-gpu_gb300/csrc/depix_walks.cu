// depix_walks.cu -- border walks of the resolved graph's components, the
// input of the reference's spline export (extractBorderPoints,
// cc_functions.cu:348-503; recorded output alex_png.txt).
//
// The walks of one frame depend on each other in scan order (a node listed
// by one walk starts none; a walk that runs into a listed or discarded node
// is dropped and discards a node), so a frame is one thread's sequential
// loop. Lanes of one warp would run their frames' walks in lockstep, each
// waiting for the longest, so a batch runs one frame per warp. A frame that
// fits keeps its graph and node state (two bitmaps) in shared memory; larger
// frames read the graph from global memory and keep a state byte per node in a
// caller-provided scratch (the lanes find the walks' start nodes by ballot and
// lane 0 walks).
#include "depix_internal.h"

namespace depix {

// The reference enumerates a node's links clockwise from up-left (clock
// positions 0..7) and maps them to node bits and back (getRealLinkIndex /
// getClockLinkIndex, cc_functions.cu:48-100, 127-183), packed as nibbles.
__device__ __forceinline__ int real_of_clock(int c) { return (int)((0x35674210u >> (4 * (c & 7))) & 0xFu); }
__device__ __forceinline__ int clock_of_real(int r) { return (int)((0x45637210u >> (4 * r)) & 0xFu); }

// getFirstLink (cc_functions.cu:107-119)
__device__ __forceinline__ int walk_first_link(unsigned v)
{
    for (int c = 0; c < 8; c++)
        if ((v >> real_of_clock(c)) & 1u) return real_of_clock(c);
    return -1;
}

// nextEdgeCounterClockwise (cc_functions.cu:265-287)
__device__ __forceinline__ int walk_next_ccw(unsigned v, int e)
{
    if (__popc(v) == 1) return e;
    const int c = clock_of_real(e);
    for (int k = c + 7; k >= c + 1; k--)
        if ((v >> real_of_clock(k)) & 1u) return real_of_clock(k);
    return e;
}

// the link a walk leaves a node of links v by after arriving along e
// (nextNodeClockwise, cc_functions.cu:296-318); the link back on a valence-1
// node, and (not in the reference) on a node without links
__device__ __forceinline__ int walk_next_cw(unsigned v, int e)
{
    const int back = 7 - e;
    if (__popc(v) == 1) return back;
    const int c = clock_of_real(back);
    for (int k = c + 1; k <= c + 7; k++)
        if ((v >> real_of_clock(k)) & 1u) return real_of_clock(k);
    return back;
}

// Walk k of frame f: nodes[f * max_nodes + offsets[k] .. + offsets[k + 1]),
// offsets at offsets + f * (max_walks + 1); counts[3 f ..]: walks, nodes, 1
// when a capacity ran out (outputs up to the last complete walk). The rules
// are those of orc_border_walks in the oracle: scan order, internal (90) and
// listed nodes start none, a node without links is a walk of its own, a walk
// is dropped when it enters an internal, listed or discarded node (its last
// node discarded, its start unlisted) or passes 8 w h + 8 steps.
// Node state of one frame: bit 0 listed, bit 1 discarded.
struct ByteState { // a byte per node (global scratch)
    uint8_t* s;
    __device__ __forceinline__ unsigned get(int p) const { return s[p]; }
    __device__ __forceinline__ void set(int p, unsigned b) const { s[p] |= (uint8_t)b; }
    __device__ __forceinline__ void clear(int p, unsigned b) const { s[p] &= (uint8_t)~b; }
};
// walk_next_cw for every node byte v and arrival link e, at [v * 8 + e]
__device__ __forceinline__ void build_cw_table(uint8_t* cw, int tid, int nthreads)
{
    for (int i = tid; i < 256 * 8; i += nthreads) cw[i] = (uint8_t)walk_next_cw((unsigned)(i >> 3), i & 7);
}

// The walks of one frame, by one warp: the lanes find the nodes that can
// start a walk (not internal) 32 at a time by ballot, lane 0 walks from each
// in scan order (re-checking the state, which its walks change). cw: the
// walk_next_cw table.
template <typename State>
__device__ void walk_frame(const uint8_t* g, int w, int h, State fl, const uint8_t* cw, int32_t* on, int8_t* oe,
                           int32_t* oo, int max_nodes, int max_walks, int32_t* cnt)
{
    const int lane = threadIdx.x & 31;
    const long long limit = 8LL * (long long)w * h + 8;
    auto node = [&](int x, int y) -> unsigned { return g[(size_t)y * w + x] & inside_mask(x, y, w, h); };
    int nw = 0, pos = 0, trunc = 0; // lane 0's
    if (lane == 0) oo[0] = 0;
    for (int y = 0; y < h && !trunc; y++)
        for (int x0 = 0; x0 < w && !trunc; x0 += 32) {
            const int xl = x0 + lane;
            unsigned cand = __ballot_sync(0xFFFFFFFFu, xl < w && node(xl, y) != 90);
            if (lane == 0) {
                while (cand) {
                    const int x = x0 + __ffs(cand) - 1;
                    cand &= cand - 1;
                    const int p = y * w + x;
                    const unsigned v0 = node(x, y);
                    if (fl.get(p) & 1u) continue;
                    if (v0 == 0) {
                        if (nw >= max_walks || pos >= max_nodes) {
                            trunc = 1;
                            break;
                        }
                        on[pos] = p;
                        oe[pos++] = -1;
                        fl.set(p, 1u);
                        oo[++nw] = pos;
                        continue;
                    }
                    fl.set(p, 1u);
                    int e = walk_first_link(v0);
                    const int arr = walk_next_ccw(v0, e);
                    const int start = pos;
                    int over = 0, last = p; // over: a node did not fit (the walk is then not recorded)
                    if (pos < max_nodes) {
                        on[pos] = p;
                        oe[pos++] = (int8_t)e;
                    } else {
                        over = 1;
                    }
                    int cx = x, cy = y, ok = 1;
                    long long steps = 0;
                    while (!(cx + dir_di(e) == x && cy + dir_dj(e) == y && 7 - e == arr)) {
                        cx += dir_di(e);
                        cy += dir_dj(e);
                        const int cp = cy * w + cx;
                        const unsigned v = node(cx, cy);
                        e = cw[v * 8 + e];
                        if (v == 90 || fl.get(cp) || ++steps > limit) {
                            fl.set(last, 2u);
                            fl.clear(p, 1u);
                            pos = start;
                            ok = 0;
                            break;
                        }
                        last = cp;
                        if (pos < max_nodes) {
                            on[pos] = cp;
                            oe[pos++] = (int8_t)e;
                        } else {
                            over = 1;
                        }
                    }
                    if (ok) {
                        if (over || nw >= max_walks) {
                            pos = start;
                            trunc = 1;
                            break;
                        }
                        for (int q = start; q < pos; q++) fl.set(on[q], 1u);
                        oo[++nw] = pos;
                    }
                }
            }
            trunc = __shfl_sync(0xFFFFFFFFu, trunc, 0);
        }
    if (lane == 0) {
        cnt[0] = nw;
        cnt[1] = pos;
        cnt[2] = trunc;
    }
}

// Frames whose graph (w h bytes) and node state (bitmaps) fit in shared
// memory, one per block: all threads load, the first warp walks, every lane
// the same walk (so that no lane waits for another's answer).
//
// Most steps are those of dropped walks: 48 of the 60 thousand steps of a mean
// 256x224 frame, four in five (181 of 190 in the worst of 128), because the
// starts along one border run into the same obstacle one after the other, each
// discarding the node before it. A path does not depend on the state, which only ends it, so
// the nodes and links of dropped walks stay in a log, and each node knows where
// in the log its first link leaves it. A walk that starts there reads its path
// from the log, 32 nodes at a time, up to the first one that is blocked by now;
// the log's walk ends in a discarded node at the latest. That leaves 15
// thousand steps a frame (17 in the worst), 12 of them of recorded walks.
//
// Bound: one dependent chain. A step is two dependent shared-memory loads, the
// node's byte, then the table that gives for (byte, arrival link) the next link
// and its offset; the state is read beside the first and the walk's branch
// resolves while the second is under way. 128 frames of 256x224: 24.6 ms when a
// step turned coordinates into an index, tested the state in packed fields and
// looked the link and its offset up apart, 15.8 without the log, 3.5 now.
constexpr int kWalkThreads = 128;

// Next-link table entries: link in bits 0-2, then its offset in the frame
// (biased to be non-negative in 16 bits)
template <typename T>
struct WalkTable {
    static constexpr int kBias = sizeof(T) == 2 ? 4095 : 0; // offsets up to w + 1
    static constexpr int kMaxW = sizeof(T) == 2 ? 4094 : 1 << 26;
    static __device__ __forceinline__ T pack(int e, int w) { return (T)(e | (dir_dj(e) * w + dir_di(e) + kBias) * 8); }
    static __device__ __forceinline__ int link(T t) { return (int)t & 7; }
    static __device__ __forceinline__ int offset(T t) { return ((int)t >> 3) - kBias; }
};

// Shared memory of a frame of n nodes: its bytes, the bitmaps (32 nodes a
// word), the table, the log and, when paths are kept, where each node that can
// start a walk leaves in it.
constexpr int kWalkStage = 256; // log entries that the walk under way can always use
struct WalkSizes {
    int n, words, log_cap, index_cap; // index_cap 0: no paths are kept
    size_t bytes;
};
template <typename T>
static WalkSizes walk_sizes(size_t n, size_t most)
{
    WalkSizes z{(int)n, (int)((n + 31) / 32), kWalkStage, 0, 0};
    const size_t plain = 32 * (size_t)z.words + 2 * 4 * (size_t)z.words + 256 * 8 * sizeof(T) + 4 * kWalkStage;
    const size_t extra = 2 * 4 * (size_t)z.words; // bitmap and rank of the nodes that can start
    z.bytes = plain;
    if (plain + extra + 8 * 1024 <= most) {
        // a third of the nodes start walks or fewer, half as many log entries
        const size_t left = most - plain - extra;
        const size_t keep = n / 6 < left / 8 ? n / 6 : left / 8;
        z.log_cap += (int)keep;
        z.index_cap = (int)(2 * keep);
        z.bytes += extra + 8 * keep;
    }
    return z;
}

template <typename T>
__global__ void __launch_bounds__(kWalkThreads) k_border_walks_smem(const uint8_t* graph, int w, int h, WalkSizes z,
                                                                    int32_t* nodes, int8_t* edges, int32_t* offsets,
                                                                    int max_nodes, int max_walks, int32_t* counts)
{
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ uint8_t first[256]; // per node byte: first link | the link that closes the walk << 4
    const int n = z.n, words = z.words;
    uint32_t* blocked = reinterpret_cast<uint32_t*>(sm + 32 * words); // internal, listed or discarded
    uint32_t* done = blocked + words;                                 // internal or listed: starts no walk
    T* next = reinterpret_cast<T*>(done + words);
    uint32_t* log = reinterpret_cast<uint32_t*>(next + 256 * 8); // node << 3 | link it is left by
    uint32_t* starts = log + z.log_cap;  // not internal
    uint32_t* rank = starts + words;     // of them before the word
    uint16_t* index = reinterpret_cast<uint16_t*>(rank + words); // per start node, by rank: its place in the log
    constexpr unsigned kNone = 0xFFFFu;
    const size_t f = blockIdx.x;
    const uint8_t* g = graph + (size_t)n * f;
    // ---- load
    if (((reinterpret_cast<uintptr_t>(g) | (unsigned)n) & 15) == 0) {
        for (int i = threadIdx.x; i < n / 16; i += kWalkThreads)
            reinterpret_cast<uint4*>(sm)[i] = __ldg(reinterpret_cast<const uint4*>(g) + i);
    } else {
        for (int i = threadIdx.x; i < n; i += kWalkThreads) sm[i] = __ldg(g + i);
    }
    for (int i = threadIdx.x; i < 256 * 8; i += kWalkThreads)
        next[i] = WalkTable<T>::pack(walk_next_cw((unsigned)(i >> 3), i & 7), w);
    for (int v = threadIdx.x; v < 256; v += kWalkThreads) {
        const int e = v ? walk_first_link((unsigned)v) : 0;
        first[v] = (uint8_t)(e | (v ? 7 - walk_next_ccw((unsigned)v, e) : 0) << 4);
    }
    for (int i = threadIdx.x; i < z.index_cap; i += kWalkThreads) index[i] = (uint16_t)kNone;
    __syncthreads();
    // links toward outside the image
    for (int x = threadIdx.x; x < w; x += kWalkThreads) {
        if (h > 1) sm[x] &= (uint8_t)inside_mask(x, 0, w, h);
        sm[(h - 1) * w + x] &= (uint8_t)inside_mask(x, h - 1, w, h);
    }
    __syncthreads();
    for (int y = threadIdx.x; y < h; y += kWalkThreads) {
        sm[y * w] &= (uint8_t)inside_mask(0, y, w, h);
        sm[y * w + w - 1] &= (uint8_t)inside_mask(w - 1, y, w, h);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < words; k += kWalkThreads / 32) {
        const int p = 32 * k + lane;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, p >= n || sm[p] == 90);
        if (lane == 0) {
            blocked[k] = done[k] = m;
            if (z.index_cap) starts[k] = ~m;
        }
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    if (z.index_cap) {
        uint32_t sum = 0;
        for (int k0 = 0; k0 < words; k0 += 32) {
            const uint32_t c = k0 + lane < words ? __popc(starts[k0 + lane]) : 0;
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            if (k0 + lane < words) rank[k0 + lane] = sum + x - c;
            sum += __shfl_sync(0xFFFFFFFFu, x, 31);
        }
        __syncwarp();
    }
    auto slot_of = [&](int p) -> int { // of a start node; index_cap or more: none
        return (int)(rank[p >> 5] + __popc(starts[p >> 5] & ((1u << (p & 31)) - 1u)));
    };
    // ---- walk
    const long long limit = 8LL * n + 8;
    int32_t* on = nodes + (size_t)max_nodes * f;
    int8_t* oe = edges + (size_t)max_nodes * f;
    int32_t* oo = offsets + (size_t)(max_walks + 1) * f;
    int nw = 0, pos = 0, trunc = 0, nlog = 0; // log entries kept
    // log entries [a, b) to the outputs from o on, as far as these reach (a
    // dropped walk's too: behind the recorded ones they mean nothing)
    auto put = [&](int a, int b, int o) {
        for (int j = a + lane; j < b && o + j - a < max_nodes; j += 32) {
            on[o + j - a] = (int)(log[j] >> 3);
            oe[o + j - a] = (int8_t)(log[j] & 7u);
        }
    };
    if (lane == 0) oo[0] = 0;
    for (int k = 0; k < words && !trunc; k++) {
        for (unsigned cand = ~done[k]; cand;) {
            const int p = 32 * k + __ffs(cand) - 1;
            const unsigned bit = cand & (0u - cand), above = ~(bit | (bit - 1u));
            const unsigned v0 = sm[p];
            if (v0 == 0) { // a walk of its own
                if (nw >= max_walks || pos >= max_nodes) {
                    trunc = 1;
                    break;
                }
                __syncwarp(); // every lane has read done[k]
                if (lane == 0) {
                    on[pos] = p;
                    oe[pos] = -1;
                    oo[nw + 1] = pos + 1;
                    blocked[k] |= bit;
                    done[k] |= bit;
                }
                nw++;
                pos++;
                __syncwarp();
                cand = ~done[k] & above;
                continue;
            }
            const unsigned was = blocked[k];
            const int f0 = first[v0];
            const int closing = p * 8 + (f0 >> 4); // entering the start along this link
            int slot = -1, at = (int)kNone;
            if (z.index_cap) {
                slot = slot_of(p);
                if (slot < z.index_cap) at = index[slot];
            }
            __syncwarp();
            if (lane == 0) blocked[k] = was | bit;
            __syncwarp();
            bool ok;
            int len, last = p; // nodes of the walk, its last one
            if (at != (int)kNone) {
                // the path from the log: entries at, at + 1, ... up to a blocked
                // one (the logged walk's last node is) or the closing link
                int j0 = at + 1;
                for (;; j0 += 32) {
                    const int j = j0 + lane;
                    const uint32_t d = j < nlog ? log[j] : 0u, before = j < nlog ? log[j - 1] : 0u;
                    const int c = (int)(d >> 3);
                    const bool close = j < nlog && c * 8 + (int)(before & 7u) == closing;
                    const bool stop = j >= nlog || close || (blocked[c >> 5] >> (c & 31) & 1u);
                    const unsigned m = __ballot_sync(0xFFFFFFFFu, stop);
                    if (m) {
                        const int q = __ffs(m) - 1;
                        ok = __shfl_sync(0xFFFFFFFFu, (int)close, q) != 0;
                        len = j0 + q - at;
                        break;
                    }
                }
                last = (int)(log[at + len - 1] >> 3);
                put(at, at + len, pos);
            } else {
                int e = f0 & 7, m = nlog; // end of the log's entries for this walk
                int cp = p + dir_dj(e) * w + dir_di(e), flushed = 0;
                ok = true;
                if (lane == 0) log[m] = (uint32_t)(p * 8 + e);
                m++;
                long long steps = 0;
                while (cp * 8 + e != closing) {
                    const unsigned v = sm[cp];
                    const unsigned b = blocked[cp >> 5];
                    const T t = next[v * 8 + e];
                    if ((b >> (cp & 31) & 1u) || ++steps > limit) {
                        ok = false;
                        break;
                    }
                    e = WalkTable<T>::link(t);
                    if (m == z.log_cap) { // full: what there is goes out, the path is not kept
                        __syncwarp();
                        put(nlog, m, pos + flushed);
                        flushed += m - nlog;
                        m = nlog;
                        __syncwarp();
                    }
                    if (lane == 0) log[m] = (uint32_t)(cp * 8 + e);
                    m++;
                    last = cp;
                    cp += WalkTable<T>::offset(t);
                }
                __syncwarp();
                put(nlog, m, pos + flushed);
                len = flushed + m - nlog;
                if (!ok && z.index_cap && flushed == 0 && m + kWalkStage <= z.log_cap) {
                    // kept; the last node, discarded now, may start a walk over
                    // an end that is no longer blocked (the walk's own start)
                    for (int j = nlog + lane; j < m - 1; j += 32) {
                        const int c = (int)(log[j] >> 3);
                        const int sl = slot_of(c);
                        if ((int)(log[j] & 7u) == (first[sm[c]] & 7) && sl < z.index_cap && index[sl] == kNone)
                            index[sl] = (uint16_t)j;
                    }
                    nlog = m;
                }
            }
            __syncwarp();
            if (!ok) {
                // dropped: its last node discarded, its start as it was
                if (lane == 0) {
                    if (!(was & bit)) blocked[k] &= ~bit;
                    blocked[last >> 5] |= 1u << (last & 31);
                }
            } else if (pos + len > max_nodes || nw >= max_walks) {
                trunc = 1;
                break;
            } else {
                // recorded: its nodes are listed
                for (int q = pos + lane; q < pos + len; q += 32) {
                    const int c = on[q];
                    atomicOr(&blocked[c >> 5], 1u << (c & 31));
                    atomicOr(&done[c >> 5], 1u << (c & 31));
                }
                pos += len;
                nw++;
                if (lane == 0) oo[nw] = pos;
            }
            __syncwarp();
            cand = ~done[k] & above;
        }
    }
    if (lane == 0) {
        counts[3 * f] = nw;
        counts[3 * f + 1] = pos;
        counts[3 * f + 2] = trunc;
    }
}

// larger frames: the graph from global memory, the state in the scratch; a
// warp per frame, four per block
__global__ void __launch_bounds__(128) k_border_walks(const uint8_t* graph, int w, int h, int nframes, uint8_t* flags,
                                                      int32_t* nodes, int8_t* edges, int32_t* offsets, int max_nodes,
                                                      int max_walks, int32_t* counts)
{
    __shared__ uint8_t cw[256 * 8];
    build_cw_table(cw, threadIdx.x, blockDim.x);
    __syncthreads();
    const int f = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (f >= nframes) return; // whole warps
    const size_t n = (size_t)w * h;
    walk_frame(graph + n * f, w, h, ByteState{flags + n * f}, cw, nodes + (size_t)max_nodes * f,
               edges + (size_t)max_nodes * f, offsets + (size_t)(max_walks + 1) * f, max_nodes, max_walks,
               counts + 3 * f);
}

constexpr size_t kWalkSmemMax = 224 * 1024;

template <typename T>
static cudaError_t launch_walks_smem(const uint8_t* graph, int w, int h, const WalkSizes& z, int nframes, int32_t* nodes,
                                     int8_t* edges, int32_t* offsets, int max_nodes, int max_walks, int32_t* counts,
                                     cudaStream_t s)
{
    cudaError_t e = cudaFuncSetAttribute(k_border_walks_smem<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kWalkSmemMax);
    if (e != cudaSuccess) return e;
    k_border_walks_smem<T><<<nframes, kWalkThreads, z.bytes, s>>>(graph, w, h, z, nodes, edges, offsets, max_nodes,
                                                                  max_walks, counts);
    return cudaGetLastError();
}

// frames wider than the 16-bit table's offsets take the 32-bit one
cudaError_t launch_border_walks(const uint8_t* graph, int w, int h, int nframes, uint8_t* flags, int32_t* nodes,
                                int8_t* edges, int32_t* offsets, int max_nodes, int max_walks, int32_t* counts,
                                cudaStream_t s)
{
    const size_t n = (size_t)w * h;
    if (n <= kWalkSmemMax) {
        const bool narrow = w <= WalkTable<uint16_t>::kMaxW;
        const WalkSizes z = narrow ? walk_sizes<uint16_t>(n, kWalkSmemMax) : walk_sizes<int32_t>(n, kWalkSmemMax);
        if (z.bytes <= kWalkSmemMax)
            return narrow ? launch_walks_smem<uint16_t>(graph, w, h, z, nframes, nodes, edges, offsets, max_nodes,
                                                        max_walks, counts, s)
                          : launch_walks_smem<int32_t>(graph, w, h, z, nframes, nodes, edges, offsets, max_nodes,
                                                       max_walks, counts, s);
    }
    cudaError_t e = cudaMemsetAsync(flags, 0, n * nframes, s);
    if (e != cudaSuccess) return e;
    k_border_walks<<<(nframes + 3) / 4, 128, 0, s>>>(graph, w, h, nframes, flags, nodes, edges, offsets, max_nodes,
                                                      max_walks, counts);
    return cudaGetLastError();
}

}  // namespace depix
