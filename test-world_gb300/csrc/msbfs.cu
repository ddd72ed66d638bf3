// msbfs.cu - fused multi-source BFS and SSSP over 64-bit source masks.
//
// The reference answers one source per call (bfsCaculateIn*/ssspCaculateIn*,
// ptGraph/main.cu:24-44); a batch of sources there is a loop of full calls
// (testBFS, main.cu:537-556).  Here one traversal serves many sources:
//
// MS-BFS (after Then et al., "The More the Merrier"): per vertex W 64-bit
//   words of frontier mask F[v] (which of up to 64*W sources reached v in the
//   last level) and seen mask S[v].  A level either pushes (active vertices OR
//   their F into the next masks of their neighbours, load-balanced over the
//   frontier's edges like the single-source expand) or, when the frontier's
//   edges are a large share of the graph and the graph is symmetric, pulls
//   (every vertex ORs its neighbours' F, stopping once all sources saw it).
//   With W = 4 one 32-byte sector read per edge serves 256 sources.  The
//   levels' frontier masks are kept, and the result rows written from them once.
// MS-SSSP: distances stored vertex-major, dist[v*64 + s], so the 64 distances
//   of a vertex are two 128-byte lines; a warp relaxes one edge for 64
//   sources at once (lane l handles sources 2l and 2l+1).  A vertex is active
//   while some source improved it in the previous round (a 64-bit mask);
//   an edge is looked at only if bounds on all 64 distances of its ends let it
//   improve one (k_mss_queue).  Rounds push, or pull when many edges are active
//   and weights are the same both ways, until no mask is set.
// Results equal k single-source calls (tests compare them row by row).
#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

#include "frontier.cuh"

namespace ptg {
namespace {

typedef unsigned long long u64;

// ---------------------------------------------------------------------------
// MS-BFS, W mask words per vertex (layout M[v*W + w])
// ---------------------------------------------------------------------------
template <int W>
__global__ void k_msb_seed(const uint32_t *srcs, uint32_t k, u64 *F, u64 *S) {
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
        uint32_t s = srcs[i];
        atomicOr(&F[(uint64_t)s * W + i / 64], 1ull << (i % 64));
        atomicOr(&S[(uint64_t)s * W + i / 64], 1ull << (i % 64));
    }
}

// Queue of vertices with a non-zero mask, and the sum of their degrees
// (ctl->m_unvisited) for the push/pull choice.
template <class OffT, int W>
__global__ void __launch_bounds__(kBlock) k_msb_queue(const u64 *M, uint64_t n, const OffT *off, uint32_t *q,
                                                      TravCtl *ctl) {
    unsigned long long degsum = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        bool act = false;
#pragma unroll
        for (int w = 0; w < W; w++) act |= M[v * W + w] != 0ull;
        if (act) {
            degsum += (unsigned long long)(off[v + 1] - off[v]);
            warp_append(q, &ctl->next_tail, (unsigned)n, &ctl->error, (uint32_t)v);
        }
    }
    degsum = block_reduce_sum(degsum);
    if (threadIdx.x == 0 && degsum) atomicAdd(&ctl->m_unvisited, degsum);
}

// Push level: every edge (u -> v) of the frontier ORs F[u] into N[v].
template <class OffT, int W>
__global__ void __launch_bounds__(kBlock) k_msb_push(const uint32_t *q, const OffT *sc, const OffT *rs,
                                                     const uint32_t *tr, const uint32_t *col, const u64 *F,
                                                     const u64 *S, u64 *N, const TravCtl *ctl) {
    __shared__ OffT s_sc[kTile + 2];
    __shared__ OffT s_rs[kTile + 2];
    __shared__ uint32_t s_u[kTile + 2];
    uint64_t E = ctl->E;
    uint64_t ntiles = (E + kTile - 1) / kTile;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint64_t t0 = tile * kTile, t1 = min(E, t0 + kTile);
        uint64_t r0 = tr[tile];
        uint32_t nrows = (uint32_t)((uint64_t)tr[tile + 1] - r0 + 1);
        bool staged = nrows <= (uint32_t)kTile + 1;
        if (staged) {
            for (uint32_t k = threadIdx.x; k <= nrows; k += kBlock) {
                s_sc[k] = sc[r0 + k];
                if (k < nrows) {
                    s_rs[k] = rs[r0 + k];
                    s_u[k] = q[r0 + k];
                }
            }
        }
        __syncthreads();
        for (uint64_t j = t0 + threadIdx.x; j < t1; j += kBlock) {
            uint64_t row = staged ? last_le(s_sc, 0, nrows, j) : last_le(sc, r0, r0 + nrows, j);
            OffT rsv = staged ? s_rs[row] : rs[row];
            OffT scv = staged ? s_sc[row] : sc[row];
            uint32_t u = staged ? s_u[row] : q[row];
            uint32_t v = __ldcs(col + (uint64_t)rsv + (j - (uint64_t)scv));
#pragma unroll
            for (int w = 0; w < W; w++) {
                u64 add = F[(uint64_t)u * W + w] & ~S[(uint64_t)v * W + w];
                if (add) atomicOr(&N[(uint64_t)v * W + w], add);
            }
        }
        __syncthreads();
    }
}

// Load a vertex's W mask words (16-byte vector loads for W >= 2).
template <int W>
__device__ __forceinline__ void load_mask(const u64 *p, u64 (&x)[W]) {
    if constexpr (W == 1) {
        x[0] = p[0];
    } else if constexpr (W == 2) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p);
        x[0] = t.x;
        x[1] = t.y;
    } else {
        // one 32-byte load: two of 16 bytes ask L1 for the sector twice, and a
        // gather of masks is bound by how many it can be asked for
        static_assert(W == 4);
        asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
                     : "l"(p)
                     : "memory");
    }
}

// OR the warp's new masks into the next level's live-source mask.
template <int W>
__device__ __forceinline__ void live_or(u64 *live_next, const u64 (&nb)[W]) {
#pragma unroll
    for (int w = 0; w < W; w++) {
        u64 x = nb[w];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x |= __shfl_xor_sync(0xffffffffu, x, o);
        if (lane_id() == 0 && x) atomicOr(&live_next[w], x);
    }
}

// After a level: N[v] &= ~S[v], S |= N, next queue built.
template <class OffT, int W>
__global__ void __launch_bounds__(kBlock) k_msb_update(uint64_t n, const OffT *off, u64 *N, u64 *S, uint32_t *q,
                                                       TravCtl *ctl, u64 *live_next) {
    unsigned long long degsum = 0;
    u64 live[W];
#pragma unroll
    for (int w = 0; w < W; w++) live[w] = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        u64 x[W];
        load_mask<W>(N + v * W, x);
        bool any = false;
#pragma unroll
        for (int w = 0; w < W; w++) any |= x[w] != 0ull;
        if (!any) continue;
        u64 s[W];
        load_mask<W>(S + v * W, s);
        any = false;
#pragma unroll
        for (int w = 0; w < W; w++) {
            const u64 nb = x[w] & ~s[w];
            if (nb != x[w]) N[v * W + w] = nb;
            if (nb) S[v * W + w] = s[w] | nb;
            live[w] |= nb;
            any |= nb != 0ull;
        }
        if (any) {
            degsum += (unsigned long long)(off[v + 1] - off[v]);
            warp_append(q, &ctl->next_tail, (unsigned)n, &ctl->error, (uint32_t)v);
        }
    }
    __syncwarp();
    live_or<W>(live_next, live);
    degsum = block_reduce_sum(degsum);
    if (threadIdx.x == 0 && degsum) atomicAdd(&ctl->m_unvisited, degsum);
}

// The frontier masks of up to kMsHist consecutive levels.
constexpr int kMsHist = 12;
static_assert(kMsHist <= 16, "a level's position has four bits");
struct MsHist {
    const u64 *m[kMsHist];
};

// Room for the frontier masks of consecutive levels in ws.ms[0]; returns how many.
// Fewer than kMsHist only cost further passes over the rows, so the masks past
// the two that a level needs take at most a quarter of the free memory (or the
// room that a server gives its lane); up to a 64th of the device's memory they
// are taken without asking.
int ms_history(ptg_ctx *ctx, uint64_t mask_bytes) {
    DevBuf &b = ctx->ws.ms[0];
    uint64_t room = ctx->mask_room;
    if (room == ~0ull && b.bytes < kMsHist * mask_bytes && kMsHist * mask_bytes > ctx->hbm_bytes / 64) {
        size_t dfree = 0, total = 0;
        PTG_CUDA_TRY(device_free_bytes(ctx->device, &dfree, &total));
        room = (dfree + b.bytes) / 4;
    } else if (room != ~0ull && b.bytes > 2 * mask_bytes + room + room / 8 + (8ull << 20)) {
        b.release();  // a server whose budget has shrunk
    }
    int hist = (int)std::min<uint64_t>(kMsHist, 2 + room / mask_bytes);
    while (true) {
        try {
            b.ensure(hist * mask_bytes);
            return hist;
        } catch (const Error &e) {
            if (e.status != PTG_ERR_OOM || hist == 2) throw;
            cudaGetLastError();
            hist = std::max(2, hist / 2);
        }
    }
}

// Rows out of the kept levels: out[s*n + v] = level0 + l for the level l whose
// mask holds source s at v (at newid[v] on a regrouped graph).  FIRST: every
// word is written, unreached where no level has it; else only the found ones.
// The position of a source's level is put together from four words of bits
// (levels with bit 0..3 of their position set), so a source takes a few
// instructions a vertex however many levels there are.  Bound by the rows'
// stores: 4.3 GB in 1.0 ms for 256 sources on 4.2 M vertices.  The rows are
// written once: writing them level by level (a fill, scattered words per
// level, then a gather to the caller's ids) moved them five times and took
// 5.7 of that call's 8.8 ms (now 3.6).  Twelve levels are what an RMAT search
// needs (9-10); with eight the second pass over the rows cost another 0.1 ms.
template <int W, bool FIRST>
__global__ void __launch_bounds__(kBlock) k_msb_levels(MsHist h, int cnt, uint64_t n, uint32_t k,
                                                       const uint32_t *newid, uint32_t level0, uint32_t *out) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t x = newid ? newid[v] : v;
        u64 any[W], p0[W], p1[W], p2[W], p3[W];
#pragma unroll
        for (int w = 0; w < W; w++) any[w] = p0[w] = p1[w] = p2[w] = p3[w] = 0ull;
#pragma unroll
        for (int l = 0; l < kMsHist; l++) {
            if (l >= cnt) break;
            u64 m[W];
            load_mask<W>(h.m[l] + x * W, m);
#pragma unroll
            for (int w = 0; w < W; w++) {
                any[w] |= m[w];
                if (l & 1) p0[w] |= m[w];
                if (l & 2) p1[w] |= m[w];
                if (l & 4) p2[w] |= m[w];
                if (l & 8) p3[w] |= m[w];
            }
        }
        uint32_t *o = out + v;
#pragma unroll
        for (int hw = 0; hw < 2 * W; hw++) {
            const int sh = (hw & 1) * 32;
            const uint32_t a = (uint32_t)(any[hw / 2] >> sh), b0 = (uint32_t)(p0[hw / 2] >> sh);
            const uint32_t b1 = (uint32_t)(p1[hw / 2] >> sh), b2 = (uint32_t)(p2[hw / 2] >> sh);
            const uint32_t b3 = (uint32_t)(p3[hw / 2] >> sh);
            const uint32_t left = k > (uint32_t)hw * 32 ? min(32u, k - (uint32_t)hw * 32) : 0u;
            if (!FIRST && !a) {
                o += (uint64_t)left * n;
                continue;
            }
#pragma unroll 8
            for (uint32_t s = 0; s < left; s++) {
                const uint32_t at = ((b0 >> s) & 1u) | (((b1 >> s) & 1u) << 1) | (((b2 >> s) & 1u) << 2) |
                                    (((b3 >> s) & 1u) << 3);
                const bool found = (a >> s) & 1u;
                if (FIRST || found) __stcs(o, found ? level0 + at : PTG_UNREACHED);
                o += n;
            }
        }
    }
}

// Pull level (symmetric graphs): N[v] = (OR of F over v's neighbours) & ~S[v],
// followed by k_msb_update.  A vertex can only gain sources that are live (in
// some frontier mask this level), so its scan stops as soon as it holds all
// live sources it has not seen; sources whose search died out (small
// components) no longer keep hubs scanning.  Work is split by degree so that
// no thread walks a long adjacency alone: vertices of degree <= small (a
// tuning value, 32 by default) are one thread each (k_msb_pull_small); the
// adjacency of every other vertex is cut into chunk-edge work items (1024 by
// default), one warp each (k_msb_pull_big),
// whose partial masks meet in N through atomicOr.  A neighbour's W words are
// one 32-byte sector for W = 4.
// Work items (vertex, chunk) of the vertices above `small`; counted first
// (items == nullptr), then written.  Item order is irrelevant.
template <class OffT>
__global__ void k_pull_items(uint64_t n, const OffT *off, uint32_t small, uint32_t chunk, uint2 *items,
                             unsigned long long *count) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t deg = (uint64_t)(off[v + 1] - off[v]);
        if (deg <= small) continue;
        uint32_t c = (uint32_t)((deg + chunk - 1) / chunk);
        unsigned long long base = atomicAdd(count, (unsigned long long)c);
        if (items)
            for (uint32_t i = 0; i < c; i++) items[base + i] = make_uint2((uint32_t)v, i);
    }
}

template <class OffT, int W>
__global__ void __launch_bounds__(kBlock) k_msb_pull_small(uint64_t n, const OffT *off, const uint32_t *col,
                                                           const u64 *F, const u64 *S, u64 *N,
                                                           const u64 *live_in, uint32_t small) {
    u64 live[W];
#pragma unroll
    for (int w = 0; w < W; w++) live[w] = live_in[w];
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        OffT b = off[v], e = off[v + 1];
        if (b == e || (uint64_t)(e - b) > small) continue;
        u64 s[W], need[W];
        load_mask<W>(S + v * W, s);
        bool none = true;
#pragma unroll
        for (int w = 0; w < W; w++) {
            need[w] = live[w] & ~s[w];
            none &= need[w] == 0ull;
        }
        if (none) continue;
        u64 acc[W];
#pragma unroll
        for (int w = 0; w < W; w++) acc[w] = 0;
        for (OffT k = b; k < e; k += 2) {
            uint32_t c0 = col[k];
            uint32_t c1 = k + 1 < e ? col[k + 1] : c0;
            u64 f0[W], f1[W];
            load_mask<W>(F + (uint64_t)c0 * W, f0);
            load_mask<W>(F + (uint64_t)c1 * W, f1);
            bool done = true;
#pragma unroll
            for (int w = 0; w < W; w++) {
                acc[w] |= f0[w] | f1[w];
                done &= (acc[w] & need[w]) == need[w];
            }
            if (done) break;
        }
#pragma unroll
        for (int w = 0; w < W; w++)
            if (acc[w] & need[w]) N[v * W + w] = acc[w] & need[w];
    }
}

// What a warp needs before it can gather (an item, its vertex's mask and offsets)
// is read for kMsbItems items side by side, and the masks meet with the warp's
// integer reduction.  One item after the other, with shuffles, left a warp
// waiting for four reads in a row 87% of the time: 256 sources on 4.2 M vertices
// and 128 M edges 2.27 -> 1.23 ms for the four pull levels (1.37 with 4 items,
// 1.48 with 16; asking for the next item's columns ahead gave 1%).
constexpr int kMsbItems = 8;
template <class OffT, int W>
__global__ void __launch_bounds__(kBlock, 4) k_msb_pull_big(const uint2 *items, uint64_t nitems, const OffT *off,
                                                         const uint32_t *col, const u64 *F, const u64 *S, u64 *N,
                                                         const u64 *live_in, uint32_t chunk) {
    constexpr int kU = 4;  // column loads in flight per lane
    u64 live[W];
#pragma unroll
    for (int w = 0; w < W; w++) live[w] = live_in[w];
    const int lane = (int)lane_id();
    const uint64_t nwarps = (uint64_t)gridDim.x * blockDim.x / 32;
    for (uint64_t i0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32 * kMsbItems; i0 < nitems; i0 += nwarps * kMsbItems) {
        // a few items side by side up to their edges: what they need, and where their rows begin
        uint32_t my_v = 0;
        OffT my_b = 0, my_e = 0;
        bool some = false;
        if (lane < kMsbItems && i0 + lane < nitems) {
            const uint2 item = items[i0 + lane];
            my_v = item.x;
            u64 s[W];
            load_mask<W>(S + (uint64_t)my_v * W, s);
            my_b = off[my_v] + (OffT)item.y * (OffT)chunk;
            my_e = off[(uint64_t)my_v + 1];
            if (my_e - my_b > (OffT)chunk) my_e = my_b + (OffT)chunk;
#pragma unroll
            for (int w = 0; w < W; w++) some |= (live[w] & ~s[w]) != 0ull;
        }
        unsigned todo = __ballot_sync(0xffffffffu, some);
        while (todo) {
            const int from = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint64_t v = __shfl_sync(0xffffffffu, my_v, from);
            const OffT b = __shfl_sync(0xffffffffu, my_b, from), e = __shfl_sync(0xffffffffu, my_e, from);
            u64 s[W], need[W];
            load_mask<W>(S + v * W, s);
#pragma unroll
            for (int w = 0; w < W; w++) need[w] = live[w] & ~s[w];
            u64 acc[W];
#pragma unroll
            for (int w = 0; w < W; w++) acc[w] = 0;
            for (OffT k0 = b; k0 < e; k0 += 32 * kU) {
                uint32_t c[kU];
#pragma unroll
                for (int j = 0; j < kU; j++) {
                    OffT k = k0 + (OffT)(j * 32 + lane);
                    c[j] = k < e ? col[k] : 0u;
                }
#pragma unroll
                for (int j = 0; j < kU; j++) {
                    if (k0 + (OffT)(j * 32 + lane) < e) {
                        u64 f[W];
                        load_mask<W>(F + (uint64_t)c[j] * W, f);
#pragma unroll
                        for (int w = 0; w < W; w++) acc[w] |= f[w];
                    }
                }
                bool done = true;
#pragma unroll
                for (int w = 0; w < W; w++) {
                    const u64 x = (u64)__reduce_or_sync(0xffffffffu, (unsigned)(acc[w] >> 32)) << 32 |
                                  __reduce_or_sync(0xffffffffu, (unsigned)acc[w]);
                    acc[w] = x;
                    done &= (x & need[w]) == need[w];
                }
                if (done) break;  // warp-uniform after the all-reduce
            }
#pragma unroll
            for (int w = 0; w < W; w++) {
                u64 x = acc[w] & need[w];
                if (lane == w && x) atomicOr(&N[v * W + w], x);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// MS-SSSP (64 sources per group)
// ---------------------------------------------------------------------------
// Source i of a group lives in distance word i of each vertex; lane l handles
// the adjacent words 2l and 2l+1, and its sources' bits in the 64-bit masks
// are l and 32 + l (so a warp's two ballots form a mask directly).
__device__ __forceinline__ u64 mss_bit(uint32_t i) { return 1ull << ((i & 1u) ? 32u + (i >> 1) : (i >> 1)); }

__global__ void k_mss_seed(const uint32_t *srcs, uint32_t k, u64 *A, uint32_t *dist, uint32_t base) {
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
        uint32_t s = srcs[i];
        atomicOr(&A[s], mss_bit(i));
        dist[(uint64_t)s * 64 + i] = base;
    }
}

// Bounds of k_mss_queue: none for distances of 2^30 and more.
constexpr uint32_t kMssFar = 1u << 30;
constexpr int kMssNone = 0x7F7F7F7F;  // dmax: no bound (any value from here on)

// MS-SSSP round: a warp relaxes one edge at a time for all 64 sources (lane l:
// sources 2l and 2l+1, one 8-byte load), eight edges per step so eight
// distance loads per lane are in flight.  Edge slots are tiled like the single-source expand.  The
// kernel is instruction-bound, so per-edge bookkeeping is done lane-parallel.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_mss_relax(const uint32_t *q, const OffT *sc, const OffT *rs,
                                                      const uint32_t *tr, const uint32_t *col, const uint32_t *w,
                                                      uint32_t *dist, const u64 *A, u64 *N, const int *dmin,
                                                      const int *dmax, const TravCtl *ctl) {
    __shared__ OffT s_sc[kTile + 2];
    __shared__ OffT s_rs[kTile + 2];
    __shared__ uint32_t s_u[kTile + 2];
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    uint64_t E = ctl->E;
    uint64_t ntiles = (E + kTile - 1) / kTile;
    constexpr int kPerWarp = kTile / (kBlock / 32);  // 256 edge slots per warp
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint64_t t0 = tile * kTile, t1 = min(E, t0 + kTile);
        uint64_t r0 = tr[tile];
        uint32_t nrows = (uint32_t)((uint64_t)tr[tile + 1] - r0 + 1);
        bool staged = nrows <= (uint32_t)kTile + 1;
        if (staged) {
            for (uint32_t k = threadIdx.x; k <= nrows; k += kBlock) {
                s_sc[k] = sc[r0 + k];
                if (k < nrows) {
                    s_rs[k] = rs[r0 + k];
                    s_u[k] = q[r0 + k];
                }
            }
        }
        __syncthreads();
        uint64_t w0 = t0 + (uint64_t)wid * kPerWarp;
        uint64_t w1 = min(t1, w0 + kPerWarp);
        if (w0 < w1) {
            uint64_t row = staged ? last_le(s_sc, 0, nrows, w0) : last_le(sc, r0, r0 + nrows, w0);
            auto row_info = [&](uint64_t r, uint64_t &next, OffT &delta, uint32_t &u) {
                next = staged ? (uint64_t)s_sc[r + 1] : (uint64_t)sc[r + 1];
                OffT rsv = staged ? s_rs[r] : rs[r];
                OffT scv = staged ? s_sc[r] : sc[r];
                delta = rsv - scv;
                u = staged ? s_u[r] : q[r];
            };
            // Edges go 32 at a time: lane b finds the row of edge b and loads
            // its target and weight once; the warp then walks the 32 edges
            // taking them from the lanes with shuffles (the row bookkeeping
            // is done once per edge, not once per edge and lane).
            uint32_t cur_u = 0xFFFFFFFFu;
            u64 am = 0;
            uint32_t du0 = 0, du1 = 0;
            for (uint64_t j = w0; j < w1; j += 32) {
                uint64_t jj = j + lane;
                bool ok = jj < w1;
                uint64_t r = row, nx;
                OffT delta;
                uint32_t ul;
                row_info(r, nx, delta, ul);
                while (ok && jj >= nx) {
                    r++;
                    row_info(r, nx, delta, ul);
                }
                uint32_t vl = 0, wl = 0;
                bool keep = false;
                if (ok) {
                    uint64_t e = (uint64_t)(OffT)(delta + (OffT)jj);
                    vl = __ldcs(col + e);
                    wl = __ldcs(w + e);
                    const int top = dmax[vl];  // see k_mss_queue
                    keep = top >= kMssNone || (long long)dmin[ul] + wl < top;
                }
                row = __shfl_sync(0xffffffffu, r, 31);
                unsigned left = __ballot_sync(0xffffffffu, keep);
                while (left) {
                    uint32_t vv[8], nd0[8], nd1[8], cur0[8], cur1[8];
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        const bool have = left != 0;
                        const uint32_t src = have ? __ffs(left) - 1 : 0;
                        left &= left - 1;
                        uint32_t ut = __shfl_sync(0xffffffffu, ul, src);
                        uint32_t wt = __shfl_sync(0xffffffffu, wl, src);
                        vv[t] = __shfl_sync(0xffffffffu, vl, src);
                        nd0[t] = nd1[t] = PTG_UNREACHED;
                        if (have) {
                            if (ut != cur_u) {  // warp-uniform: a new tail vertex
                                cur_u = ut;
                                am = A[ut];
                                uint2 d = reinterpret_cast<const uint2 *>(dist + (uint64_t)ut * 64)[lane];
                                du0 = d.x;
                                du1 = d.y;
                            }
                            if ((am >> lane) & 1ull) nd0[t] = du0 + wt;
                            if ((am >> (32 + lane)) & 1ull) nd1[t] = du1 + wt;
                        }
                    }
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        cur0[t] = cur1[t] = 0u;
                        if ((nd0[t] & nd1[t]) != PTG_UNREACHED) {
                            uint2 c = reinterpret_cast<const uint2 *>(dist + (uint64_t)vv[t] * 64)[lane];
                            cur0[t] = c.x;
                            cur1[t] = c.y;
                        }
                    }
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        bool i0 = nd0[t] < cur0[t], i1 = nd1[t] < cur1[t];
                        if (i0) atomicMin(&dist[(uint64_t)vv[t] * 64 + 2 * lane], nd0[t]);
                        if (i1) atomicMin(&dist[(uint64_t)vv[t] * 64 + 2 * lane + 1], nd1[t]);
                        unsigned b0 = __ballot_sync(0xffffffffu, i0), b1 = __ballot_sync(0xffffffffu, i1);
                        if (lane == 0 && (b0 | b1)) atomicOr(&N[vv[t]], (u64)b0 | ((u64)b1 << 32));
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Dense MS-SSSP round on a graph whose edges carry the same weight both ways
// (graph_weights_symmetric): every vertex takes the least candidate over its
// neighbours in registers and writes its own distances once.  Pushing the same
// round sends two reductions of 8 sectors per edge to L2 and takes three times
// the instructions per edge: 2.4 and 2.1 ms in the two heaviest rounds of 64
// sources on RMAT-20, 0.52 ms a round on average here.  Work is split as in the MS-BFS pull:
// rows of up to `small` edges by 32-vertex groups, longer ones in chunks, a
// warp each; 32 edges are loaded side by side, those that pass the bound of
// k_mss_queue are taken 8 at a time by the whole warp, all 64 sources alike:
// where a source is not active its candidate was offered before and improves
// nothing, and a test would cost as much as the candidate.  A row in several
// chunks meets in atomics.  Distances read may be this round's already (they
// only fall, and an improved vertex is queued for the next round).
struct MssEdge {
    uint32_t u, w;  // neighbour and weight
};

template <class OffT>
__device__ __forceinline__ void mss_pull_row(OffT b, OffT e, uint64_t v, bool alone, const uint32_t *col,
                                             const uint32_t *w, uint32_t *dist, const u64 *A, u64 *N,
                                             const int *dmin, int top, MssEdge *pass) {
    const unsigned lane = lane_id();
    bool loaded = false;
    uint2 own = make_uint2(0u, 0u), best = own;
    // the next 32 edges, and what says whether they pass, are on their way
    // while the present ones are taken (one step after the other: 7.0 instead
    // of 5.1 ms for the eight pull rounds of 128 sources on RMAT-20; rows side
    // by side as in k_msb_pull_big need more registers and gave that back)
    bool ok = b + (OffT)lane < e;
    uint32_t ul = ok ? __ldcs(col + b + lane) : 0u, wl = ok ? __ldcs(w + b + lane) : 0u;
    bool some = ok && A[ul] != 0ull;
    int least = ok ? dmin[ul] : 0;
    for (OffT k0 = b; k0 < e; k0 += 32) {
        const OffT kn = k0 + 32 + (OffT)lane;
        const bool okn = kn < e;
        const uint32_t un = okn ? __ldcs(col + kn) : 0u, wn = okn ? __ldcs(w + kn) : 0u;
        const bool keep = some && (top >= kMssNone || (long long)least + wl < top);
        const uint32_t uk = ul, wk = wl;
        ul = un;
        wl = wn;
        some = okn && A[un] != 0ull;
        least = okn ? dmin[un] : 0;
        const unsigned left = __ballot_sync(0xffffffffu, keep);
        if (!left) continue;
        // the edges that pass, side by side in shared memory, padded with
        // the vertex itself (reading them back broadcast takes one instruction
        // where shuffles took nine)
        const int cnt = __popc(left), at = keep ? __popc(left & lanemask_lt()) : cnt + __popc(~left & lanemask_lt());
        __syncwarp();
        pass[at] = MssEdge{keep ? uk : (uint32_t)v, keep ? wk : 0u};
        __syncwarp();
        if (!loaded) {
            own = reinterpret_cast<const uint2 *>(dist + v * 64)[lane];
            best = own;
            loaded = true;
        }
        auto take = [&](auto count, int i) {
            constexpr int kN = decltype(count)::value;
            uint2 d[kN];
#pragma unroll
            for (int t = 0; t < kN; t++) d[t] = reinterpret_cast<const uint2 *>(dist + (uint64_t)pass[i + t].u * 64)[lane];
#pragma unroll
            for (int t = 0; t < kN; t++) {
                const uint32_t add = pass[i + t].w;
                best.x = __viaddmin_u32(min(d[t].x, ~add), add, best.x);
                best.y = __viaddmin_u32(min(d[t].y, ~add), add, best.y);
            }
        };
        int i = 0;
        for (; i + 4 < cnt; i += 8) take(std::integral_constant<int, 8>{}, i);
        if (i < cnt) take(std::integral_constant<int, 4>{}, i);
    }
    if (!loaded) return;
    const bool i0 = best.x < own.x, i1 = best.y < own.y;
    const unsigned b0 = __ballot_sync(0xffffffffu, i0), b1 = __ballot_sync(0xffffffffu, i1);
    if (!(b0 | b1)) return;
    if (alone) {
        reinterpret_cast<uint2 *>(dist + v * 64)[lane] = best;
        if (lane == 0) N[v] = (u64)b0 | ((u64)b1 << 32);
    } else {
        if (i0) atomicMin(&dist[v * 64 + 2 * lane], best.x);
        if (i1) atomicMin(&dist[v * 64 + 2 * lane + 1], best.y);
        if (lane == 0) atomicOr(&N[v], (u64)b0 | ((u64)b1 << 32));
    }
}

template <class OffT>
__global__ void __launch_bounds__(kBlock, 5) k_mss_pull(const uint2 *items, uint64_t nitems, uint32_t small,
                                                     uint32_t chunk, uint64_t n, const OffT *off, const uint32_t *col,
                                                     const uint32_t *w, uint32_t *dist, const u64 *A, u64 *N,
                                                     const int *dmin, const int *dmax) {
    __shared__ __align__(16) MssEdge s_pass[kBlock / 32][32];
    MssEdge *pass = s_pass[threadIdx.x >> 5];
    const unsigned lane = lane_id();
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32), wid = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5;
    for (uint64_t i = wid; i < nitems; i += nwarps) {
        const uint2 it = items[i];
        const OffT row = off[it.x], end = off[(uint64_t)it.x + 1];
        const OffT b = row + (OffT)it.y * (OffT)chunk;
        const OffT e = end - b > (OffT)chunk ? b + (OffT)chunk : end;
        mss_pull_row<OffT>(b, e, it.x, end - row <= (OffT)chunk, col, w, dist, A, N, dmin, dmax[it.x], pass);
    }
    for (uint64_t wb = wid; wb * 32 < n; wb += nwarps) {
        const uint64_t v = wb * 32 + lane;
        const OffT b = v < n ? off[v] : (OffT)0, e = v < n ? off[v + 1] : (OffT)0;
        const int top = v < n ? dmax[v] : 0;
        unsigned rows = __ballot_sync(0xffffffffu, b < e && (uint64_t)(e - b) <= small);
        while (rows) {
            const int j = __ffs(rows) - 1;
            rows &= rows - 1;
            mss_pull_row<OffT>(__shfl_sync(0xffffffffu, b, j), __shfl_sync(0xffffffffu, e, j), wb * 32 + j, true, col, w,
                               dist, A, N, dmin, __shfl_sync(0xffffffffu, top, j), pass);
        }
    }
}

// The vertex of the highest degree (the smallest such id).
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_mss_hub(const OffT *off, uint64_t n, u64 *best) {
    u64 b = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const u64 deg = min((u64)(off[v + 1] - off[v]), 0xffffffffull);
        b = max(b, deg << 32 | (0xffffffffull - v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if (lane_id() == 0) atomicMax(best, b);
}

// After a round: the queue of the vertices with a new mask, the sum of their
// degrees (ctl->m_unvisited), the sources that go on (live_next), and per
// queued vertex the bounds that k_mss_relax drops edges by.  Source s improves
// v over an edge (u, v) of weight w only if dist[u][s] + w < dist[v][s], with
// both sides taken less the source's distance to a hub, base[s]: so only if
// dmin[u] + w < dmax[v], the least such value of u's active sources and the
// largest of v's live ones.  Less base[s] the sources agree on how far a
// vertex lies, and the bound lets through little more than improves (RMAT-14,
// rounds 3 to 7: 69, 25, 12, 7, 5% of the edges, of which 46, 16, 7, 3, 2% improve a
// source; the plain distances would let 95 ... 63% through).  The sources in
// `live` are those that had an active vertex a round ago: one whose search has
// ended, or that never reached this component, does not hold dmax up.  A
// dmax[v] formed earlier stays a bound, as distances only fall.  With `refresh`
// (a round over many edges follows) base is brought up to date, and dmax is
// formed anew for all vertices if that changed it, or if sources have dropped
// out of live.  Distances of 2^30 and more: no bound.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_mss_queue(const u64 *M, uint64_t n, const OffT *off, uint32_t *q,
                                                      TravCtl *ctl, const uint32_t *dist, int *dmin, int *dmax,
                                                      const u64 *hub, const uint32_t *base_was, uint32_t *base,
                                                      const u64 *was, const u64 *live, u64 *live_next, int refresh) {
    const unsigned lane = lane_id();
    const u64 lm = *live;
    const bool l0 = (lm >> lane) & 1ull, l1 = (lm >> (32 + lane)) & 1ull;
    // this lane's two sources' distances to the hub, 0 while there is none
    const uint64_t h = 0xffffffffull - (*hub & 0xffffffffull);
    uint2 b = reinterpret_cast<const uint2 *>(dist + h * 64)[lane];
    if (b.x >= kMssFar) b.x = 0;
    if (b.y >= kMssFar) b.y = 0;
    const uint2 bw = reinterpret_cast<const uint2 *>(base_was)[lane];
    if (!refresh) b = bw;
    const bool all = __any_sync(0xffffffffu, b.x != bw.x || b.y != bw.y) || (refresh && *was != lm);
    if (blockIdx.x == 0 && threadIdx.x < 32) reinterpret_cast<uint2 *>(base)[lane] = b;
    unsigned long long degsum = 0;
    u64 on = 0;
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t wb = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5; wb * 32 < n; wb += nwarps) {
        const uint64_t v = wb * 32 + lane;
        const u64 m = v < n ? M[v] : 0ull;
        on |= m;
        if (m) {
            degsum += (unsigned long long)(off[v + 1] - off[v]);
            warp_append(q, &ctl->next_tail, (unsigned)n, &ctl->error, (uint32_t)v);
        }
        __syncwarp();
        unsigned todo = all ? __ballot_sync(0xffffffffu, v < n) : __ballot_sync(0xffffffffu, m != 0);
        while (todo) {  // four vertices' distances in flight, the warp's lanes across the sources
            uint32_t at[4];
            uint2 d[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                at[t] = todo ? __ffs(todo) - 1 : 32u;
                todo &= todo - 1;
                d[t] = make_uint2(0u, 0u);
                if (at[t] < 32) d[t] = reinterpret_cast<const uint2 *>(dist + (wb * 32 + at[t]) * 64)[lane];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (at[t] >= 32) break;
                const u64 am = __shfl_sync(0xffffffffu, m, at[t]);
                const bool a0 = (am >> lane) & 1ull, a1 = (am >> (32 + lane)) & 1ull;
                const bool far0 = d[t].x >= kMssFar, far1 = d[t].y >= kMssFar;
                const int x0 = (int)d[t].x - (int)b.x, x1 = (int)d[t].y - (int)b.y;  // below 2^30 either way unless far
                const int lo = min(a0 ? (far0 ? INT_MIN : x0) : INT_MAX, a1 ? (far1 ? INT_MIN : x1) : INT_MAX);
                const int hi = max(l0 ? (far0 ? kMssNone : x0) : INT_MIN, l1 ? (far1 ? kMssNone : x1) : INT_MIN);
                const int mn = __reduce_min_sync(0xffffffffu, lo), mx = __reduce_max_sync(0xffffffffu, hi);
                if (lane == 0) {
                    if (am) dmin[wb * 32 + at[t]] = mn;
                    dmax[wb * 32 + at[t]] = mx;
                }
            }
        }
    }
    u64 x[1] = {on};
    live_or<1>(live_next, x);
    degsum = block_reduce_sum(degsum);
    if (threadIdx.x == 0 && degsum) atomicAdd(&ctl->m_unvisited, degsum);
}

// dist[x*64 + s] -> out[s*n + v] for s < k, x = newid[v] on a regrouped graph
// (else v).  Tiles of 64 vertices x 64 sources; a warp has 8 vertices' rows in
// flight and writes 256 bytes of a result row.  (With 32 vertices, an element
// of one row at a time per thread: 250 us for 64 sources on 1 M vertices, now
// 85; 0.5 GB moved.)
constexpr int kTrVerts = 64;
__global__ void __launch_bounds__(kBlock) k_mss_transpose(const uint32_t *dist, uint64_t n, uint32_t k,
                                                          const uint32_t *newid, uint32_t *out) {
    constexpr int kEach = kTrVerts / (kBlock / 32);
    __shared__ uint32_t t[kTrVerts][65];
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    for (uint64_t v0 = (uint64_t)blockIdx.x * kTrVerts; v0 < n; v0 += (uint64_t)gridDim.x * kTrVerts) {
        const uint64_t mine = min(v0 + wid * kEach + lane % kEach, n - 1);
        const uint32_t x = newid ? newid[mine] : (uint32_t)mine;
        uint2 d[kEach];
#pragma unroll
        for (int i = 0; i < kEach; i++)
            d[i] = __ldcs(reinterpret_cast<const uint2 *>(dist + (uint64_t)__shfl_sync(0xffffffffu, x, i) * 64) + lane);
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            t[wid * kEach + i][2 * lane] = d[i].x;
            t[wid * kEach + i][2 * lane + 1] = d[i].y;
        }
        __syncthreads();
        for (uint32_t s = wid; s < k; s += kBlock / 32) {
            uint32_t *row = out + (uint64_t)s * n + v0;
#pragma unroll
            for (int j = 0; j < kTrVerts; j += 32)
                if (v0 + j + lane < n) __stcs(row + j + lane, t[j + lane][s]);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
struct MsState {
    ptg_ctx *ctx;
    Workspace *ws;
    cudaStream_t st;
    TravCtl *d_ctl, *h_ctl;
    uint32_t *q, *qn;
};

// Frontier degree scan + tile rows for the queue in ws.q[0] (count in ctl->F).
template <class OffT>
void ms_scan(ptg_ctx *ctx, Workspace &ws, const OffT *off, uint64_t m, uint64_t F, TravCtl *d_ctl) {
    cudaStream_t st = ctx->stream;
    const int sms = ctx->sm_count;
    OffT *sc = ws.scan.as<OffT>(), *rs = ws.rowstart.as<OffT>();
    unsigned long long *bsum = ws.bsum.as<unsigned long long>();
    const uint32_t *q = ws.q[0].as<uint32_t>();
    if (F <= kSmallFrontier) {  // the scan and the tile rows in one CTA
        launch(ctx, "k_scan_small", k_scan_small<OffT>, 1, kBlock, 0, st, q, d_ctl, off, (OffT)0, (OffT)m, sc, rs,
               ws.tiles.as<uint32_t>(), 1);
        return;
    }
    int nb = grid_for(F, kBlock, 1024);
    launch(ctx, "k_scan_reduce", k_scan_reduce<OffT>, nb, kBlock, 0, st, q, (const TravCtl *)d_ctl, off, (OffT)0, (OffT)m,
           bsum);
    launch(ctx, "k_scan_bsums", k_scan_bsums, 1, kBlock, 0, st, bsum, nb, d_ctl, 1);
    launch(ctx, "k_scan_write", k_scan_write<OffT>, nb, kBlock, 0, st, q, (const TravCtl *)d_ctl, off, (OffT)0, (OffT)m,
           (const unsigned long long *)bsum, sc, rs);
    launch(ctx, "k_tile_rows", k_tile_rows<OffT>, sms * 4, kBlock, 0, st, (const OffT *)sc, (const TravCtl *)d_ctl,
           ws.tiles.as<uint32_t>());
}

// ws.bsum: scan partials | 256 sources | MS-BFS: all-sources mask, two
// live-source masks; MS-SSSP: four live-source words, the hub, two bases
constexpr uint64_t kMsSmall = 1024 * 8 + 256 * 4 + 5 * 8 + 2 * 64 * 4;

template <class OffT>
void ms_prepare(ptg_graph *g) {
    Workspace &ws = g->ctx->ws;
    uint64_t n = g->n, m = g->m;
    ws.q[0].ensure(n * 4);
    ws.q[1].ensure(n * 4);
    ws.scan.ensure((n + 1) * sizeof(OffT));
    ws.rowstart.ensure((n + 1) * sizeof(OffT));
    ws.tiles.ensure((m / kTile + 4) * 4);
    ws.bsum.ensure(kMsSmall);
    ws.ctl.ensure(sizeof(TravCtl));
    ws.h_ctl.ensure(sizeof(TravCtl));
    ensure_level_msg(ws);
}

// Chunked work items of the high-degree vertices, built once per graph.
template <class OffT>
void build_pull_items(ptg_graph *g) {
    ptg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const OffT *off = g->d_off.as<OffT>();
    unsigned long long *cnt = ctx->ws.bsum.as<unsigned long long>();
    int grid = grid_for(g->n, kBlock, ctx->sm_count * 8);
    PTG_CUDA_TRY(cudaMemsetAsync(cnt, 0, 8, st));
    const uint32_t small = ctx->tuning.ms_pull_small, chunk = ctx->tuning.ms_pull_chunk;
    launch(ctx, "k_pull_items", k_pull_items<OffT>, grid, kBlock, 0, st, g->n, off, small, chunk, (uint2 *)nullptr,
           cnt);
    unsigned long long total = 0;
    PTG_CUDA_TRY(cudaMemcpyAsync(&total, cnt, 8, cudaMemcpyDeviceToHost, st));
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    if (total) {
        g->d_pull_items.ensure(total * sizeof(uint2));
        PTG_CUDA_TRY(cudaMemsetAsync(cnt, 0, 8, st));
        launch(ctx, "k_pull_items", k_pull_items<OffT>, grid, kBlock, 0, st, g->n, off, small, chunk,
               g->d_pull_items.as<uint2>(), cnt);
    }
    g->pull_small = small;
    g->pull_chunk = chunk;
    g->n_pull_items = total;
    g->pull_items_built = true;
}

// End of a multi-source round on the device: the round's outcome goes to
// the host through the level message (seq last, after a system-scope
// fence) and the control block restarts with the new queue's size.
__global__ void k_ms_round_end(TravCtl *ctl, LevelMsg *msg, uint32_t seq) {
    TravCtl c = *ctl;
    volatile LevelMsg *m = msg;
    m->F = c.next_tail;
    m->error = c.error;
    m->frontier_E = c.m_unvisited;
    m->E = c.E;
    TravCtl upd{};
    upd.F = c.next_tail;
    *ctl = upd;
    __threadfence_system();
    m->seq = seq;
}

// The round's outcome (new queue size, unvisited edges, scanned edges),
// then the new queue taken and the counters reset.  Through the mapped
// level message when there is one, else by copying the control block back.
inline void ms_next(ptg_ctx *ctx, Workspace &ws, uint64_t &F, uint64_t &Eact, uint64_t &E) {
    cudaStream_t st = ctx->stream;
    TravCtl *d_ctl = ws.ctl.as<TravCtl>(), *h_ctl = ws.h_ctl.as<TravCtl>();
    if (ws.d_msg) {
        launch(ctx, "k_ms_round_end", k_ms_round_end, 1, 1, 0, st, d_ctl, ws.d_msg, ws.msg_seq + 1);
        ws.msg_seq++;
        const LevelMsg msg = wait_level_msg(ctx, st);
        PTG_REQUIRE(msg.error == 0, PTG_ERR_CUDA, "frontier overflow in multi-source round");
        F = msg.F;
        Eact = msg.frontier_E;
        E = msg.E;
    } else {
        PTG_CUDA_TRY(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(TravCtl), cudaMemcpyDeviceToHost, st));
        PTG_CUDA_TRY(cudaStreamSynchronize(st));
        PTG_REQUIRE(h_ctl->error == 0, PTG_ERR_CUDA, "frontier overflow in multi-source round");
        F = h_ctl->next_tail;
        Eact = h_ctl->m_unvisited;
        E = h_ctl->E;
        TravCtl upd{};
        upd.F = (uint32_t)F;
        PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &upd, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
    }
    std::swap(ws.q[0].p, ws.q[1].p);
    std::swap(ws.q[0].bytes, ws.q[1].bytes);
    std::swap(ws.q[0].dev, ws.q[1].dev);
}

template <class OffT, int W>
void msbfs_impl(ptg_graph *g, const uint32_t *h_srcs, uint32_t k, uint32_t *d_rows, uint32_t flags, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n, m = g->m;
    const int sms = ctx->sm_count;
    const OffT *off = g->d_off.as<OffT>();
    const uint32_t *col = g->d_col.as<uint32_t>();
    uint32_t base = (flags & PTG_LEVEL_ZERO_BASED) ? 0u : 1u;
    ms_prepare<OffT>(g);
    // ms[0]: the levels' frontier masks (two at least: a level and the next);
    // ms[1]: sources seen per vertex
    const uint64_t mask_words = (n * W + 31) / 32 * 32, mask_bytes = mask_words * 8;
    ws.ms[1].ensure(mask_bytes);
    const int hist = ms_history(ctx, mask_bytes);
    if (g->symmetric && !g->pull_items_built) build_pull_items<OffT>(g);
    u64 *S = ws.ms[1].as<u64>();
    MsHist h{};
    for (int i = 0; i < hist; i++) h.m[i] = ws.ms[0].as<u64>() + i * mask_words;
    unsigned long long *bsum = ws.bsum.as<unsigned long long>();
    uint32_t *d_srcs = reinterpret_cast<uint32_t *>(bsum + 1024);
    u64 *d_all = reinterpret_cast<u64 *>(d_srcs + 256);
    TravCtl *d_ctl = ws.ctl.as<TravCtl>();
    PTG_CUDA_TRY(cudaMemsetAsync(S, 0, n * 8 * W, st));
    PTG_CUDA_TRY(cudaMemsetAsync((void *)h.m[0], 0, n * 8 * W, st));
    u64 all[W];
    for (int w = 0; w < W; w++) {
        int bits = std::max(0, std::min(64, (int)k - 64 * w));
        all[w] = bits == 64 ? ~0ull : ((1ull << bits) - 1ull);
    }
    PTG_CUDA_TRY(cudaMemcpyAsync(d_srcs, h_srcs, k * 4, cudaMemcpyHostToDevice, st));
    map_sources_dev(g, d_srcs, k);
    launch(ctx, "k_msb_seed", k_msb_seed<W>, 1, 256, 0, st, (const uint32_t *)d_srcs, k, (u64 *)h.m[0], S);
    TravCtl init{};
    PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &init, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
    int vgrid = grid_for(n, kBlock, sms * 8);
    launch(ctx, "k_msb_queue", k_msb_queue<OffT, W>, vgrid, kBlock, 0, st, h.m[0], n, off,
           ws.q[1].as<uint32_t>(), d_ctl);
    uint64_t F, Eact, E;
    ms_next(ctx, ws, F, Eact, E);
    // the kept levels: h.m[0] is level `level0`, h.m[cnt - 1] the current
    // frontier, and the first `written` of them are in the rows already
    uint32_t level0 = base;
    int cnt = 1, written = 0, round = 0;
    bool first = true;
    auto write_levels = [&] {
        MsHist part{};
        for (int i = written; i < cnt; i++) part.m[i - written] = h.m[i];
        const uint32_t *newid = g->relabeled ? g->d_newid.as<uint32_t>() : nullptr;
        const int grid = grid_for(n, kBlock, sms * 8);
        if (first)
            launch(ctx, "k_msb_levels", k_msb_levels<W, true>, grid, kBlock, 0, st, part, cnt - written, n, k, newid,
                   level0 + (uint32_t)written, d_rows);
        else
            launch(ctx, "k_msb_levels", k_msb_levels<W, false>, grid, kBlock, 0, st, part, cnt - written, n, k, newid,
                   level0 + (uint32_t)written, d_rows);
        first = false;
    };
    // live[c]: OR of every frontier mask of the current level (the sources
    // still expanding); the seed frontier holds all of them.
    u64 *d_live[2] = {d_all + 4, d_all + 8};
    PTG_CUDA_TRY(cudaMemcpyAsync(d_live[0], all, sizeof(all), cudaMemcpyHostToDevice, st));
    const uint32_t max_rounds = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, n + 16);
    while (F > 0) {
        if (rr.iterations >= max_rounds) throw Error{PTG_ERR_TIMEOUT, "iteration limit reached"};
        rr.iterations++;
        if (cnt == hist) {  // full: the rows take the kept levels, the frontier stays
            write_levels();
            std::swap(h.m[0], h.m[cnt - 1]);
            level0 += (uint32_t)cnt - 1;
            cnt = written = 1;
        }
        const u64 *Mc = h.m[cnt - 1];
        u64 *Mn = (u64 *)h.m[cnt];
        PTG_CUDA_TRY(cudaMemsetAsync(d_live[round ^ 1], 0, 8 * W, st));
        bool pull = g->symmetric && Eact * 10 > m;
        PTG_CUDA_TRY(cudaMemsetAsync(Mn, 0, n * 8 * W, st));
        if (pull) {
            launch(ctx, "k_msb_pull_small", k_msb_pull_small<OffT, W>, vgrid, kBlock, 0, st, n, off, col,
                   Mc, (const u64 *)S, Mn, (const u64 *)d_live[round], g->pull_small);
            if (g->n_pull_items)
                launch(ctx, "k_msb_pull_big", k_msb_pull_big<OffT, W>, sms * 32, kBlock, 0, st,
                       (const uint2 *)g->d_pull_items.p, g->n_pull_items, off, col, Mc,
                       (const u64 *)S, Mn, (const u64 *)d_live[round], g->pull_chunk);
        } else {
            ms_scan<OffT>(ctx, ws, off, m, F, d_ctl);
            launch(ctx, "k_msb_push", k_msb_push<OffT, W>, sms * 8, kBlock, 0, st, (const uint32_t *)ws.q[0].p,
                   (const OffT *)ws.scan.p, (const OffT *)ws.rowstart.p, (const uint32_t *)ws.tiles.p, col,
                   Mc, (const u64 *)S, Mn, (const TravCtl *)d_ctl);
        }
        launch(ctx, "k_msb_update", k_msb_update<OffT, W>, vgrid, kBlock, 0, st, n, off, Mn, S,
               ws.q[1].as<uint32_t>(), d_ctl, d_live[round ^ 1]);
        PTG_CUDA_TRY(cudaGetLastError());
        ms_next(ctx, ws, F, Eact, E);
        rr.edges_relaxed += pull ? 0 : E;
        round ^= 1;
        cnt++;
    }
    write_levels();
    PTG_CUDA_TRY(cudaGetLastError());
}

template <class OffT>
void mssssp_impl(ptg_graph *g, const uint32_t *h_srcs, uint32_t k, uint32_t *d_rows, uint32_t flags,
                 RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n, m = g->m;
    const int sms = ctx->sm_count;
    const OffT *off = g->d_off.as<OffT>();
    const uint32_t *col = g->d_col.as<uint32_t>();
    const uint32_t *wt = g->d_w.as<uint32_t>();
    uint32_t base = (flags & PTG_LEVEL_ZERO_BASED) ? 0u : 1u;
    ms_prepare<OffT>(g);
    ws.ms[0].ensure(n * 8);
    ws.ms[1].ensure(n * 8);
    u64 *M0 = ws.ms[0].as<u64>(), *M1 = ws.ms[1].as<u64>();
    unsigned long long *bsum = ws.bsum.as<unsigned long long>();
    uint32_t *d_srcs = reinterpret_cast<uint32_t *>(bsum + 1024);
    TravCtl *d_ctl = ws.ctl.as<TravCtl>();
    ws.aux.ensure(n * 64 * 4 + 2 * n * 4);
    uint32_t *dist = ws.aux.as<uint32_t>();
    int *dmin = reinterpret_cast<int *>(dist + n * 64), *dmax = dmin + n;
    PTG_CUDA_TRY(cudaMemsetAsync(dist, 0xFF, n * 64 * 4, st));
    PTG_CUDA_TRY(cudaMemsetAsync(M0, 0, n * 8, st));
    PTG_CUDA_TRY(cudaMemsetAsync(M1, 0, n * 8, st));
    PTG_CUDA_TRY(cudaMemcpyAsync(d_srcs, h_srcs, k * 4, cudaMemcpyHostToDevice, st));
    map_sources_dev(g, d_srcs, k);
    launch(ctx, "k_mss_seed", k_mss_seed, 1, 64, 0, st, (const uint32_t *)d_srcs, k, M0, dist, base);
    TravCtl init{};
    PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &init, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
    int vgrid = grid_for(n, kBlock, sms * 8);
    // live sources of the last rounds, four words used in turn: two read, one
    // written, one cleared for the next round
    u64 *d_live = reinterpret_cast<u64 *>(d_srcs + 256);
    PTG_CUDA_TRY(cudaMemsetAsync(d_live, 0xFF, 16, st));
    PTG_CUDA_TRY(cudaMemsetAsync(d_live + 2, 0, 16, st));
    const bool can_pull = graph_weights_symmetric(g);
    if (can_pull && !g->pull_items_built) build_pull_items<OffT>(g);
    // the hub, and the sources' distances to it as of the last two rounds
    u64 *d_hub = d_live + 4;
    uint32_t *d_base = reinterpret_cast<uint32_t *>(d_hub + 1);
    PTG_CUDA_TRY(cudaMemsetAsync(d_hub, 0, 8, st));
    PTG_CUDA_TRY(cudaMemsetAsync(d_base, 0, 64 * 4, st));
    PTG_CUDA_TRY(cudaMemsetAsync(dmax, 0x7F, n * 4, st));  // kMssNone
    launch(ctx, "k_mss_hub", k_mss_hub<OffT>, vgrid, kBlock, 0, st, off, n, d_hub);
    uint32_t round = 0;
    auto queue = [&](const u64 *M, bool refresh) {
        launch(ctx, "k_mss_queue", k_mss_queue<OffT>, vgrid, kBlock, 0, st, M, n, off, ws.q[1].as<uint32_t>(), d_ctl,
               (const uint32_t *)dist, dmin, dmax, (const u64 *)d_hub, (const uint32_t *)d_base + round % 2 * 64,
               d_base + (round + 1) % 2 * 64, (const u64 *)d_live + round % 4,
               (const u64 *)d_live + (round + 1) % 4, d_live + (round + 2) % 4, refresh ? 1 : 0);
        PTG_CUDA_TRY(cudaMemsetAsync(d_live + round % 4, 0, 8, st));
        round++;
    };
    queue(M0, false);
    uint64_t F, Eact, E;
    ms_next(ctx, ws, F, Eact, E);
    int cur = 0;
    const uint32_t max_rounds = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, 4 * n + 16);
    while (F > 0) {
        if (rr.iterations >= max_rounds) throw Error{PTG_ERR_TIMEOUT, "iteration limit reached"};
        rr.iterations++;
        u64 *Mc = cur ? M1 : M0, *Mn = cur ? M0 : M1;
        PTG_CUDA_TRY(cudaMemsetAsync(Mn, 0, n * 8, st));
        // 64 sources on RMAT-20, two batches: 7.4 ms with the line at m / 5, 8.0 at
        // m / 2 and 7.6 at m / 16 (a pull round reads every edge's filter)
        const bool pull = can_pull && Eact * 5 > m;
        const uint64_t scanned = Eact;
        if (pull) {
            launch(ctx, "k_mss_pull", k_mss_pull<OffT>, sms * 40, kBlock, 0, st, (const uint2 *)g->d_pull_items.p,
                   g->n_pull_items, g->pull_small, g->pull_chunk, n, off, col, wt, dist, (const u64 *)Mc, Mn,
                   (const int *)dmin, (const int *)dmax);
        } else {
            ms_scan<OffT>(ctx, ws, off, m, F, d_ctl);
            launch(ctx, "k_mss_relax", k_mss_relax<OffT>, sms * 6, kBlock, 0, st, (const uint32_t *)ws.q[0].p,
                   (const OffT *)ws.scan.p, (const OffT *)ws.rowstart.p, (const uint32_t *)ws.tiles.p, col, wt, dist,
                   (const u64 *)Mc, Mn, (const int *)dmin, (const int *)dmax, (const TravCtl *)d_ctl);
        }
        // a refresh reads every distance, which a round over a large part of the edges repays
        queue(Mn, Eact * 8 > m);
        PTG_CUDA_TRY(cudaGetLastError());
        ms_next(ctx, ws, F, Eact, E);
        rr.edges_relaxed += pull ? scanned : E;
        cur ^= 1;
    }
    launch(ctx, "k_mss_transpose", k_mss_transpose, grid_for(n, kTrVerts, sms * 8), kBlock, 0, st,
           (const uint32_t *)dist, n, k, (const uint32_t *)(g->relabeled ? g->d_newid.p : nullptr), d_rows);
    PTG_CUDA_TRY(cudaGetLastError());
}

}  // namespace

// Builds the per-graph tables of the fused passes (pull work items) now
// rather than on first use.
void ms_prepare_graph(ptg_graph *g) {
    if (g->out_of_core || !g->symmetric) return;
    graph_weights_symmetric(g);
    if (g->pull_items_built) return;
    g->ctx->ws.bsum.ensure(kMsSmall);
    if (g->off64) build_pull_items<unsigned long long>(g);
    else build_pull_items<uint32_t>(g);
}

// Sources per fused group: 256 for BFS (4 mask words), 64 for SSSP.
uint32_t ms_group_size(bool weighted) { return weighted ? 64u : 256u; }

// The masks go back to the device's block cache after a call (from where the next
// one takes them) unless they are small: they are up to 13 x 32 bytes per vertex,
// memory that a graph created meanwhile may need.
void ms_done(ptg_ctx *ctx) {
    if (ctx->ws.ms[0].bytes > (256ull << 20)) ctx->ws.ms[0].release();
}

// One group of at most ms_group_size() sources; d_rows receives k rows of n
// values.  Returns false when the fused path does not apply (out-of-core).
bool ms_group(ptg_graph *g, const uint32_t *h_srcs, uint32_t k, uint32_t *d_rows, bool weighted,
              uint32_t flags, RunResult &rr) {
    if (g->out_of_core || k == 0 || k > ms_group_size(weighted)) return false;
    bool o64 = g->off64;
    if (weighted) {
        if (o64) mssssp_impl<unsigned long long>(g, h_srcs, k, d_rows, flags, rr);
        else mssssp_impl<uint32_t>(g, h_srcs, k, d_rows, flags, rr);
    } else {
        // levels go to the rows once, by caller id, from the kept masks
        if (k <= 64) {
            if (o64) msbfs_impl<unsigned long long, 1>(g, h_srcs, k, d_rows, flags, rr);
            else msbfs_impl<uint32_t, 1>(g, h_srcs, k, d_rows, flags, rr);
        } else if (k <= 128) {
            if (o64) msbfs_impl<unsigned long long, 2>(g, h_srcs, k, d_rows, flags, rr);
            else msbfs_impl<uint32_t, 2>(g, h_srcs, k, d_rows, flags, rr);
        } else {
            if (o64) msbfs_impl<unsigned long long, 4>(g, h_srcs, k, d_rows, flags, rr);
            else msbfs_impl<uint32_t, 4>(g, h_srcs, k, d_rows, flags, rr);
        }
    }
    return true;
}

}  // namespace ptg
