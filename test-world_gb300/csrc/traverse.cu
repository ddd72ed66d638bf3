// traverse.cu - frontier traversal engine: BFS (direction-optimizing), SSSP
// (near/far buckets over integer atomicMin), CC min-label propagation, and the
// out-of-core partition streamer they share.
//
// Reference path replaced (ptGraph/main.cu):
//   bfsCaculateInOpt 1180-1418, bfsCaculateInAsync 1420-1678,
//   bfsCaculateInAsyncSwap 1681-2059, bfsCaculateInShare 1041-1123,
//   ssspCaculateInOpt 678-889, ssspCaculateInShare 563-638,
//   ccCaculateInOpt 222-440, ccCaculateInShare 961-1035.
// Kernels replaced (ptGraph/gpu_kernels.cu): the relax kernels 118-448 (one
// atomicMin + label per improved target), the compaction kernels 3-116 plus
// Thrust reduce/exclusive_scan over all n vertices every round, and the
// fragment kernels 450-485.
//
// Graphs whose edges are all in HBM run in one launch (resident.cu); what
// follows is for graphs with streamed partitions.
//
// What changes on GB300:
//  * The next frontier is a bitmap: the relax kernel's improvements set bits
//    with fire-and-forget atomic reductions (no return value awaited), and
//    k_compact turns the bitmap into a queue in one pass over its words
//    (n/8 bytes), so no O(n) label scan over 4-byte labels is needed per
//    round (reference: setLabeling + Thrust scan + compaction over n).
//  * Edges are expanded load-balanced: the frontier's degrees are scanned,
//    and each 256-thread CTA takes a 2048-edge tile of the flattened edge
//    space (k_tile_rows precomputes each tile's first row).  A thread owns 8
//    consecutive edge slots, walks the rows they cross in registers and keeps
//    8 loads in flight; the column stream is read with an L2 evict-first
//    policy.  A hub's edges spread over many CTAs (reference: one thread
//    walks a whole adjacency list, gpu_kernels.cu:126).
//  * SSSP with a bucket width keeps a near frontier below a moving threshold
//    and a far pile above it.
//  * Edges past the resident prefix live in pinned host memory
//    and are cut into fixed-size partitions.  Each round the active edges of
//    every partition are counted.  Mostly active partitions are copied
//    (cudaMemcpyAsync on a copy stream into 2-3 staging buffers, ordered with
//    events) and relaxed edge-centrically, those with few active edges are read
//    in place by a kernel, row by row, and the rest are skipped (reference: 20
//    CPU threads gather active adjacency into a unified-memory buffer the GPU
//    page-faults on, main.cu:1126-1156, 1336-1378).  The count is on the host
//    while the resident edges are relaxed, so copies start meanwhile.  SSSP of
//    a directed RMAT-22 with half of its edges streamed: 11.6 -> 4.8 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

#include "frontier.cuh"

namespace ptg {
namespace {

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void k_fill_u32(uint32_t *a, uint64_t n, uint32_t v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        a[i] = v;
}

__global__ void k_iota_u32(uint32_t *a, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        a[i] = (uint32_t)i;
}

__global__ void k_fill_bits(uint32_t *bm, uint64_t n) {
    uint64_t words = (n + 31) / 32;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < words;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t left = n - i * 32;
        bm[i] = left >= 32 ? 0xffffffffu : ((1u << left) - 1u);
    }
}

// Seed a single-source frontier.
__global__ void k_seed(uint32_t *value, uint32_t src, uint32_t base, uint32_t *q, uint32_t *bm, TravCtl *ctl) {
    value[src] = base;
    q[0] = src;
    bm[src >> 5] |= 1u << (src & 31u);
    ctl->F = 1;
}

// Where a relaxation pushes.  The next frontier is a bitmap; its queue is
// built afterwards by k_compact, so no relaxation waits for an atomic's
// result: the updates below compile to fire-and-forget reductions.
struct PushTargets {
    uint32_t *value;
    uint32_t *bm_next;
    uint32_t *far_bm;  // near/far SSSP: vertices parked above the threshold (nullptr: none)
    TravCtl *ctl;
};

// Relax one edge whose candidate nd beat the probed value of v: the
// reference's rule (gpu_kernels.cu:126-131) as a reduction, then v joins the
// near frontier, or the far pile if nd is at or above the threshold.  When
// another thread improved v further in between, v is still active, so the
// extra mark is harmless.
__device__ __forceinline__ void relax(const PushTargets &t, uint32_t v, uint32_t nd,
                                      uint32_t threshold) {
    atomicMin(&t.value[v], nd);
    uint32_t bit = 1u << (v & 31u);
    if (nd < threshold || t.far_bm == nullptr) atomicOr(&t.bm_next[v >> 5], bit);
    else atomicOr(&t.far_bm[v >> 5], bit);
}

__device__ __forceinline__ void relax_probe(const PushTargets &t, uint32_t v, uint32_t nd,
                                            uint32_t threshold) {
    if (nd < t.value[v]) relax(t, v, nd, threshold);
}

// Vertex of set bit r of a warp's 32 bitmap words (word wd0 + lane in lane
// `lane`, pre = inclusive popcount prefix over the lanes); every lane calls
// it, each with its own r < the warp's total.
__device__ __forceinline__ uint32_t warp_bit_vertex(uint32_t word, uint32_t pre, uint64_t wd0, uint32_t r) {
    uint32_t lo = 0;  // first lane whose inclusive prefix exceeds r
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1) {
        const uint32_t x = __shfl_sync(0xffffffffu, pre, lo + step - 1);
        if (x <= r) lo += step;
    }
    lo = min(lo, 31u);
    const uint32_t w = __shfl_sync(0xffffffffu, word, lo);
    const uint32_t ex = __shfl_sync(0xffffffffu, pre, lo) - __popc(w);
    return (uint32_t)((wd0 + lo) * 32 + __fns(w, 0, (int)(r - ex) + 1));
}

__device__ __forceinline__ void compact_body(const uint32_t *bm, uint64_t words, uint32_t *q, TravCtl *ctl,
                                             uint32_t *far_bm);

// Builds the frontier queue from its bitmap (a warp per 32 words, one atomic
// per CTA step for the CTA's place in the queue: a per-warp atomic on the one
// tail counter serialised dense levels) and takes near vertices out of the far
// pile (SSSP).
// `clear` (this level's frontier bitmap, read by nothing after this kernel)
// is zeroed for reuse as the level after next's bitmap; with `advance` the
// last CTA to finish ends the level: the next frontier's size becomes the
// current one and the counter restarts.
__global__ void __launch_bounds__(kBlock) k_compact(const uint32_t *bm, uint64_t words, uint32_t *q, TravCtl *ctl,
                                                    uint32_t *far_bm, uint32_t *clear, int advance) {
    if (clear)
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < words;
             i += (uint64_t)gridDim.x * blockDim.x)
            clear[i] = 0u;
    compact_body(bm, words, q, ctl, far_bm);
    if (advance) {
        __syncthreads();  // this CTA's counter updates are issued
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&ctl->compact_done, 1u) == gridDim.x - 1) {
                __threadfence();
                ctl->F = atomicExch(&ctl->next_tail, 0u);
                ctl->compact_done = 0u;
            }
        }
    }
}

// The queue of the set bits of bm (vertex order), its size added to
// ctl->next_tail.
__device__ __forceinline__ void compact_body(const uint32_t *bm, uint64_t words, uint32_t *q, TravCtl *ctl,
                                             uint32_t *far_bm) {
    constexpr int kWarps = kBlock / 32;
    __shared__ uint32_t s_warp[kWarps];
    __shared__ uint32_t s_base;
    const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
    const uint64_t step = (uint64_t)gridDim.x * kWarps;
    for (uint64_t c0 = (uint64_t)blockIdx.x * kWarps; c0 * 32 < words; c0 += step) {
        uint64_t wd = (c0 + wid) * 32 + lane;
        uint32_t word = wd < words ? bm[wd] : 0u;
        if (word && far_bm) far_bm[wd] &= ~word;
        uint32_t cnt = __popc(word), pre = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= (unsigned)o) pre += y;
        }
        if (lane == 31) s_warp[wid] = pre;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t run = 0;
            for (int w = 0; w < kWarps; w++) {
                uint32_t t = s_warp[w];
                s_warp[w] = run;
                run += t;
            }
            s_base = run ? atomicAdd(&ctl->next_tail, run) : 0u;
        }
        __syncthreads();
        const uint32_t wbase = s_base + s_warp[wid];
        const uint32_t wtotal = __shfl_sync(0xffffffffu, pre, 31);
        __syncthreads();  // s_warp / s_base are rewritten by the next step
        // the warp's set bits in vertex order, 32 at a time (bit r to lane
        // r % 32): coalesced queue stores
        const uint64_t wd0 = (c0 + wid) * 32;
        for (uint32_t r0 = 0; r0 < wtotal; r0 += 32) {  // warp-uniform bound
            const uint32_t r = r0 + lane;
            const uint32_t v = warp_bit_vertex(word, pre, wd0, r < wtotal ? r : 0u);
            if (r < wtotal) q[wbase + r] = v;
        }
    }
}

// Load-balanced top-down expansion of the frontier's (resident) edges.
// mode: 0 BFS (+1), 1 SSSP (+w), 2 CC (propagate value).
// Each CTA takes a 2048-edge tile of the flattened frontier edge space and
// each thread 8 consecutive edge slots of it: one binary search (in shared
// memory) finds the row of its first slot, later slots advance the row with
// a register compare.  A thread loads all 8 targets (and weights) before it
// probes any of them, keeping 8 independent memory chains in flight; edge
// loads go through L1 (the 32 threads of a warp cover 1 KB of consecutive
// edges) with an L2 evict-first hint.
constexpr int kExpandPerThread = kTile / kBlock;
constexpr int kStageRows = (kTile + 2 + kBlock - 1) / kBlock;  // rows (+1 sentinel) a thread stages
template <class OffT, int MODE>
__global__ void __launch_bounds__(kBlock, 4) k_expand(const uint32_t *q, const OffT *sc, const OffT *rs,
                                                   const uint32_t *tr, const uint32_t *col,
                                                   const uint32_t *w, PushTargets t) {
    __shared__ OffT s_sc[kTile + 2];
    __shared__ OffT s_rs[kTile + 2];
    __shared__ uint32_t s_val[kTile + 2];
    const TravCtl *ctl = t.ctl;
    uint64_t E = ctl->E;
    uint32_t thr = ctl->threshold;
    uint64_t ntiles = (E + kTile - 1) / kTile;
    const uint64_t pol = l2_evict_first_policy();
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint64_t t0 = tile * kTile, t1 = min(E, t0 + kTile);
        uint32_t len = (uint32_t)(t1 - t0);
        // rows r0..r1 cover the tile (r1 may start exactly at t1: one spare row)
        uint64_t r0 = tr[tile];
        uint32_t nrows = (uint32_t)((uint64_t)tr[tile + 1] - r0 + 1);
        if (nrows <= (uint32_t)kTile + 1) {
            // stage the tile's rows (scan values, row starts, source values);
            // a thread's row loads go out together, then its value loads (a
            // tile of short rows has up to 2049 rows, 9 per thread, and one
            // round trip per row and load kind left it latency-bound)
            OffT scv[kStageRows], rsv[kStageRows];
            uint32_t qv[kStageRows];
#pragma unroll
            for (int i = 0; i < kStageRows; i++) {
                const uint32_t k = threadIdx.x + i * kBlock;
                scv[i] = k <= nrows ? sc[r0 + k] : (OffT)0;
                rsv[i] = k < nrows ? rs[r0 + k] : (OffT)0;
                qv[i] = k < nrows ? q[r0 + k] : 0u;
            }
            uint32_t vv[kStageRows];
#pragma unroll
            for (int i = 0; i < kStageRows; i++)
                vv[i] = threadIdx.x + i * kBlock < nrows ? t.value[qv[i]] : 0u;
#pragma unroll
            for (int i = 0; i < kStageRows; i++) {
                const uint32_t k = threadIdx.x + i * kBlock;
                if (k <= nrows) s_sc[k] = scv[i];
                if (k < nrows) {
                    s_rs[k] = rsv[i];
                    s_val[k] = vv[i];
                }
            }
            __syncthreads();
            uint32_t s0 = threadIdx.x * kExpandPerThread;
            if (s0 < len) {
                uint64_t j0 = t0 + s0;
                uint32_t row = (uint32_t)last_le(s_sc, 0, nrows, j0);
                uint64_t next = (uint64_t)s_sc[row + 1];
                OffT delta = s_rs[row] - s_sc[row];  // edge index = delta + slot (mod 2^bits)
                uint32_t uval = s_val[row];
                uint32_t v[kExpandPerThread], nd[kExpandPerThread];
#pragma unroll
                for (int b = 0; b < kExpandPerThread; b++) {
                    uint64_t j = j0 + b;
                    v[b] = PTG_UNREACHED;
                    nd[b] = PTG_UNREACHED;
                    if (s0 + b < len) {
                        while (j >= next) {  // next row (skips zero-degree rows)
                            row++;
                            next = (uint64_t)s_sc[row + 1];
                            delta = s_rs[row] - s_sc[row];
                            uval = s_val[row];
                        }
                        uint64_t e = (uint64_t)(OffT)(delta + (OffT)j);
                        v[b] = ld_edge(col + e, pol);
                        nd[b] = MODE == 0 ? uval + 1u : (MODE == 1 ? uval + ld_edge(w + e, pol) : uval);
                    }
                }
                {
                    uint32_t cur[kExpandPerThread];
#pragma unroll
                    for (int b = 0; b < kExpandPerThread; b++)
                        cur[b] = v[b] != PTG_UNREACHED ? t.value[v[b]] : 0u;
#pragma unroll
                    for (int b = 0; b < kExpandPerThread; b++)
                        if (nd[b] < cur[b]) relax(t, v[b], nd[b], thr);
                }
            }
        } else {
            // more rows than slots (zero-degree rows): search each edge's row
            for (uint64_t j = t0 + threadIdx.x; j < t1; j += kBlock) {
                uint64_t row = last_le(sc, r0, r0 + nrows, j);
                uint64_t e = (uint64_t)rs[row] + (j - (uint64_t)sc[row]);
                uint32_t uval = t.value[q[row]];
                uint32_t v = __ldcs(col + e);
                uint32_t nd = MODE == 0 ? uval + 1u : (MODE == 1 ? uval + __ldcs(w + e) : uval);
                relax_probe(t, v, nd, thr);
            }
        }
        __syncthreads();
    }
}

// Sum and least of the resident edge weights (out[0], out[1]).
__global__ void __launch_bounds__(kBlock) k_weight_sum(const uint32_t *w, uint64_t m, unsigned long long *out) {
    unsigned long long s = 0;
    uint32_t least = 0xFFFFFFFFu;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        s += w[i];
        least = min(least, w[i]);
    }
    s = block_reduce_sum(s);
    if (threadIdx.x == 0 && s) atomicAdd(out, s);
    least = __reduce_min_sync(0xffffffffu, least);
    if (lane_id() == 0) atomicMin(out + 1, (unsigned long long)least);
}

constexpr uint64_t kHotSmemParts = 4096;  // partitions counted in shared memory by k_mark_partitions

// Out-of-core: mark the streamed partitions that hold edges of frontier
// vertices (the reference's setFragmentData, gpu_kernels.cu:450-462, which
// flags 4096-edge fragments of active vertices).
template <class OffT>
__global__ void k_mark_partitions(const uint32_t *q, const TravCtl *ctl, const OffT *off,
                                  uint64_t resident_edges, uint64_t part_edges, uint64_t nparts,
                                  unsigned long long *hits) {
    // hits: edges of frontier vertices per partition this level, summed per
    // CTA in shared memory when the partition count allows (the dynamic shared
    // size is then nparts * 8)
    extern __shared__ unsigned long long s_hits[];
    const bool local = nparts <= kHotSmemParts;
    if (local) {
        for (uint64_t i = threadIdx.x; i < nparts; i += blockDim.x) s_hits[i] = 0;
        __syncthreads();
    }
    uint64_t F = ctl->F;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < F;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t u = q[i];
        uint64_t b = off[u], e = off[u + 1];
        if (e <= resident_edges || e <= b) continue;
        if (b < resident_edges) b = resident_edges;
        uint64_t p0 = b / part_edges, p1 = (e - 1) / part_edges;
        for (uint64_t p = p0; p <= p1 && p < nparts; p++) {
            uint64_t lo = max(b, p * part_edges), hi = min(e, (p + 1) * part_edges);
            if (local) atomicAdd(&s_hits[p], (unsigned long long)(hi - lo));
            else atomicAdd(&hits[p], (unsigned long long)(hi - lo));
        }
    }
    if (local) {
        __syncthreads();
        for (uint64_t i = threadIdx.x; i < nparts; i += blockDim.x)
            if (s_hits[i]) atomicAdd(&hits[i], s_hits[i]);
    }
}

// A source vertex is active in a streamed partition if it is in this
// level's frontier or, for SSSP and label propagation (which converge under
// any order), if it improved earlier in this level: partitions streamed later
// in a level then see the improvements of earlier ones (Gauss-Seidel order),
// so fewer levels, and fewer re-copies, are needed.  Such a vertex stays in
// the next frontier as well.  BFS keeps level-synchronous order (a vertex
// found in this level must not pass on this level's value).
template <int MODE>
__device__ __forceinline__ bool part_active(const uint32_t *bm_cur, const PushTargets &t, uint32_t u) {
    return bit_test(bm_cur, u) || (MODE != 0 && bit_test(t.bm_next, u));
}

__device__ __forceinline__ uint32_t ld_host(const HostEdges &h, uint64_t x) {
    return __ldcs((x < h.lo ? h.head : x >= h.hi ? h.tail : h.mid) + x);
}

// Out-of-core: relaxes the frontier's streamed edges where they lie in host
// memory, in the partitions that `direct` names, so that only their rows cross
// the link.  Tiles of the scanned rows as k_expand, but a warp reads neighbouring
// edges with each load, so a row arrives in whole sectors.  Bound by the link:
// 160-200 GB/s on RMAT rows of 16 edges, where copies reach 211.
template <class OffT, int MODE>
__global__ void __launch_bounds__(kBlock) k_expand_host(const uint32_t *q, const OffT *sc, const OffT *rs,
                                                        const uint32_t *tr, HostEdges col, HostEdges w,
                                                        const uint8_t *direct, uint64_t part_edges, PushTargets t) {
    const uint64_t E = t.ctl->E, ntiles = (E + kTile - 1) / kTile;
    const uint32_t thr = t.ctl->threshold;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t t1 = min(E, (tile + 1) * kTile), r0 = tr[tile], r1 = (uint64_t)tr[tile + 1] + 1;
        uint64_t e[kItems];
        uint32_t uval[kItems], v[kItems], nd[kItems];
#pragma unroll
        for (int b = 0; b < kItems; b++) {
            const uint64_t j = tile * kTile + b * kBlock + threadIdx.x;
            e[b] = ~0ull;
            uval[b] = 0;
            if (j < t1) {
                const uint64_t row = last_le(sc, r0, r1, j);
                const uint64_t x = (uint64_t)rs[row] + (j - (uint64_t)sc[row]);
                if (direct[x / part_edges]) {
                    e[b] = x;
                    uval[b] = t.value[q[row]];
                }
            }
        }
#pragma unroll
        for (int b = 0; b < kItems; b++) {
            v[b] = e[b] != ~0ull ? ld_host(col, e[b]) : PTG_UNREACHED;
            nd[b] = MODE == 1 && e[b] != ~0ull ? ld_host(w, e[b]) : 0u;
        }
#pragma unroll
        for (int b = 0; b < kItems; b++) {
            if (v[b] == PTG_UNREACHED) continue;
            nd[b] = MODE == 0 ? uval[b] + 1u : uval[b] + nd[b];
            relax_probe(t, v[b], nd[b], thr);
        }
    }
}

// Out-of-core: relax every edge of one staged partition whose source vertex
// is in the frontier bitmap.  Edge-centric tiles; the source row of each edge
// is found by binary search over the tile's offsets (staged in shared memory).
template <class OffT, int MODE>
__global__ void __launch_bounds__(kBlock) k_relax_partition(uint64_t e_begin, uint64_t e_end,
                                                            uint64_t v_first, uint64_t v_last,
                                                            const OffT *off,
                                                            const uint32_t *stage_col,
                                                            const uint32_t *stage_w,
                                                            const uint32_t *bm_cur, PushTargets t) {
    __shared__ OffT s_off[kTile + 2];
    __shared__ uint32_t s_val[kTile + 1];
    uint32_t thr = t.ctl->threshold;
    uint64_t E = e_end - e_begin;
    uint64_t ntiles = (E + kTile - 1) / kTile;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint64_t t0 = e_begin + tile * kTile, t1 = min(e_end, t0 + kTile);
        uint64_t r0 = block_last_le(off, v_first, v_last + 1, t0);
        uint64_t r1 = block_last_le(off, r0, v_last + 1, t1 - 1);
        uint64_t nrows = r1 - r0 + 1;
        bool staged = nrows <= (uint64_t)kTile;
        if (staged) {
            for (uint64_t k = threadIdx.x; k < nrows; k += kBlock) {
                uint32_t u = (uint32_t)(r0 + k);
                s_off[k] = off[u];
                s_val[k] = part_active<MODE>(bm_cur, t, u) ? t.value[u] : PTG_UNREACHED;
            }
            if (threadIdx.x == 0) s_off[nrows] = off[r0 + nrows];
        }
        __syncthreads();
        if (staged) {
            // as k_expand: a thread's 8 consecutive edge slots, one search for
            // the first slot's row, the rest by a register compare; all 8
            // targets (and weights) loaded, then all 8 probes in flight (the
            // value array of a graph that does not fit HBM is far larger than
            // L2, so each probe is a DRAM round trip)
            const uint32_t len = (uint32_t)(t1 - t0), s0 = threadIdx.x * kExpandPerThread;
            if (s0 < len) {
                const uint64_t j0 = t0 + s0;
                uint32_t row = (uint32_t)last_le(s_off, 0, nrows, j0);
                uint64_t next = (uint64_t)s_off[row + 1];
                uint32_t uval = s_val[row];
                uint32_t v[kExpandPerThread], nd[kExpandPerThread];
#pragma unroll
                for (int b = 0; b < kExpandPerThread; b++) {
                    const uint64_t j = j0 + b;
                    v[b] = PTG_UNREACHED;
                    nd[b] = PTG_UNREACHED;
                    if (s0 + b < len) {
                        while (j >= next) {  // next row (skips zero-degree rows)
                            row++;
                            next = (uint64_t)s_off[row + 1];
                            uval = s_val[row];
                        }
                        if (uval != PTG_UNREACHED) {
                            const uint64_t le = j - e_begin;
                            v[b] = __ldcs(stage_col + le);
                            nd[b] = MODE == 0 ? uval + 1u : (MODE == 1 ? uval + __ldcs(stage_w + le) : uval);
                        }
                    }
                }
                uint32_t cur[kExpandPerThread];
#pragma unroll
                for (int b = 0; b < kExpandPerThread; b++) cur[b] = v[b] != PTG_UNREACHED ? t.value[v[b]] : 0u;
#pragma unroll
                for (int b = 0; b < kExpandPerThread; b++)
                    if (nd[b] < cur[b]) relax(t, v[b], nd[b], thr);
            }
        } else {
            // more rows than slots (zero-degree rows): search each edge's row
            for (uint64_t j = t0 + threadIdx.x; j < t1; j += kBlock) {
                uint64_t u = last_le(off, r0, r0 + nrows, j);
                uint32_t uval = part_active<MODE>(bm_cur, t, (uint32_t)u) ? t.value[u] : PTG_UNREACHED;
                if (uval == PTG_UNREACHED) continue;
                uint64_t le = j - e_begin;
                uint32_t v = __ldcs(stage_col + le);
                uint32_t nd = MODE == 0 ? uval + 1u : (MODE == 1 ? uval + __ldcs(stage_w + le) : uval);
                relax_probe(t, v, nd, thr);
            }
        }
        __syncthreads();
    }
}

// Whether every edge carries the same weight both ways: sum over the edges
// u < v of a hash of (u, v, w), less the same over the edges u > v; zero when the
// two lists of (smaller end, larger end, weight) are the same (and, where they
// differ, with a probability of about 2^-64: the hash is keyed with a random
// number per check, as weights can be chosen that defeat a fixed one).  Also the
// weights' sum and minimum, as k_weight_sum.  A warp walks an equal run of edges,
// 8 consecutive ones per lane and step; the rows that begin in a step's 256 edges
// are written at their first edge in shared memory, and a running maximum gives
// each edge its row.  (Tiles of a CTA with a search of their row bounds each: 3.07
// ms on RMAT-24, 1.83 now; half of it is the hash.)
constexpr uint32_t kBalStep = 256;
template <class OffT>
__global__ void __launch_bounds__(kBlock, 4) k_weight_balance(uint64_t m, uint64_t n, const OffT *off, const uint32_t *col,
                                                              const uint32_t *w, unsigned long long key,
                                                              unsigned long long *out) {
    constexpr int kEach = kBalStep / 32;
    __shared__ __align__(16) uint32_t s_row[kBlock / 32][kBalStep];
    uint32_t *rows = s_row[threadIdx.x >> 5];
    const unsigned lane = lane_id();
    const uint64_t warps = (uint64_t)gridDim.x * (kBlock / 32), warp = (uint64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
    const uint64_t share = ((m + warps - 1) / warps + kBalStep - 1) / kBalStep * kBalStep;
    const uint64_t end = min(m, (warp + 1) * share);
    unsigned long long sum = 0, total = 0;
    uint32_t least = 0xFFFFFFFFu, row = 0;  // row: the last that begins at or before the step's first edge
    if (warp * share < end) row = (uint32_t)last_le(off, (uint64_t)0, n, warp * share);
    for (uint64_t t = warp * share; t < end; t += kBalStep) {
        const uint64_t t1 = min(m, t + kBalStep), j0 = t + lane * kEach;
        uint32_t vs[kEach], ws[kEach];
        if (j0 + kEach <= t1) {  // (the arrays start on 256 bytes and j0 is a multiple of 8)
#pragma unroll
            for (int i = 0; i < kEach; i += 4) {
                const uint4 x = *reinterpret_cast<const uint4 *>(col + j0 + i), y = *reinterpret_cast<const uint4 *>(w + j0 + i);
                vs[i] = x.x, vs[i + 1] = x.y, vs[i + 2] = x.z, vs[i + 3] = x.w;
                ws[i] = y.x, ws[i + 1] = y.y, ws[i + 2] = y.z, ws[i + 3] = y.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kEach; i++) {
                vs[i] = j0 + i < t1 ? col[j0 + i] : 0u;
                ws[i] = j0 + i < t1 ? w[j0 + i] : 0xFFFFFFFFu;
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kEach; i += 4) *reinterpret_cast<uint4 *>(rows + lane * kEach + i) = make_uint4(0, 0, 0, 0);
        __syncwarp();
        // 128 row starts at a time: the runs of short rows would otherwise take
        // most of the time, a dependent load per 32 rows
        uint64_t r = (uint64_t)row + 1;
        for (int c = 128; c == 128; r += c) {
            uint64_t x[4];
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = r + 32 * i + lane < n ? (uint64_t)off[r + 32 * i + lane] : t1;
            c = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool in = x[i] < t1;
                // (of several rows that begin at one edge all but the last are empty)
                if (in) atomicMax(&rows[x[i] - t], (uint32_t)(r + 32 * i + lane));
                c += __popc(__ballot_sync(0xffffffffu, in));
            }
        }
        __syncwarp();
        uint32_t at[kEach], last = 0;
#pragma unroll
        for (int i = 0; i < kEach; i++) at[i] = last = max(last, rows[lane * kEach + i]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, last, o);
            if (lane >= (unsigned)o) last = max(last, y);
        }
        uint32_t before = __shfl_up_sync(0xffffffffu, last, 1);
        before = lane ? max(before, row) : row;
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            least = min(least, ws[i]);
            if (j0 + i >= t1) continue;
            const uint32_t u = max(at[i], before), v = vs[i];
            unsigned long long h = (((unsigned long long)min(u, v) << 32 | max(u, v)) ^ key) * 0x9E3779B97F4A7C15ull;
            h = (h ^ (h >> 32) ^ ws[i]) * 0xBF58476D1CE4E5B9ull;
            h = (h ^ (h >> 32)) * 0x94D049BB133111EBull;
            h ^= h >> 32;
            if (u < v) sum += h;
            if (u > v) sum -= h;
            total += ws[i];
        }
        row = (uint32_t)(r - 1);
    }
    sum = block_reduce_sum(sum);
    if (threadIdx.x == 0 && sum) atomicAdd(out, sum);
    __syncthreads();
    total = block_reduce_sum(total);
    if (threadIdx.x == 0 && total) atomicAdd(out + 1, total);
    least = __reduce_min_sync(0xffffffffu, least);
    if (lane == 0) atomicMin(out + 2, (unsigned long long)least);
}

// Near/far: smallest distance in the far pile (a bitmap).
__global__ void __launch_bounds__(kBlock) k_far_min(const uint32_t *far_bm, uint64_t words,
                                                    const uint32_t *value, TravCtl *ctl) {
    uint32_t best = PTG_UNREACHED;
    for (uint64_t wd = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; wd < words;
         wd += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t word = far_bm[wd];
        while (word) {
            int b = __ffs(word) - 1;
            word &= word - 1;
            best = min(best, value[wd * 32 + b]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_down_sync(0xffffffffu, best, o));
    if (lane_id() == 0 && best != PTG_UNREACHED) atomicMin(&ctl->far_min, (unsigned long long)best);
}

// Near/far: move the far vertices below the new threshold into the (empty)
// near frontier bitmap; k_compact then builds its queue.
__global__ void __launch_bounds__(kBlock) k_far_split(uint32_t *far_bm, uint64_t words,
                                                      const uint32_t *value, uint32_t *bm,
                                                      const TravCtl *ctl) {
    uint32_t thr = ctl->threshold;
    for (uint64_t wd = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; wd < words;
         wd += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t word = far_bm[wd];
        if (!word) continue;
        uint32_t moved = 0, rest = word;
        while (rest) {
            int b = __ffs(rest) - 1;
            rest &= rest - 1;
            if (value[wd * 32 + b] < thr) moved |= 1u << b;
        }
        if (moved) {
            far_bm[wd] = word & ~moved;
            bm[wd] |= moved;
        }
    }
}

// Hot-partition cache (the reference's visit-counted fragment promotion,
// gpu_kernels.cu:254-282 and 475-485, where a 4096-edge fragment whose visit
// record exceeds 3600 becomes a swap candidate).  part_visits[p] accumulates
// the edges of frontier vertices that fell in partition p; a partition is hot
// once that exceeds hot_threshold visits per 4096 edges.  A hot partition
// takes a free slot, or the slot of the coldest cached partition if that one
// has fewer visits; a cached partition is relaxed from its slot without a
// copy, in this and every later traversal of the graph.
//
// The slot that hot partition p may take in a round with these active edges per
// partition, -1 if none: not one whose partition the round has yet to use.
int hot_victim(const ptg_graph *g, uint64_t p, uint64_t edges, const unsigned long long *hits) {
    if (g->cache_static) return -1;
    if ((double)g->part_visits[p] * 4096.0 <= (double)g->hot_threshold * (double)edges) return -1;
    int victim = -1;
    for (uint32_t s = 0; s < g->cache_slots; s++) {
        const int64_t q = g->slots[s].part;
        if (q < 0) return (int)s;
        if (hits[q] && (uint64_t)q > p) continue;
        if (victim < 0 || g->part_visits[q] < g->part_visits[g->slots[victim].part]) victim = (int)s;
    }
    return victim >= 0 && g->part_visits[g->slots[victim].part] < g->part_visits[p] ? victim : -1;
}

// The slot of a partition that is copied now: its own, or one that it takes; -1
// to use a staging buffer.
int hot_slot(ptg_graph *g, uint64_t p, uint64_t edges, const unsigned long long *hits) {
    if (g->slot_of[p] >= 0) return g->slot_of[p];
    const int victim = hot_victim(g, p, edges, hits);
    if (victim < 0) return -1;
    HotSlot &hs = g->slots[victim];
    if (hs.part >= 0) g->slot_of[hs.part] = -1;
    uint64_t bytes = g->partition_edges * 4;
    hs.col.ensure(bytes);
    if (g->weighted) hs.w.ensure(bytes);
    hs.part = (int64_t)p;
    hs.has_col = hs.has_w = false;
    g->slot_of[p] = victim;
    return victim;
}

// Whether partition p, of which a round reads few edges (they would be read in
// place), is in a cache slot or takes one now.  A hot partition's edges were about
// all read over the link by then, and it is copied once to end that: into a
// free slot, or one whose partition this round does not use and that was visited
// less than half as often (copying costs more than reading in place, so two
// partitions of about the same use must not take a slot from each other in turn).
bool sparse_slot(ptg_graph *g, uint64_t p, uint64_t edges, const unsigned long long *hits) {
    if (g->slot_of[p] >= 0) return true;
    const int victim = hot_victim(g, p, edges, hits);
    if (victim < 0) return false;
    const int64_t q = g->slots[victim].part;
    if (q >= 0 && (hits[q] || g->part_visits[q] * 2 >= g->part_visits[p])) return false;
    return hot_slot(g, p, edges, hits) >= 0;
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
// Scan of the frontier's degrees, of the edges in [from, to) only: prefix sums
// and row starts in ws.scan / ws.rowstart, and the row that every tile begins in.
template <class OffT>
void scan_frontier(ptg_ctx *ctx, const uint32_t *q, uint64_t F, TravCtl *ctl, const OffT *off, OffT from, OffT to,
                   bool count, uint32_t *tr) {
    constexpr int kScanBlocks = 1024;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    OffT *sc = ws.scan.as<OffT>(), *rs = ws.rowstart.as<OffT>();
    if (F <= kSmallFrontier) {  // one CTA: the scan and the tile rows
        launch(ctx, "k_scan_small", k_scan_small<OffT>, 1, kBlock, 0, st, q, ctl, off, from, to, sc, rs, tr, (int)count);
        return;
    }
    const int blocks = grid_for(F, kBlock, kScanBlocks);
    ws.bsum.ensure(kScanBlocks * 8);
    unsigned long long *bsum = ws.bsum.as<unsigned long long>();
    launch(ctx, "k_scan_reduce", k_scan_reduce<OffT>, blocks, kBlock, 0, st, q, ctl, off, from, to, bsum);
    launch(ctx, "k_scan_bsums", k_scan_bsums, 1, kBlock, 0, st, bsum, blocks, ctl, (int)count);
    launch(ctx, "k_scan_write", k_scan_write<OffT>, blocks, kBlock, 0, st, q, ctl, off, from, to, bsum, sc, rs);
    launch(ctx, "k_tile_rows", k_tile_rows<OffT>, ctx->sm_count * 4, kBlock, 0, st, sc, ctl, tr);
}

void set_weight_stats(ptg_graph *g, unsigned long long sum, uint32_t least) {
    g->mean_weight = std::max(1.0, (double)sum / (double)g->resident_edges);
    g->min_weight = least;
}

// Mean and least resident edge weight, measured once per graph.
void measure_mean_weight(ptg_graph *g) {
    if (g->mean_weight != 0 || g->resident_edges == 0 || !g->weighted) return;
    ptg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    ctx->ws.bsum.ensure(1024 * 8);
    unsigned long long *acc = ctx->ws.bsum.as<unsigned long long>();
    unsigned long long h[2] = {0, 0xFFFFFFFFull};
    PTG_CUDA_TRY(cudaMemcpyAsync(acc, h, 16, cudaMemcpyHostToDevice, st));
    launch(ctx, "k_weight_sum", k_weight_sum, grid_for(g->resident_edges, kBlock, ctx->sm_count * 8), kBlock, 0, st,
           g->d_w.as<uint32_t>(), g->resident_edges, acc);
    PTG_CUDA_TRY(cudaMemcpyAsync(h, acc, 16, cudaMemcpyDeviceToHost, st));
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    set_weight_stats(g, h[0], (uint32_t)h[1]);
}

template <class OffT>
void traverse_impl(ptg_graph *g, TravKind kind, uint32_t src, uint32_t *d_value, uint32_t flags,
                   uint32_t delta, uint32_t max_iters, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n;
    const int sms = ctx->sm_count;
    const uint64_t words = (n + 31) / 32;

    ws.q[0].ensure(n * 4);
    ws.q[1].ensure(n * 4);
    ws.bm[0].ensure(words * 4);
    ws.bm[1].ensure(words * 4);
    ws.scan.ensure((n + 1) * sizeof(OffT));
    ws.rowstart.ensure((n + 1) * sizeof(OffT));
    ws.tiles.ensure((g->resident_edges / kTile + 4) * sizeof(uint32_t));
    ws.ctl.ensure(sizeof(TravCtl));
    ws.h_ctl.ensure(sizeof(TravCtl));
    // Near/far buckets save edge work in HBM; a streamed graph is bound by the
    // host link, and what its rounds read again hardly falls with them, so it
    // relaxes in label-correcting rounds unless a bucket width is asked for
    // (RMAT-24 all streamed: 9 rounds, 3.9 GB over the link and 21.9 ms, with
    // buckets of 32 (mean weight) 18 rounds, 3.7 GB and 22.0 ms).
    const bool use_far = kind == TRAV_SSSP && !(flags & PTG_REFERENCE_SCHEDULE) && delta != 0;
    if (use_far) ws.farbm.ensure(words * 4);
    TravCtl *d_ctl = ws.ctl.as<TravCtl>();
    TravCtl *h_ctl = ws.h_ctl.as<TravCtl>();
    const OffT *off = g->d_off.as<OffT>();
    const uint32_t *col = g->d_col.as<uint32_t>();
    const uint32_t *wt = g->d_w.as<uint32_t>();
    OffT clip = (OffT)g->resident_edges;

    // ---- initial state ----
    TravCtl init{};
    init.threshold = PTG_UNREACHED;
    PTG_CUDA_TRY(cudaMemsetAsync(ws.bm[0].p, 0, words * 4, st));
    PTG_CUDA_TRY(cudaMemsetAsync(ws.bm[1].p, 0, words * 4, st));
    uint32_t base = (flags & PTG_LEVEL_ZERO_BASED) ? 0u : 1u;
    int fill_grid = grid_for(n, kBlock, sms * 8);
    if (kind == TRAV_CCPROP) {
        launch(ctx, "k_iota_u32", k_iota_u32, fill_grid, kBlock, 0, st, d_value, n);
        launch(ctx, "k_iota_u32", k_iota_u32, fill_grid, kBlock, 0, st, ws.q[0].as<uint32_t>(), n);
        launch(ctx, "k_fill_bits", k_fill_bits, grid_for(words, kBlock, sms * 8), kBlock, 0, st,
               ws.bm[0].as<uint32_t>(), n);
        init.F = (uint32_t)n;
    } else {
        launch(ctx, "k_fill_u32", k_fill_u32, fill_grid, kBlock, 0, st, d_value, n, PTG_UNREACHED);
        init.F = 1;
        if (use_far) {
            init.threshold = bucket_end(base, delta);
            PTG_CUDA_TRY(cudaMemsetAsync(ws.farbm.p, 0, words * 4, st));
        }
    }
    PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &init, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
    if (kind != TRAV_CCPROP)
        launch(ctx, "k_seed", k_seed, 1, 1, 0, st, d_value, src, base, ws.q[0].as<uint32_t>(),
               ws.bm[0].as<uint32_t>(), d_ctl);
    PTG_CUDA_TRY(cudaGetLastError());

    int cur = 0;
    uint64_t F = init.F;
    bool far_nonempty = false;
    const int compact_grid = grid_for((words + 31) / 32, kBlock / 32, sms * 8);
    uint32_t threshold = init.threshold;
    if (max_iters == 0) max_iters = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, 4 * n + 16);

    bool link_open = false;  // a level's copies were recorded between link_ev[0] and link_ev[1]
    // per level and partition: active edges, and whether they are read in place
    const uint64_t P = g->num_partitions;
    ws.flags.ensure(P * 9);
    ws.h_flags.ensure(P * 9);
    unsigned long long *h_hits = ws.h_flags.as<unsigned long long>();
    uint8_t *h_direct = reinterpret_cast<uint8_t *>(h_hits + P);
    unsigned long long *d_hits = ws.flags.as<unsigned long long>();
    uint8_t *d_direct = reinterpret_cast<uint8_t *>(d_hits + P);
    const bool need_w = kind == TRAV_SSSP;
    int stage_next = 0;

    while (true) {
        if (F == 0) {
            if (!use_far || !far_nonempty) break;
            // advance the threshold past the smallest far distance
            unsigned long long big = ~0ull;
            PTG_CUDA_TRY(cudaMemcpyAsync(&d_ctl->far_min, &big, 8, cudaMemcpyHostToDevice, st));
            launch(ctx, "k_far_min", k_far_min, grid_for(words, kBlock, sms * 8), kBlock, 0, st,
                   (const uint32_t *)ws.farbm.as<uint32_t>(), words, (const uint32_t *)d_value, d_ctl);
            PTG_CUDA_TRY(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(TravCtl), cudaMemcpyDeviceToHost, st));
            PTG_CUDA_TRY(cudaStreamSynchronize(st));
            if (h_ctl->far_min == ~0ull) break;  // far pile empty
            threshold = bucket_end(h_ctl->far_min, delta);
            TravCtl upd = *h_ctl;
            upd.threshold = threshold;
            upd.next_tail = 0;
            PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &upd, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
            // bm[cur] is clear (it was the previous round's empty next bitmap)
            launch(ctx, "k_far_split", k_far_split, grid_for(words, kBlock, sms * 8), kBlock, 0, st,
                   ws.farbm.as<uint32_t>(), words, (const uint32_t *)d_value, ws.bm[cur].as<uint32_t>(),
                   (const TravCtl *)d_ctl);
            launch(ctx, "k_compact", k_compact, compact_grid, kBlock, 0, st,
                   (const uint32_t *)ws.bm[cur].as<uint32_t>(), words, ws.q[cur].as<uint32_t>(), d_ctl,
                   (uint32_t *)nullptr, (uint32_t *)nullptr, 0);
            PTG_CUDA_TRY(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(TravCtl), cudaMemcpyDeviceToHost, st));
            PTG_CUDA_TRY(cudaStreamSynchronize(st));
            F = h_ctl->next_tail;
            upd = *h_ctl;
            upd.F = (uint32_t)F;
            upd.next_tail = 0;
            PTG_CUDA_TRY(cudaMemcpyAsync(d_ctl, &upd, sizeof(TravCtl), cudaMemcpyHostToDevice, st));
            continue;
        }
        if (rr.iterations >= max_iters) throw Error{PTG_ERR_TIMEOUT, "iteration limit reached"};
        rr.iterations++;
        uint32_t *q_cur = ws.q[cur].as<uint32_t>(), *q_nxt = ws.q[cur ^ 1].as<uint32_t>();
        uint32_t *bm_cur = ws.bm[cur].as<uint32_t>(), *bm_nxt = ws.bm[cur ^ 1].as<uint32_t>();
        // bm_nxt is clear: zeroed at the start, then by each level's
        // compaction as the bitmap it had just finished with
        PushTargets pt{d_value, bm_nxt, use_far ? ws.farbm.as<uint32_t>() : nullptr, d_ctl};
        uint32_t *tr = ws.tiles.as<uint32_t>();
        // which partitions hold active edges: known on the host while the
        // resident edges are relaxed, so that copies start meanwhile
        PTG_CUDA_TRY(cudaMemsetAsync(d_hits, 0, P * 8, st));
        launch(ctx, "k_mark_partitions", k_mark_partitions<OffT>, grid_for(F, kBlock, sms * 8), kBlock,
               P <= kHotSmemParts ? P * 8 : 0, st, q_cur, d_ctl, off, g->resident_edges, g->partition_edges, P, d_hits);
        PTG_CUDA_TRY(cudaMemcpyAsync(h_hits, d_hits, P * 8, cudaMemcpyDeviceToHost, st));
        PTG_CUDA_TRY(cudaEventRecord(g->hits_ready, st));
        scan_frontier<OffT>(ctx, q_cur, F, d_ctl, off, (OffT)0, clip, true, tr);
        OffT *sc = ws.scan.as<OffT>(), *rs = ws.rowstart.as<OffT>();
        const int eg = sms * (int)ctx->tuning.expand_ctas_per_sm;
        if (kind == TRAV_BFS)
            launch(ctx, "k_expand_bfs", k_expand<OffT, 0>, eg, kBlock, 0, st, q_cur, sc, rs, tr, col, wt, pt);
        else if (kind == TRAV_SSSP)
            launch(ctx, "k_expand_sssp", k_expand<OffT, 1>, eg, kBlock, 0, st, q_cur, sc, rs, tr, col, wt, pt);
        else
            launch(ctx, "k_expand_cc", k_expand<OffT, 2>, eg, kBlock, 0, st, q_cur, sc, rs, tr, col, wt, pt);
        PTG_CUDA_TRY(cudaGetLastError());
        {
            // stream the active partitions past the resident prefix
            const bool hot = g->cache_slots > 0;
            PTG_CUDA_TRY(cudaEventSynchronize(g->hits_ready));
            link_open = false;
            // A partition of which at most three quarters are active is read in
            // place, else copied.  SSSP of directed RMAT graphs with the line at
            // (never, 1/4, 1/2, 3/4, 7/8, always): RMAT-22 half streamed 10.9,
            // 6.2, 4.9, 4.8, 4.8, 5.2 ms; RMAT-24 all streamed 55, 26.6, 21.9,
            // 21.4, 21.4, 23.3 ms; BFS of the former 4.5, 2.0, 1.9, 1.9, 1.9, 1.9.
            const bool readable = g->in_place[0].mid && (!need_w || g->in_place[1].mid);
            uint64_t active = 0, direct = 0;  // streamed edges of the frontier; those read in place
            uint64_t spared = 0;              // edges that are not copied for that
            for (uint64_t p = g->resident_partitions; p < P && hot; p++) g->part_visits[p] += h_hits[p];
            for (uint64_t p = g->resident_partitions; p < P; p++) {
                const uint64_t e0 = p * g->partition_edges, e1 = std::min<uint64_t>(g->m, e0 + g->partition_edges);
                // (what is in a cache slot, or is copied into one now, needs no link)
                h_direct[p] = h_hits[p] && h_hits[p] * 4 <= (e1 - e0) * 3 && readable &&
                              !(hot && sparse_slot(g, p, e1 - e0, h_hits));
                rr.parts_skipped += !h_hits[p];
                active += h_hits[p];
                if (h_direct[p]) {
                    direct += h_hits[p];
                    spared += e1 - e0 - h_hits[p];
                }
            }
            // the kernel walks the other partitions' active edges too, more than
            // four times as fast as the link would bring the spared ones
            if (spared * 4 < active) {
                std::memset(h_direct + g->resident_partitions, 0, P - g->resident_partitions);
                direct = 0;
            }
            for (uint64_t p = g->resident_partitions; p < P; p++) rr.parts_streamed += h_direct[p];
            if (direct) {
                ws.tiles.ensure((active / kTile + 4) * sizeof(uint32_t));
                tr = ws.tiles.as<uint32_t>();
                std::memset(h_direct, 0, g->resident_partitions);
                PTG_CUDA_TRY(cudaMemcpyAsync(d_direct, h_direct, P, cudaMemcpyHostToDevice, st));
                scan_frontier<OffT>(ctx, q_cur, F, d_ctl, off, clip, (OffT)g->m, false, tr);
                PTG_CUDA_TRY(cudaEventRecord(g->link_ev[0], st));
                link_open = true;
                const int hg = grid_for(active, kTile, sms * 8);
                if (kind == TRAV_BFS)
                    launch(ctx, "k_expand_host_bfs", k_expand_host<OffT, 0>, hg, kBlock, 0, st, q_cur, sc, rs, tr,
                           g->in_place[0], g->in_place[1], d_direct, g->partition_edges, pt);
                else if (kind == TRAV_SSSP)
                    launch(ctx, "k_expand_host_sssp", k_expand_host<OffT, 1>, hg, kBlock, 0, st, q_cur, sc, rs, tr,
                           g->in_place[0], g->in_place[1], d_direct, g->partition_edges, pt);
                else
                    launch(ctx, "k_expand_host_cc", k_expand_host<OffT, 2>, hg, kBlock, 0, st, q_cur, sc, rs, tr,
                           g->in_place[0], g->in_place[1], d_direct, g->partition_edges, pt);
                PTG_CUDA_TRY(cudaGetLastError());
                PTG_CUDA_TRY(cudaEventRecord(g->direct_done, st));
                rr.link_bytes += direct * (need_w ? 8 : 4);
            }
            cudaStream_t cs = ctx->copy_stream;
            for (uint64_t p = g->resident_partitions; p < P; p++) {
                if (!h_hits[p] || h_direct[p]) continue;
                uint64_t e0 = p * g->partition_edges;
                uint64_t e1 = std::min<uint64_t>(g->m, e0 + g->partition_edges);
                const uint32_t *sc_ = nullptr, *sw_ = nullptr;
                const int slot = hot ? hot_slot(g, p, e1 - e0, h_hits) : -1;
                // a partition copies into a cache slot (kept for later levels and
                // queries) or into the next staging buffer
                bool copy_col = true, copy_w = need_w;
                void *dcol, *dw;
                cudaEvent_t ready, freed;
                if (slot >= 0) {
                    HotSlot &hs = g->slots[slot];
                    copy_col = !hs.has_col;
                    copy_w = need_w && !hs.has_w;
                    dcol = hs.col.p;
                    dw = hs.w.p;
                    ready = hs.ready;
                    freed = hs.freed;
                    if (!copy_col && !copy_w) rr.parts_cached++;
                } else {
                    int b = stage_next;
                    stage_next = (stage_next + 1) % (int)g->n_stage;
                    dcol = g->stage_col[b].p;
                    dw = g->stage_w[b].p;
                    ready = g->stage_ready[b];
                    freed = g->stage_free[b];
                }
                if (copy_col || copy_w) {
                    PTG_CUDA_TRY(cudaStreamWaitEvent(cs, freed, 0));
                    if (!link_open) {
                        PTG_CUDA_TRY(cudaEventRecord(g->link_ev[0], cs));
                        link_open = true;
                    }
                    if (copy_col) {
                        stream_edges(g, 0, dcol, e0, e1, cs);
                        rr.link_bytes += (e1 - e0) * 4;
                    }
                    if (copy_w) {
                        stream_edges(g, 1, dw, e0, e1, cs);
                        rr.link_bytes += (e1 - e0) * 4;
                    }
                    PTG_CUDA_TRY(cudaEventRecord(ready, cs));
                    PTG_CUDA_TRY(cudaStreamWaitEvent(st, ready, 0));
                    rr.parts_streamed++;
                    if (slot >= 0) {
                        g->slots[slot].has_col = true;
                        g->slots[slot].has_w |= copy_w;
                    }
                }
                sc_ = static_cast<const uint32_t *>(dcol);
                sw_ = static_cast<const uint32_t *>(dw);
                uint64_t vf = g->part_first_vertex[p], vl = g->part_first_vertex[p + 1];
                int pg = grid_for(e1 - e0, kTile, sms * 8);
                if (kind == TRAV_BFS)
                    launch(ctx, "k_relax_partition_bfs", k_relax_partition<OffT, 0>, pg, kBlock, 0, st, e0,
                           e1, vf, vl, off, sc_, sw_, bm_cur, pt);
                else if (kind == TRAV_SSSP)
                    launch(ctx, "k_relax_partition_sssp", k_relax_partition<OffT, 1>, pg, kBlock, 0, st, e0,
                           e1, vf, vl, off, sc_, sw_, bm_cur, pt);
                else
                    launch(ctx, "k_relax_partition_cc", k_relax_partition<OffT, 2>, pg, kBlock, 0, st, e0,
                           e1, vf, vl, off, sc_, sw_, bm_cur, pt);
                PTG_CUDA_TRY(cudaGetLastError());
                PTG_CUDA_TRY(cudaEventRecord(freed, st));
            }
            if (direct) PTG_CUDA_TRY(cudaStreamWaitEvent(cs, g->direct_done, 0));
            if (link_open) PTG_CUDA_TRY(cudaEventRecord(g->link_ev[1], cs));
        }
        // next frontier: queue from the bitmap; its last CTA ends the level in
        // the control block
        launch(ctx, "k_compact", k_compact, compact_grid, kBlock, 0, st, (const uint32_t *)bm_nxt, words, q_nxt, d_ctl,
               use_far ? ws.farbm.as<uint32_t>() : (uint32_t *)nullptr, bm_cur, 1);
        PTG_CUDA_TRY(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(TravCtl), cudaMemcpyDeviceToHost, st));
        PTG_CUDA_TRY(cudaStreamSynchronize(st));
        const uint32_t level_error = h_ctl->error;
        F = h_ctl->F;
        PTG_REQUIRE(level_error == 0, PTG_ERR_CUDA, "frontier overflow in relax");
        if (link_open) {
            // the level's copies and reads in place, first start to last end (the
            // compute stream waited on every one of them before the sync
            // above; the event that follows them on the copy stream is due)
            float lms = 0.f;
            PTG_CUDA_TRY(cudaEventSynchronize(g->link_ev[1]));
            PTG_CUDA_TRY(cudaEventElapsedTime(&lms, g->link_ev[0], g->link_ev[1]));
            rr.link_ms += lms;
            link_open = false;
        }
        if (use_far) far_nonempty = true;
        cur ^= 1;
    }
    PTG_CUDA_TRY(cudaMemcpyAsync(h_ctl, d_ctl, sizeof(TravCtl), cudaMemcpyDeviceToHost, st));
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    rr.edges_relaxed = h_ctl->edges_done;
}

}  // namespace

// One launch for a graph whose edges are all in HBM (resident.cu).
void build_nonzero_bits(ptg_graph *g);
void run_resident(ptg_graph *g, TravKind kind, uint32_t src, uint32_t *d_value, uint32_t base, uint32_t delta,
                  bool allow_pull, uint32_t max_iters, RunResult &rr);

// Builds the per-graph tables the single-source traversals would otherwise
// build on first use (vertices with edges, SSSP bucket width).
void trav_prepare_graph(ptg_graph *g) {
    if (g->out_of_core) return;
    if (g->symmetric) build_nonzero_bits(g);
    measure_mean_weight(g);
}

bool graph_weights_symmetric(ptg_graph *g) {
    if (g->weights_symmetric < 0) {
        g->weights_symmetric = 0;
        if (g->symmetric && g->weighted && !g->out_of_core && g->m) {
            ptg_ctx *ctx = g->ctx;
            cudaStream_t st = ctx->stream;
            ctx->ws.bsum.ensure(1024 * 8);
            unsigned long long *acc = ctx->ws.bsum.as<unsigned long long>();
            unsigned long long h[3] = {0, 0, 0xFFFFFFFFull};
            PTG_CUDA_TRY(cudaMemcpyAsync(acc, h, 24, cudaMemcpyHostToDevice, st));
            const int grid = grid_for(g->m, kTile, ctx->sm_count * 4);
            std::random_device rd;
            const unsigned long long key = (unsigned long long)rd() << 32 | rd();
            if (g->off64)
                launch(ctx, "k_weight_balance", k_weight_balance<unsigned long long>, grid, kBlock, 0, st, g->m, g->n,
                       g->d_off.as<unsigned long long>(), g->d_col.as<uint32_t>(), g->d_w.as<uint32_t>(), key, acc);
            else
                launch(ctx, "k_weight_balance", k_weight_balance<uint32_t>, grid, kBlock, 0, st, g->m, g->n,
                       g->d_off.as<uint32_t>(), g->d_col.as<uint32_t>(), g->d_w.as<uint32_t>(), key, acc);
            PTG_CUDA_TRY(cudaMemcpyAsync(h, acc, 24, cudaMemcpyDeviceToHost, st));
            PTG_CUDA_TRY(cudaStreamSynchronize(st));
            set_weight_stats(g, h[1], (uint32_t)h[2]);
            g->weights_symmetric = h[0] == 0;
        }
    }
    return g->weights_symmetric == 1;
}


// Default SSSP bucket width of an in-HBM graph: the tuned multiple (0.75) of
// the mean edge weight, a quarter of that from 2^25 edges on and up to 4 times
// it as the graph shrinks.  Narrow buckets relax fewer edges twice, and their
// number costs little since a bucket that holds few edges doubles the width of
// the next ones; on a small graph a bucket is a few barriers either way.
// Milliseconds a search at widths 4 / 6 / 12 / 24 / 96 (mean weight 32): RMAT-24 3.43
// / 3.48 / 3.94 / 4.85 / 6.20, RMAT-22 1.09 / 1.13 / 1.35 / 1.41 / 1.71, RMAT-20
// (2^24.9 edges) 0.58 / 0.60 / 0.58 / 0.61 / 0.62, 4 K vertices 0.20 / 0.19 / 0.19 / 0.18 /
// 0.16.  Where the scale changes it matters little: 0.45 to 0.48 ms at any of them
// with 2^23.9 and 2^24.4 edges, 0.37 to 0.42 (widest 0.36) with 2^22.9 and 2^23.4.
uint32_t default_delta(ptg_graph *g) {
    const float tuned = g->ctx->tuning.sssp_delta_scale;
    if (!(tuned > 0.f)) return 0;  // label-correcting rounds
    measure_mean_weight(g);
    const double r = 33554432.0 / (double)std::max<uint64_t>(1, g->m);
    const double scale = tuned * std::min(4.0, std::max(0.25, 0.25 * r * r));
    return (uint32_t)std::min(1e9, std::max(1.0, g->mean_weight > 0 ? g->mean_weight * scale : 64.0 * scale));
}

void run_traversal(ptg_graph *g, TravKind kind, uint32_t src, uint32_t *d_value, uint32_t flags,
                   uint32_t delta, uint32_t max_iters, RunResult &rr) {
    if (g->out_of_core) {
        if (g->off64) traverse_impl<unsigned long long>(g, kind, src, d_value, flags, delta, max_iters, rr);
        else traverse_impl<uint32_t>(g, kind, src, d_value, flags, delta, max_iters, rr);
        return;
    }
    bool pull = g->symmetric && !(flags & (PTG_NO_DIRECTION_OPT | PTG_REFERENCE_SCHEDULE));
    if (kind == TRAV_SSSP) pull = pull && g->m > kSsspPullEdges && graph_weights_symmetric(g);
    if (kind != TRAV_SSSP || (flags & PTG_REFERENCE_SCHEDULE)) delta = 0;
    else if (delta == 0) delta = default_delta(g);
    if (max_iters == 0) max_iters = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, 4 * g->n + 16);
    Workspace &ws = g->ctx->ws;
    uint32_t *val = d_value;
    if (g->relabeled && kind == TRAV_CCPROP) {  // in the stored vertex order, mapped to caller ids after
        ws.relab[0].ensure(g->n * 4);
        ws.relab[1].ensure(g->n * 4);
        val = ws.relab[0].as<uint32_t>();
    }
    run_resident(g, kind, src, val, (flags & PTG_LEVEL_ZERO_BASED) ? 0u : 1u, delta, pull, max_iters, rr);
    if (val != d_value) cc_labels_out(g, val, ws.relab[1].as<uint32_t>(), d_value);
    PTG_CUDA_TRY(cudaGetLastError());
}

}  // namespace ptg
