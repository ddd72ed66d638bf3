// cc.cu - connected components to min-vertex labels by hooking and pointer
// jumping, for one graph and for a batch of independent graphs.
//
// Reference: ccCaculateInOpt (ptGraph/main.cu:222-440) and ccCaculateInShare
// (961-1035) start from value[i] = i with every vertex active (283-286) and
// push the smaller label along out-edges with atomicMin (cc_kernel,
// gpu_kernels.cu:136-150) until nothing changes: one full relax round per
// hop of the longest shortest path.  On a symmetric graph the fixed point is
// "label = smallest vertex id in the component".
//
// Here (symmetric graphs): parent[v] = v; every edge u->v with v < u links the
// two trees' roots, always hanging the larger root under the smaller one
// (compare-and-swap, retried on contention), so every root is the smallest id
// of its tree; a final pass points every vertex at its root.  That is one
// pass over the edges instead of one per hop.  Directed graphs keep the
// reference's label propagation (traverse.cu), whose fixed point differs.
// The edge pass is edge-centric (2048-edge tiles, source rows found by binary
// search over the tile's offsets), and out-of-core graphs hook their streamed
// partitions one after another: linking is order-independent.
#include <algorithm>

#include "ptg_device.cuh"

namespace ptg {
namespace {

// Root of v with path splitting (parents only ever point to smaller ids).
__device__ __forceinline__ uint32_t find_root(uint32_t *parent, uint32_t v) {
    uint32_t cur = parent[v];
    if (cur != v) {
        uint32_t prev = v, next;
        while (cur > (next = parent[cur])) {
            parent[prev] = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

__device__ __forceinline__ void hook(uint32_t *parent, uint32_t u, uint32_t v) {
    uint32_t ru = find_root(parent, u), rv = find_root(parent, v);
    for (int guard = 0; guard < (1 << 20) && ru != rv; guard++) {
        if (ru < rv) {
            uint32_t t = ru;
            ru = rv;
            rv = t;
        }
        // ru > rv: hang ru under rv if ru is still a root
        uint32_t old = atomicCAS(&parent[ru], ru, rv);
        if (old == ru) return;
        ru = find_root(parent, old);
        rv = find_root(parent, rv);
    }
}

__global__ void k_iota(uint32_t *a, uint64_t n, uint64_t base) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        a[i] = (uint32_t)(base + i);
}

// Hook every edge in [e_begin, e_end) whose target is below its source.
// col_base[j - e_begin] is edge j's target (resident array or staging buffer).
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_hook(uint64_t e_begin, uint64_t e_end, uint64_t v_first,
                                                 uint64_t v_last, const OffT *off,
                                                 const uint32_t *col_base, uint32_t *parent) {
    __shared__ OffT s_off[kTile + 2];
    uint64_t E = e_end - e_begin;
    uint64_t ntiles = (E + kTile - 1) / kTile;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        uint64_t t0 = e_begin + tile * kTile, t1 = min(e_end, t0 + kTile);
        uint64_t r0 = block_last_le(off, v_first, v_last + 1, t0);
        uint64_t r1 = block_last_le(off, r0, v_last + 1, t1 - 1);
        uint64_t nrows = r1 - r0 + 1;
        bool staged = nrows <= (uint64_t)kTile;
        if (staged) {
            for (uint64_t k = threadIdx.x; k <= nrows; k += kBlock) s_off[k] = off[r0 + k];
        }
        __syncthreads();
        for (uint64_t j = t0 + threadIdx.x; j < t1; j += kBlock) {
            uint64_t u = staged ? r0 + last_le(s_off, 0, nrows, j) : last_le(off, r0, r0 + nrows, j);
            uint32_t v = col_base[j - e_begin];
            if (v < u) hook(parent, (uint32_t)u, v);
        }
        __syncthreads();
    }
}

// Point every vertex at its root; labels become local ids (minus base).
__global__ void k_compress(uint32_t *parent, uint64_t n, uint64_t first, uint32_t base) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t v = first + i;
        uint32_t r = parent[v];
        while (r != parent[r]) r = parent[r];
        parent[v] = r;
    }
}

// Every vertex's root as an id within its graph.  The graph is searched once
// per warp where its 32 vertices lie in one.
__global__ void __launch_bounds__(kBlock) k_localize(const uint32_t *parent, uint64_t n, const uint64_t *vtx_begin,
                                                     uint32_t num_graphs, uint32_t *labels) {
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t w = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5; w * 32 < n; w += nwarps) {
        const uint64_t v = w * 32 + lane_id();
        uint64_t g = last_le(vtx_begin, 0, num_graphs, w * 32);
        if (v >= n) continue;
        if (w * 32 + 31 >= vtx_begin[g + 1]) g = last_le(vtx_begin, g, num_graphs, v);
        uint32_t r = parent[v], up;
        while ((up = parent[r]) != r) r = up;
        labels[v] = (uint32_t)(r - vtx_begin[g]);
    }
}

template <class OffT>
void cc_hook_impl(ptg_graph *g, uint32_t *d_label, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int sms = ctx->sm_count;
    const uint64_t n = g->n;
    const OffT *off = g->d_off.as<OffT>();
    launch(ctx, "k_iota", k_iota, grid_for(n, kBlock, sms * 8), kBlock, 0, st, d_label, n, (uint64_t)0);
    uint64_t res = g->resident_edges;
    if (res > 0) {
        uint64_t v_last = g->out_of_core ? g->part_first_vertex[g->resident_partitions] : n - 1;
        if (v_last >= n) v_last = n - 1;
        launch(ctx, "k_hook", k_hook<OffT>, grid_for(res, kTile, sms * 16), kBlock, 0, st, (uint64_t)0, res,
               (uint64_t)0, v_last, off, g->d_col.as<uint32_t>(), d_label);
        PTG_CUDA_TRY(cudaGetLastError());
    }
    rr.edges_relaxed = g->m;
    if (g->out_of_core) {
        int b = 0;
        for (uint64_t p = g->resident_partitions; p < g->num_partitions; p++) {
            uint64_t e0 = p * g->partition_edges, e1 = std::min<uint64_t>(g->m, e0 + g->partition_edges);
            cudaStream_t cs = ctx->copy_stream;
            PTG_CUDA_TRY(cudaStreamWaitEvent(cs, g->stage_free[b], 0));
            stream_edges(g, 0, g->stage_col[b].p, e0, e1, cs);
            PTG_CUDA_TRY(cudaEventRecord(g->stage_ready[b], cs));
            PTG_CUDA_TRY(cudaStreamWaitEvent(st, g->stage_ready[b], 0));
            launch(ctx, "k_hook_partition", k_hook<OffT>, grid_for(e1 - e0, kTile, sms * 16), kBlock, 0, st,
                   e0, e1, g->part_first_vertex[p], g->part_first_vertex[p + 1], off,
                   g->stage_col[b].as<uint32_t>(), d_label);
            PTG_CUDA_TRY(cudaGetLastError());
            PTG_CUDA_TRY(cudaEventRecord(g->stage_free[b], st));
            rr.link_bytes += (e1 - e0) * 4;
            rr.parts_streamed++;
            b = (b + 1) % (int)g->n_stage;
        }
    }
    launch(ctx, "k_compress", k_compress, grid_for(n, kBlock, sms * 8), kBlock, 0, st, d_label, n,
           (uint64_t)0, 0u);
    PTG_CUDA_TRY(cudaGetLastError());
    rr.iterations = 1;
}

// ---------------------------------------------------------------------------
// Afforest (Sutton, Ben-Nun, Barak 2018) on symmetric graphs: link every
// vertex to its first neighbours, compress, find each graph's largest
// component from a few samples, then link the remaining edges only of
// vertices outside it.  An edge between the giant component and a vertex w
// outside it is still linked from w's side, so the result is unchanged; on
// RMAT and ER graphs almost every vertex is in the giant component and most
// of the edge list is never read.
// ---------------------------------------------------------------------------
constexpr uint32_t kAffFirst = 2;     // edges of every row that the first two passes link
constexpr uint32_t kAffLong = 1024;   // edges per work item of a longer row

// Every vertex hangs under its first neighbour when that one is smaller
// (stored-order rows list hubs first, given rows their smallest id): a forest
// without one atomic, where hooking the same edges took a root search and a
// compare-and-swap each.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_aff_init(const OffT *off, const uint32_t *col, uint64_t n,
                                                     uint32_t *parent) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const OffT b = off[v];
        parent[v] = b < off[v + 1] ? min((uint32_t)v, col[b]) : (uint32_t)v;
    }
}

// Roots that the first two edges of a vertex join: their parents are lowered
// to the least of them, without a retry when several edges lower the same
// root (k_aff_sample links what is lost).  The parents are flat before
// (k_compress), and every value written is one that was read, so only entries
// of roots change, by edges that are linked again later.  Without these
// rounds the threads race in k_aff_sample to join many trees, one
// compare-and-swap after another on the same few roots.  On a degree-grouped
// graph nearly every vertex hangs under a hub already, whose second edge
// leads to another hub: every 32nd warp's vertices suffice to join the hubs
// (16 us, and k_aff_sample takes 20 instead of 47-430 us at 3 M vertices and 46 M
// edges; all vertices would race here, 165 us, and every 256th warp's leave
// trees, 26-47 us in k_aff_sample).  In the given order the trees are many
// and small: two rounds over all vertices take 131 us, and k_aff_sample 41
// instead of 733 us (512 Erdos-Renyi graphs, 4 M vertices; one round: 143 us).
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_aff_join(const OffT *off, const uint32_t *col, uint64_t n, uint32_t every,
                                                     uint32_t *parent) {
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t w = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5; w * every * 32 < n; w += nwarps) {
        const uint64_t v = w * every * 32 + lane_id();
        if (v >= n) continue;
        const OffT b = off[v], e = off[v + 1];
        if (b == e) continue;
        const uint32_t c0 = col[b], c1 = e - b > (OffT)1 ? col[b + 1] : c0;
        const uint32_t r = parent[v], r0 = parent[c0], r1 = parent[c1], lo = min(r, min(r0, r1));
        if (r != lo && lo < *(volatile const uint32_t *)&parent[r]) atomicMin(&parent[r], lo);
        if (r0 != lo && lo < *(volatile const uint32_t *)&parent[r0]) atomicMin(&parent[r0], lo);
        if (r1 != lo && lo < *(volatile const uint32_t *)&parent[r1]) atomicMin(&parent[r1], lo);
    }
}

// The first two edges of every vertex linked for good.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_aff_sample(const OffT *off, const uint32_t *col, uint64_t n,
                                                       uint32_t *parent) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const OffT b = off[v], e = off[v + 1];
        if (b == e) continue;
        const uint32_t c0 = col[b], c1 = e - b > (OffT)1 ? col[b + 1] : c0;
        if (c0 > (uint32_t)v) hook(parent, (uint32_t)v, c0);
        if (c1 != c0) hook(parent, (uint32_t)v, c1);
    }
}

// Largest component of each graph: the majority root of 9 spread samples,
// marked in a bitmap.  vb == nullptr: one graph of n vertices.
__global__ void k_aff_giant(const uint64_t *vb, uint32_t num_graphs, uint64_t n, const uint32_t *parent,
                            uint32_t *mark) {
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < num_graphs; g += gridDim.x * blockDim.x) {
        uint64_t v0 = vb ? vb[g] : 0, nv = vb ? vb[g + 1] - v0 : n;
        if (nv == 0) continue;
        uint32_t lab[9];
#pragma unroll
        for (int i = 0; i < 9; i++) {
            uint64_t h = (uint64_t)(g + 1) * 0x9E3779B97F4A7C15ull + (uint64_t)i * 0xBF58476D1CE4E5B9ull;
            h ^= h >> 31;
            lab[i] = (uint32_t)(v0 + h % nv);
        }
        bool moved = true;
        while (moved) {  // the nine walks to the roots side by side
            uint32_t up[9];
            moved = false;
#pragma unroll
            for (int i = 0; i < 9; i++) up[i] = parent[lab[i]];
#pragma unroll
            for (int i = 0; i < 9; i++) {
                moved |= up[i] != lab[i];
                lab[i] = up[i];
            }
        }
        uint32_t best = lab[0];
        int bestc = 0;
        for (int i = 0; i < 9; i++) {
            int c = 0;
            for (int j = 0; j < 9; j++) c += lab[j] == lab[i];
            if (c > bestc) {
                bestc = c;
                best = lab[i];
            }
        }
        atomicOr(&mark[best >> 5], 1u << (best & 31u));
    }
}

// Links the edges from the kAffFirst-th on of every vertex outside its
// graph's giant component, and points every vertex at its root (or at the
// giant's).  Work goes by vertices: nearly all are in the giant, so a warp
// reads 32 vertices' parents and offsets and is done, and the edge list is
// not walked at all.  (Going by 2048-edge tiles with a row search per edge,
// this pass read the offsets of every edge's row only to skip it: 2.13 ms of
// a 2.8 ms RMAT-24 call, 356 us at 3 M vertices and 46 M edges.)  The edges
// of a warp's remaining rows are dealt to its lanes evenly; rows above
// kAffLong edges are queued in pieces for k_aff_long, so no warp walks one
// alone.  A walk stops at the marked root even when another warp hangs that
// root under a smaller one meanwhile: the mark decides, so two vertices that
// skip each other's edge always share that root.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_aff_finish(const OffT *off, const uint32_t *col, uint64_t n,
                                                       const uint32_t *mark, uint32_t *parent, uint2 *items,
                                                       unsigned long long *count) {
    const unsigned lane = lane_id();
    const uint64_t nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t w = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5; w * 32 < n; w += nwarps) {
        const uint64_t v = w * 32 + lane;
        OffT b = 0, e = 0;
        bool skip = true;
        if (v < n) {
            b = off[v];
            e = off[v + 1];
            const uint32_t up = parent[v];
            uint32_t r = up;
            skip = bit_test(mark, (uint32_t)v) || bit_test(mark, r);
            while (!skip) {
                const uint32_t p = parent[r];
                if (p == r) break;
                r = p;
                skip = bit_test(mark, r);
            }
            if (r != up) parent[v] = r;
        }
        const uint64_t rem = !skip && e - b > (OffT)kAffFirst ? (uint64_t)(e - b) - kAffFirst : 0;
        unsigned longs = __ballot_sync(0xffffffffu, rem > kAffLong);
        while (longs) {
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const uint64_t pieces = (__shfl_sync(0xffffffffu, rem, src) + kAffLong - 1) / kAffLong;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(count, (unsigned long long)pieces);
            at = __shfl_sync(0xffffffffu, at, 0);
            for (uint64_t i = lane; i < pieces; i += 32) items[at + i] = make_uint2((uint32_t)(w * 32) + src, (uint32_t)i);
        }
        const uint32_t cnt = rem > kAffLong ? 0u : (uint32_t)rem;
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {  // warp-uniform bound
            const uint32_t t = min(t0 + lane, total - 1);
            uint32_t src = 0;  // first lane whose inclusive sum exceeds t
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xffffffffu, incl, src + step - 1) <= t) src += step;
            const uint32_t at = t - (__shfl_sync(0xffffffffu, incl, src) - __shfl_sync(0xffffffffu, cnt, src));
            const OffT base = __shfl_sync(0xffffffffu, b, src);
            if (t0 + lane < total) hook(parent, (uint32_t)(w * 32) + src, __ldcs(col + base + kAffFirst + at));
        }
    }
}

// The pieces that k_aff_finish queued, a warp each.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_aff_long(const OffT *off, const uint32_t *col, const uint2 *items,
                                                     const unsigned long long *count, uint32_t *parent) {
    const uint64_t total = *count, nwarps = (uint64_t)gridDim.x * (kBlock / 32);
    for (uint64_t i = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5; i < total; i += nwarps) {
        const uint2 it = items[i];
        const OffT b = off[it.x] + (OffT)kAffFirst + (OffT)it.y * (OffT)kAffLong, e = off[(uint64_t)it.x + 1];
        const OffT end = e - b > (OffT)kAffLong ? b + (OffT)kAffLong : e;
        for (OffT k = b + lane_id(); k < end; k += 32) hook(parent, it.x, __ldcs(col + k));
    }
}

// The Afforest sequence up to the last link, on a resident CSR of one or
// more graphs; the caller's last pass walks the remaining parents.  `grouped`:
// vertices in degree order, rows listing hubs first (relabel.cu).
template <class OffT>
void afforest(ptg_ctx *ctx, const OffT *off, const uint32_t *col, uint64_t n, uint64_t m, const uint64_t *d_vb,
              uint32_t num_graphs, bool grouped, uint32_t *parent) {
    cudaStream_t st = ctx->stream;
    Workspace &ws = ctx->ws;
    const int sms = ctx->sm_count;
    const uint64_t words = (n + 31) / 32;
    ws.bm[0].ensure(words * 4);              // the marked roots
    ws.scan.ensure((m / (kAffLong / 2) + 1) * sizeof(uint2));  // a row has at most 2 pieces per kAffLong edges
    ws.bsum.ensure(1024 * 8);
    uint32_t *mark = ws.bm[0].as<uint32_t>();
    uint2 *items = ws.scan.as<uint2>();
    unsigned long long *count = ws.bsum.as<unsigned long long>();
    const int vgrid = grid_for(n, kBlock, sms * 8);
    PTG_CUDA_TRY(cudaMemsetAsync(mark, 0, words * 4, st));
    PTG_CUDA_TRY(cudaMemsetAsync(count, 0, 8, st));
    launch(ctx, "k_aff_init", k_aff_init<OffT>, vgrid, kBlock, 0, st, off, col, n, parent);
    launch(ctx, "k_compress", k_compress, vgrid, kBlock, 0, st, parent, n, (uint64_t)0, 0u);
    const uint32_t every = grouped ? 32u : 1u;
    for (int r = 0; r < (grouped ? 1 : 2); r++) {
        launch(ctx, "k_aff_join", k_aff_join<OffT>, grid_for(n / every + 1, kBlock, sms * 8), kBlock, 0, st, off, col,
               n, every, parent);
        launch(ctx, "k_compress", k_compress, vgrid, kBlock, 0, st, parent, n, (uint64_t)0, 0u);
    }
    launch(ctx, "k_aff_sample", k_aff_sample<OffT>, vgrid, kBlock, 0, st, off, col, n, parent);
    launch(ctx, "k_aff_giant", k_aff_giant, grid_for(num_graphs, 64, sms * 4), 64, 0, st, d_vb, num_graphs, n,
           (const uint32_t *)parent, mark);
    launch(ctx, "k_aff_finish", k_aff_finish<OffT>, vgrid, kBlock, 0, st, off, col, n, (const uint32_t *)mark, parent,
           items, count);
    launch(ctx, "k_aff_long", k_aff_long<OffT>, grid_for(m / kAffLong + 1, kBlock / 32, sms * 8), kBlock, 0, st, off,
           col, (const uint2 *)items, (const unsigned long long *)count, parent);
    PTG_CUDA_TRY(cudaGetLastError());
}

}  // namespace

void run_cc_hook(ptg_graph *g, uint32_t *d_label, RunResult &rr) {
    if (!g->out_of_core && g->m > 0) {
        // resident symmetric graph: Afforest
        Workspace &ws = g->ctx->ws;
        uint32_t *out = d_label;
        if (g->relabeled) {
            // labels in the stored vertex order first, then the minimum caller id per component
            ws.relab[0].ensure(g->n * 4);
            ws.relab[1].ensure(g->n * 4);
            d_label = ws.relab[0].as<uint32_t>();
        }
        if (g->off64)
            afforest<unsigned long long>(g->ctx, g->d_off.as<unsigned long long>(), g->d_col.as<uint32_t>(), g->n,
                                         g->m, nullptr, 1, g->relabeled, d_label);
        else
            afforest<uint32_t>(g->ctx, g->d_off.as<uint32_t>(), g->d_col.as<uint32_t>(), g->n, g->m, nullptr, 1,
                               g->relabeled, d_label);
        if (!g->relabeled)
            launch(g->ctx, "k_compress", k_compress, grid_for(g->n, kBlock, g->ctx->sm_count * 8), kBlock, 0,
                   g->ctx->stream, d_label, g->n, (uint64_t)0, 0u);
        if (g->relabeled) cc_labels_out(g, d_label, ws.relab[1].as<uint32_t>(), out);
        rr.edges_relaxed = g->m;
        rr.iterations = 1;
        return;
    }
    if (g->off64) cc_hook_impl<unsigned long long>(g, d_label, rr);
    else cc_hook_impl<uint32_t>(g, d_label, rr);
}

void run_cc_batch(ptg_ctx *ctx, uint32_t num_graphs, const uint64_t *vtx_begin,
                  const uint64_t *offsets, const uint32_t *col, uint32_t *labels, RunResult &rr) {
    cudaStream_t st = ctx->stream;
    const int sms = ctx->sm_count;
    uint64_t n = vtx_begin[num_graphs];
    uint64_t m = offsets[n];
    PTG_REQUIRE(n < 0xFFFFFFFFull, PTG_ERR_INVALID, "batched CC needs fewer than 2^32 vertices in total");
    // one block for the uploaded CSR and the labels (of at least the size
    // that the block cache keeps: small batches don't pay for a cudaMalloc
    // and a cudaFree per array and call)
    auto up = [](uint64_t x) { return (x + 255) & ~(uint64_t)255; };
    const uint64_t o_col = up((n + 1) * 8), o_parent = o_col + up(m * 4), o_vb = o_parent + up(n * 4);
    DevBuf block;
    block.ensure(std::max<uint64_t>(1ull << 20, o_vb + (num_graphs + 1) * 8ull));
    char *base = block.as<char>();
    auto *d_off = reinterpret_cast<unsigned long long *>(base);
    auto *d_col = reinterpret_cast<uint32_t *>(base + o_col);
    auto *d_parent = reinterpret_cast<uint32_t *>(base + o_parent);
    auto *d_vb = reinterpret_cast<uint64_t *>(base + o_vb);
    auto *d_labels = reinterpret_cast<uint32_t *>(base);  // over the offsets, read by then
    PTG_CUDA_TRY(cudaMemcpyAsync(d_off, offsets, (n + 1) * 8, cudaMemcpyHostToDevice, st));
    if (m) PTG_CUDA_TRY(cudaMemcpyAsync(d_col, col, m * 4, cudaMemcpyHostToDevice, st));
    PTG_CUDA_TRY(cudaMemcpyAsync(d_vb, vtx_begin, (num_graphs + 1) * 8, cudaMemcpyHostToDevice, st));
    PTG_CUDA_TRY(cudaEventRecord(ctx->ev0, st));
    // one Afforest pass over the concatenated CSR links the edges of every
    // graph, however uneven the graphs are
    afforest<unsigned long long>(ctx, d_off, d_col, n, m, d_vb, num_graphs, false, d_parent);
    launch(ctx, "k_localize", k_localize, grid_for(n, kBlock, sms * 8), kBlock, 0, st,
           (const uint32_t *)d_parent, n, (const uint64_t *)d_vb, num_graphs, d_labels);
    PTG_CUDA_TRY(cudaGetLastError());
    PTG_CUDA_TRY(cudaEventRecord(ctx->ev1, st));
    PTG_CUDA_TRY(cudaMemcpyAsync(labels, d_labels, n * 4, cudaMemcpyDeviceToHost, st));
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    rr.device_ms = ms;
    rr.edges_relaxed = m;
    rr.iterations = 1;
}

}  // namespace ptg
