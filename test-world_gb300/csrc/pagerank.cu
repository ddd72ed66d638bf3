// pagerank.cu - pull PageRank and personalized PageRank as degree-binned SpMV.
//
// The reference has no PageRank: prCaculateInShare (ptGraph/main.cu:891-959)
// runs frontier bookkeeping with its kernel call commented out (937) and
// prCaculateInOpt is declared (52) but never defined.  The semantics here:
//   r0 = 1/n (PPR: r0 = e_src)
//   r' = (1-d)/n + d * (sum_{u -> v} r[u]/deg(u) + dangling/n)
//   (PPR: r' = d * sum + [v == src] * ((1-d) + d * dangling))
// with dangling = sum of r over zero-degree vertices and a fixed number of
// iterations.  Ranks and contributions are stored in FP32; per-vertex sums
// are compensated two-float sums, because GB300 runs FP32 adds at 64x its FP64
// rate.  A lane collects the exact errors of its additions in one float (ff_term):
// over the n <= 128 terms that a lane adds (pr_chunk / 32 where that is tuned up)
// what is lost stays below about n^2 2^-48, 2^-34 of the sum, and the partials of
// the lanes and pieces meet in renormalized two-floats.  The ranks are the same
// bits as with a renormalization after each term.
//
// Pull over a symmetric CSR (in-edges == out-edges), as a degree-binned
// SpMV: rows are grouped once per graph by degree (a thread, 8 lanes or a
// warp per row, and warp-sized pieces of the longest rows), each lane keeps
// its own two-float partial, and partials meet through shuffles in a fixed
// order, so the result of a row does not depend on scheduling.  An iteration is
// one launch: its warps take units of rows from counters, longest first, and
// the warp that ends a long row's last piece adds the row's partial sums in
// order.  The gathered contributions of a scale-24 graph (67 MB) stay in L2;
// DRAM carries the column stream, so the gathers' L2 sector traffic is the bound.
#include <algorithm>

#include "ptg_device.cuh"

namespace ptg {

namespace {

struct ff {
    float hi, lo;
};

// Knuth's two-sum, renormalized (compensated two-float accumulation).
__device__ __forceinline__ ff ff_add(ff a, float b) {
    float s = a.hi + b;
    float bb = s - a.hi;
    float e = (a.hi - (s - bb)) + (b - bb);
    e += a.lo;
    float h = s + e;
    return ff{h, e - (h - s)};
}

__device__ __forceinline__ ff ff_add(ff a, ff b) {
    float s = a.hi + b.hi;
    float bb = s - a.hi;
    float e = (a.hi - (s - bb)) + (b.hi - bb);
    e += a.lo + b.lo;
    float h = s + e;
    return ff{h, e - (h - s)};
}

// One more term for a lane's running sum: the exact error of each addition
// (Knuth) collects in lo, renormalized once at the end (ff_end).  7 operations
// a term where the renormalized sum takes 11; 8 sources a neighbour make that
// count.
__device__ __forceinline__ void ff_term(ff &a, float b) {
    const float s = a.hi + b, bb = s - a.hi;
    a.lo += (a.hi - (s - bb)) + (b - bb);
    a.hi = s;
}

__device__ __forceinline__ ff ff_end(ff a) {
    const float h = a.hi + a.lo;
    return ff{h, a.lo - (h - a.hi)};
}

__device__ __forceinline__ double ff_dbl(ff a) { return (double)a.hi + (double)a.lo; }

struct PrArgs {
    uint64_t n, m;
    const void *off;          // OffT[n+1]
    const uint32_t *col;
    const float *contrib_in;  // [n]
    float *contrib_out;       // [n]
    float *rank_out;          // [n] or nullptr (written on the last iteration)
    const double *dangling_in;
    double *dangling_out;
    double *dangling_next;    // cleared for the next iteration
    double d;
    double teleport, spread;  // (1-d)/n and d/n
    int personalized;
    uint32_t src;
};

// Two-float product (fma gives the exact rounding error of hi*hi).
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
    float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    float h = p + e;
    return ff{h, e - (h - p)};
}

__device__ __forceinline__ ff ff_of(double x) {
    float h = (float)x;
    return ff{h, (float)(x - (double)h)};
}

// Per-iteration constants of the update, as two-floats (computed once per CTA
// in FP64 from the previous iteration's dangling mass, kept in shared memory):
//   PR : r = base + d * sum,   base = (1-d)/n + d * dangling / n
//   PPR: r = d * sum (+ bonus at src), bonus = (1-d) + d * dangling
struct PrConst {
    ff base, d, bonus;
};

__device__ __forceinline__ PrConst pr_const(const PrArgs &a) {
    const double dang = *a.dangling_in;
    PrConst c;
    c.d = ff_of(a.d);
    c.base = a.personalized ? ff{0.f, 0.f} : ff_of(a.teleport + a.spread * dang);
    c.bonus = a.personalized ? ff_of((1.0 - a.d) + a.d * dang) : ff{0.f, 0.f};
    return c;
}

template <class OffT>
__device__ __forceinline__ void finalize_row(const PrArgs &a, const PrConst &c, uint64_t v, OffT deg,
                                             ff sum, ff &dang_local) {
    ff r = ff_add(c.base, ff_mul(c.d, sum));
    if (a.personalized && v == a.src) r = ff_add(r, c.bonus);
    float rf = r.hi + r.lo;
    if (a.rank_out) a.rank_out[v] = rf;
    if (deg == 0) {
        dang_local = ff_add(dang_local, rf);
        a.contrib_out[v] = 0.f;
    } else {
        a.contrib_out[v] = rf / (float)deg;
    }
}

// contrib0 = r0 / deg, dangling0 = sum of r0 over zero-degree vertices.
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_pr_init(const OffT *off, uint64_t n, int personalized,
                                                    uint32_t src, float *contrib, double *dangling) {
    double dl = 0.0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        float r = personalized ? (v == src ? 1.f : 0.f) : (float)(1.0 / (double)n);
        OffT deg = off[v + 1] - off[v];
        if (deg == 0) {
            dl += r;
            contrib[v] = 0.f;
        } else {
            contrib[v] = r / (float)deg;
        }
    }
    double s = block_reduce_sum(dl);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(dangling, s);
}

// ---------------------------------------------------------------------------
// Degree-binned SpMV, one launch per iteration.  Rows are split once per graph
// by degree (mid and chunk are tuning values, 256 and 4096 by default, recorded
// with the bins):
//   deg <= kPrSmall          one thread per row (all rows are looked at)
//   kPrSmall < deg <= mid    8 lanes per row (list `mid`)
//   mid < deg <= chunk       one warp per row (list `big`)
//   deg > chunk              chunk-edge pieces, one warp each; the warp that
//                            finishes a row's last piece adds the partial
//                            sums in piece order
// Every lane keeps its own two-float partial (independent dependency chains),
// partials meet through shuffles in a fixed order, so a row's sum depends
// only on the row.  The lists hold rows in ascending order, so rank and
// contribution stores of neighbouring lanes fall in the same lines.
//
// Warps take units of work (a piece, a few big rows, 32 mid rows, some hundred
// small ones) from a counter, longest first, the next one fetched while the
// present one runs.  Five launches on four streams per iteration, joined by
// events, cost 25-40 us an iteration whatever the graph's size, and ended with
// one thread per long row adding its pieces.  20 iterations: RMAT-24 28.9 ->
// 28.2 ms, 2^14 vertices 0.43 -> 0.22 ms.
// ---------------------------------------------------------------------------
constexpr uint32_t kPrSmall = 4;
constexpr int kPrMinBlocks = 6;  // CTAs per SM (40 registers; 8 at 32: 1.45 instead of 1.41 ms on RMAT-24)

struct PrBins {
    const uint32_t *mid;
    uint64_t n_mid;
    const uint32_t *big;
    uint64_t n_big;
    const uint2 *items;  // (row, chunk)
    uint64_t n_items;
    float2 *partial;     // [n_items * sources]
    uint32_t *left;      // [n_items] pieces done, at the row's first item; zero between iterations
    uint32_t chunk;      // edges per piece of a long row
    // units: n_items pieces, then big rows / big_step, mid rows / mid_step, all rows / small_step
    uint32_t big_step, mid_step, small_step;
    uint64_t big_units, mid_units, small_units;
    uint64_t mid_share;  // ceil(2^32 mid_units / (big_units + mid_units))
    unsigned slices;                   // kSlices, fewer for fewer CTAs
    unsigned *counter, *counter_next;  // units handed out; the next iteration's, cleared
};

__device__ __forceinline__ ff ff_shfl_xor(ff s, int o, int width) {
    return ff{__shfl_xor_sync(0xffffffffu, s.hi, o, width), __shfl_xor_sync(0xffffffffu, s.lo, o, width)};
}

// Runs f(unit) for the units a warp gets (warp-uniform).  The units are dealt
// to bins.slices slices, the CTAs likewise, and each slice hands its own out
// from a counter: one counter for all warps serialises when units are short
// (RMAT-18: 36 K units an iteration, 0.95 ms for 20 iterations, 0.63 with 16 slices).
constexpr unsigned kSlices = 16, kSlicePad = 32;  // counters 128 bytes apart
template <class F>
__device__ __forceinline__ void for_units(const PrBins &bins, F &&f) {
    const uint64_t total = bins.n_items + bins.big_units + bins.mid_units + bins.small_units;
    const unsigned slice = blockIdx.x % bins.slices;
    const unsigned warps = (gridDim.x - slice + bins.slices - 1) / bins.slices * (kBlock / 32);  // in this slice
    uint64_t i = blockIdx.x / bins.slices * (kBlock / 32) + (threadIdx.x >> 5);
    while (true) {
        const uint64_t u = i * bins.slices + slice;
        if (u >= total) return;
        unsigned nx = 0;
        if (lane_id() == 0) nx = warps + atomicAdd(bins.counter + slice * kSlicePad, 1u);
        f(u);
        i = __shfl_sync(0xffffffffu, nx, 0);
    }
}

// Clears the next iteration's counters (read by nothing in this one).
__device__ __forceinline__ void clear_next(const PrBins &bins) {
    if (blockIdx.x == 0 && threadIdx.x < kSlices) bins.counter_next[threadIdx.x * kSlicePad] = 0u;
}

// Unit u of the big and mid rows together, dealt evenly between the two: the
// mid unit's number (true) or the big unit's.  (Big rows first and mid rows
// after: 1.46 instead of 1.41 ms an iteration on RMAT-24.)
__device__ __forceinline__ bool mid_unit(const PrBins &bins, uint64_t &u) {
    const uint64_t before = (u * bins.mid_share) >> 32, after = ((u + 1) * bins.mid_share) >> 32;
    u = after > before ? before : u - before;
    return after > before;
}

// Sum of the neighbours' values at edges k, k + STRIDE, ... below e, in order,
// U column loads and gathers in flight.  Past the end zeros are added, which
// change nothing: the last edges go together too, not one after another.
template <int STRIDE, int U, class OffT>
__device__ __forceinline__ ff row_sum(const PrArgs &a, OffT k, OffT e) {
    ff s{0.f, 0.f};
    for (; k < e; k += U * STRIDE) {
        float x[U];
#pragma unroll
        for (int t = 0; t < U; t++) x[t] = k + t * STRIDE < e ? a.contrib_in[__ldcs(a.col + k + t * STRIDE)] : 0.f;
#pragma unroll
        for (int t = 0; t < U; t++) ff_term(s, x[t]);
    }
    return ff_end(s);
}

template <class OffT>
__global__ void __launch_bounds__(kBlock, kPrMinBlocks) k_pr_iter(PrArgs a, PrBins bins) {
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    __shared__ PrConst c;
    const unsigned lane = lane_id();
    ff dl{0.f, 0.f};
    if (threadIdx.x == 0) c = pr_const(a);
    __syncthreads();
    clear_next(bins);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.dangling_next = 0.0;
    for_units(bins, [&](uint64_t u) {
        if (u < bins.n_items) {  // a piece of a long row
            const uint2 item = bins.items[u];
            const OffT row = off[item.x], end = off[(uint64_t)item.x + 1];
            const OffT b = row + (OffT)item.y * (OffT)bins.chunk;
            const OffT e = end - b > (OffT)bins.chunk ? b + (OffT)bins.chunk : end;
            ff s = row_sum<32, 8>(a, b + (OffT)lane, e);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s = ff_add(s, ff_shfl_xor(s, o, 32));
            const uint32_t pieces = (uint32_t)(((uint64_t)(end - row) + bins.chunk - 1) / bins.chunk);
            const uint64_t first = u - item.y;
            uint32_t done = 0;
            if (lane == 0) {
                bins.partial[u] = make_float2(s.hi, s.lo);
                __threadfence();
                done = atomicAdd(&bins.left[first], 1u) + 1u;
                __threadfence();
            }
            if (__shfl_sync(0xffffffffu, done, 0) != pieces) return;
            ff sum{0.f, 0.f};
            for (uint32_t i0 = 0; i0 < pieces; i0 += 32) {
                const float2 p = i0 + lane < pieces ? __ldcg(&bins.partial[first + i0 + lane]) : make_float2(0.f, 0.f);
                const uint32_t cnt = min(32u, pieces - i0);
                for (uint32_t i = 0; i < cnt; i++)
                    sum = ff_add(sum, ff{__shfl_sync(0xffffffffu, p.x, i), __shfl_sync(0xffffffffu, p.y, i)});
            }
            if (lane == 0) {
                bins.left[first] = 0u;
                finalize_row<OffT>(a, c, item.x, end - row, sum, dl);
            }
            return;
        }
        u -= bins.n_items;
        const bool rest = u >= bins.big_units + bins.mid_units;
        const bool mid = !rest && mid_unit(bins, u);
        if (!rest && !mid) {  // a warp per row, their ends together
            const uint64_t i = u * bins.big_step + lane;
            const bool mine = lane < bins.big_step && i < bins.n_big;
            const uint32_t v = mine ? bins.big[i] : 0u;
            const OffT b = mine ? off[v] : (OffT)0, e = mine ? off[(uint64_t)v + 1] : (OffT)0;
            ff keep{0.f, 0.f};
            for (uint32_t t = 0; t < bins.big_step; t++) {
                ff s = row_sum<32, 8>(a, __shfl_sync(0xffffffffu, b, t) + (OffT)lane, __shfl_sync(0xffffffffu, e, t));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s = ff_add(s, ff_shfl_xor(s, o, 32));
                if (lane == t) keep = s;
            }
            if (mine) finalize_row<OffT>(a, c, v, e - b, keep, dl);
            return;
        }
        if (mid) {  // 8 lanes per row; lane l ends the unit's row l
            const uint64_t i = u * bins.mid_step + lane;
            const bool mine = lane < bins.mid_step && i < bins.n_mid;
            const uint32_t v = mine ? bins.mid[i] : 0u;
            const OffT b = mine ? off[v] : (OffT)0, e = mine ? off[(uint64_t)v + 1] : (OffT)0;
            ff keep{0.f, 0.f};
            for (uint32_t t = 0; t < bins.mid_step; t += 4) {
                const int from = (int)(t + (lane >> 3));
                ff s = row_sum<8, 8>(a, __shfl_sync(0xffffffffu, b, from) + (OffT)(lane & 7u),
                                     __shfl_sync(0xffffffffu, e, from));
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) s = ff_add(s, ff_shfl_xor(s, o, 8));
                const ff got{__shfl_sync(0xffffffffu, s.hi, (lane & 3u) * 8), __shfl_sync(0xffffffffu, s.lo, (lane & 3u) * 8)};
                if ((lane & ~3u) == t) keep = got;
            }
            if (mine) finalize_row<OffT>(a, c, v, e - b, keep, dl);
            return;
        }
        u -= bins.big_units + bins.mid_units;
        const uint64_t end = min(a.n, (u + 1) * bins.small_step);
        for (uint64_t v = u * bins.small_step + lane; v < end; v += 32) {
            const OffT b = off[v], deg = off[v + 1] - b;
            if ((uint64_t)deg > kPrSmall) continue;
            float x[kPrSmall];
#pragma unroll
            for (uint32_t t = 0; t < kPrSmall; t++)
                x[t] = t < (uint32_t)deg ? a.contrib_in[__ldcs(a.col + b + t)] : 0.f;
            ff s{0.f, 0.f};
#pragma unroll
            for (uint32_t t = 0; t < kPrSmall; t++)
                if (t < (uint32_t)deg) ff_term(s, x[t]);
            finalize_row<OffT>(a, c, v, deg, ff_end(s), dl);
        }
    });
    const double sd = block_reduce_sum(ff_dbl(dl));
    if (threadIdx.x == 0 && sd != 0.0) atomicAdd(a.dangling_out, sd);
}

// ---------------------------------------------------------------------------
// Personalized PageRank for K = 4 or 8 sources at once over the same degree
// bins.  Values are vertex-major (x[v*K + s]); a thread keeps four sources, so
// a neighbour's values are one 16-byte load of one thread (K = 4) or of two
// side by side (K = 8), which then ask L1 for its 32-byte sector once.  (One
// thread loading both halves looked the sector up twice, and L1 was what the
// pass waited for: 70% of its wavefronts' peak.)  The threads stand for the
// lanes of the single-source kernel above: the same edges in the same order,
// partials met in the same tree, so each source's ranks are bit-identical to a
// single-source ptg_ppr of that source.  The first two steps of the tree halve
// the sources a thread goes on with, and a row's sources are ended side by
// side in different lanes.  8 sources, 20 iterations: RMAT-20 7.46 -> 3.4 ms,
// RMAT-24 100.8 -> 58.8 ms. 
// ---------------------------------------------------------------------------
struct MsArgs {
    uint64_t n;
    const void *off;
    const uint32_t *col;
    const float *cin;       // [n*K]
    float *cout;            // [n*K] contributions, or ranks on the last iteration
    const double *dang_in;  // [K]
    double *dang_out;       // [K], zero on entry
    double *dang_next;      // [K], cleared for the next iteration
    const uint32_t *src;    // [K] (0xFFFFFFFF: unused lane)
    double d;
    int last;
};

// Per-iteration constants of a pass, in shared memory (FP64 once per CTA).
template <int K>
struct MsConst {
    ff d, bonus[K];
    uint32_t src[K];
};

// Rank of source s at v from its sum, as a contribution (or the rank itself on
// the last iteration), with the dangling mass of a source without edges.
template <class OffT, int K>
__device__ __forceinline__ float ms_value(const MsArgs &a, const MsConst<K> &c, uint32_t v, OffT deg, uint32_t s,
                                          ff sum) {
    ff r = ff_add(ff{0.f, 0.f}, ff_mul(c.d, sum));
    if (v == c.src[s]) r = ff_add(r, c.bonus[s]);
    const float rf = r.hi + r.lo;
    if (deg == 0 && rf != 0.f) atomicAdd(&a.dang_out[s], (double)rf);
    return a.last ? rf : (deg == 0 ? 0.f : rf / (float)deg);
}

// Neighbours in flight per thread in the batched passes, and their CTAs per
// SM (48 registers).  RMAT-20: 171 us an iteration, 189 with two in flight; 8
// in flight at 4 CTAs per SM 163, but a graph whose values leave L2 wants the
// warps.  The order of additions does not depend on it.
constexpr int kPrkBatch = 4;
constexpr int kPrkMinBlocks = 5;

// The four values at x[u*K + 4*half ...].
template <int K>
__device__ __forceinline__ void ms_load(const MsArgs &a, uint32_t u, uint32_t half, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4 *>(a.cin + (uint64_t)u * K + 4 * half);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}

// Sums, in order, of the values of the neighbours at edges k, k + STRIDE, ...
// below e; SETS sums side by side, of the edges SHIFT further each; U steps'
// column and value loads in flight.
template <int K, int U, int SETS, int STRIDE, int SHIFT, class OffT>
__device__ __forceinline__ void ms_run(const MsArgs &a, OffT k, OffT e, uint32_t half, ff (&acc)[SETS][4]) {
#pragma unroll
    for (int i = 0; i < SETS; i++)
#pragma unroll
        for (int s = 0; s < 4; s++) acc[i][s] = ff{0.f, 0.f};
    for (; k + (OffT)((U - 1) * STRIDE + (SETS - 1) * SHIFT) < e; k += (OffT)(U * STRIDE)) {
        float x[U][SETS][4];
#pragma unroll
        for (int t = 0; t < U; t++)
#pragma unroll
            for (int i = 0; i < SETS; i++) ms_load<K>(a, __ldcs(a.col + k + t * STRIDE + i * SHIFT), half, x[t][i]);
#pragma unroll
        for (int t = 0; t < U; t++)
#pragma unroll
            for (int i = 0; i < SETS; i++)
#pragma unroll
                for (int s = 0; s < 4; s++) ff_term(acc[i][s], x[t][i][s]);
    }
    if (k < e) {  // the last edges go together too; the zeros added past the end change nothing
        float x[U][SETS][4];
#pragma unroll
        for (int t = 0; t < U; t++)
#pragma unroll
            for (int i = 0; i < SETS; i++) {
#pragma unroll
                for (int s = 0; s < 4; s++) x[t][i][s] = 0.f;
                if (k + (OffT)(t * STRIDE + i * SHIFT) < e)
                    ms_load<K>(a, __ldcs(a.col + k + t * STRIDE + i * SHIFT), half, x[t][i]);
            }
#pragma unroll
        for (int t = 0; t < U; t++)
#pragma unroll
            for (int i = 0; i < SETS; i++)
#pragma unroll
                for (int s = 0; s < 4; s++) ff_term(acc[i][s], x[t][i][s]);
    }
#pragma unroll
    for (int i = 0; i < SETS; i++)
#pragma unroll
        for (int s = 0; s < 4; s++) acc[i][s] = ff_end(acc[i][s]);
}

// The partials of WIDTH single-source lanes (H threads each, side by side)
// added in a tree of distances WIDTH/2 ... 1; the first two steps halve the
// sources a thread goes on with.  Returns the thread's source of its four, the
// total in `sum`; threads that differ in the bits of ms_copies hold the same.
template <int H, int WIDTH>
__device__ __forceinline__ uint32_t ms_tree(const ff (&acc)[4], ff &sum) {
    const unsigned lane = lane_id();
    constexpr int o0 = WIDTH / 2 * H, o1 = WIDTH / 4 * H;
    const bool up0 = (lane & o0) != 0, up1 = (lane & o1) != 0;
    ff two[2];
#pragma unroll
    for (int i = 0; i < 2; i++)
        two[i] = ff_add(up0 ? acc[i + 2] : acc[i], ff_shfl_xor(up0 ? acc[i] : acc[i + 2], o0, 32));
    sum = ff_add(up1 ? two[1] : two[0], ff_shfl_xor(up1 ? two[0] : two[1], o1, 32));
#pragma unroll
    for (int o = WIDTH / 8 * H; o >= H; o >>= 1) sum = ff_add(sum, ff_shfl_xor(sum, o, 32));
    return (up0 ? 2u : 0u) + (up1 ? 1u : 0u);
}

template <int H, int WIDTH>
__device__ __forceinline__ bool ms_owner() {
    return (lane_id() & (unsigned)((WIDTH / 4 - 1) * H)) == 0;
}

// A warp's sum of edges [b, e) as the 32 lanes of the single-source kernel
// form it; `source` of the K is this thread's.
template <int K, class OffT>
__device__ __forceinline__ ff ms_row32(const MsArgs &a, OffT b, OffT e, uint32_t half, uint32_t &source) {
    constexpr int H = K / 4, kLanes = 32 / H;
    const unsigned vlane = lane_id() / H;
    ff acc[H][4], sum;
    ms_run<K, kPrkBatch / H, H, 32, kLanes>(a, b + (OffT)vlane, e, half, acc);
    if (H == 2)
#pragma unroll
        for (int s = 0; s < 4; s++) acc[0][s] = ff_add(acc[0][s], acc[H - 1][s]);  // distance 16
    source = half * 4 + ms_tree<H, kLanes>(acc[0], sum);
    return sum;
}

// A vertex without edges that is none of the pass's sources keeps 0 in both
// value buffers (both start zeroed), so it is skipped: on RMAT graphs about
// half the vertices are isolated, and writing their K values each iteration
// was a third of the small rows' time.
template <class OffT, int K>
__global__ void __launch_bounds__(kBlock, kPrkMinBlocks) k_prk_iter(MsArgs a, PrBins bins) {
    constexpr int H = K / 4;
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const unsigned lane = lane_id();
    const uint32_t half = lane & (H - 1), vlane = lane / H;
    clear_next(bins);
    if (blockIdx.x == 0 && threadIdx.x < K) a.dang_next[threadIdx.x] = 0.0;
    __shared__ MsConst<K> c;
    if (threadIdx.x < K) {
        c.bonus[threadIdx.x] = ff_of((1.0 - a.d) + a.d * a.dang_in[threadIdx.x]);
        c.src[threadIdx.x] = a.src[threadIdx.x];
        if (threadIdx.x == 0) c.d = ff_of(a.d);
    }
    __syncthreads();
    for_units(bins, [&](uint64_t u) {
        uint32_t source;
        if (u < bins.n_items) {  // a piece of a long row
            const uint2 item = bins.items[u];
            const OffT row = off[item.x], end = off[(uint64_t)item.x + 1];
            const OffT b = row + (OffT)item.y * (OffT)bins.chunk;
            const OffT e = end - b > (OffT)bins.chunk ? b + (OffT)bins.chunk : end;
            const ff part = ms_row32<K>(a, b, e, half, source);
            const uint32_t pieces = (uint32_t)(((uint64_t)(end - row) + bins.chunk - 1) / bins.chunk);
            const uint64_t first = u - item.y;
            if (ms_owner<H, 32 / H>()) bins.partial[u * K + source] = make_float2(part.hi, part.lo);
            __threadfence();
            __syncwarp();
            uint32_t done = 0;
            if (lane == 0) {
                done = atomicAdd(&bins.left[first], 1u) + 1u;
                __threadfence();
            }
            if (__shfl_sync(0xffffffffu, done, 0) != pieces) return;
            if (lane < K) {  // a lane per source adds the pieces in order
                ff sum{0.f, 0.f};
                for (uint32_t i = 0; i < pieces; i++) {
                    const float2 p = __ldcg(&bins.partial[(first + i) * K + lane]);
                    sum = ff_add(sum, ff{p.x, p.y});
                }
                a.cout[(uint64_t)item.x * K + lane] = ms_value<OffT, K>(a, c, item.x, end - row, lane, sum);
            }
            if (lane == 0) bins.left[first] = 0u;
            return;
        }
        u -= bins.n_items;
        const bool rest = u >= bins.big_units + bins.mid_units;
        const bool mid = !rest && mid_unit(bins, u);
        if (!rest && !mid) {  // a warp per row
            for (uint32_t t = 0; t < bins.big_step; t++) {
                const uint64_t i = u * bins.big_step + t;
                if (i >= bins.n_big) break;
                const uint32_t v = bins.big[i];
                const OffT b = off[v], e = off[(uint64_t)v + 1];
                const ff sum = ms_row32<K>(a, b, e, half, source);
                if (ms_owner<H, 32 / H>()) a.cout[(uint64_t)v * K + source] = ms_value<OffT, K>(a, c, v, e - b, source, sum);
            }
            return;
        }
        if (mid) {  // 8 single-source lanes per row
            const uint64_t i = u * bins.mid_step + lane;
            const bool mine = lane < bins.mid_step && i < bins.n_mid;
            const uint32_t v = mine ? bins.mid[i] : 0u;
            const OffT b = mine ? off[v] : (OffT)0, e = mine ? off[(uint64_t)v + 1] : (OffT)0;
            for (uint32_t t = 0; t < bins.mid_step; t += 4 / H) {
                const int from = (int)(t + lane / (8 * H));
                const OffT rb = __shfl_sync(0xffffffffu, b, from), re = __shfl_sync(0xffffffffu, e, from);
                const uint32_t rv = __shfl_sync(0xffffffffu, v, from);
                ff acc[1][4], sum;
                ms_run<K, kPrkBatch, 1, 8, 0>(a, rb + (OffT)(vlane & 7u), re, half, acc);
                source = half * 4 + ms_tree<H, 8>(acc[0], sum);
                if (rb < re && ms_owner<H, 8>()) a.cout[(uint64_t)rv * K + source] = ms_value<OffT, K>(a, c, rv, re - rb, source, sum);
            }
            return;
        }
        u -= bins.big_units + bins.mid_units;
        const uint64_t end = min(a.n, (u + 1) * bins.small_step);
        for (uint64_t v = u * bins.small_step + vlane; v < end; v += 32 / H) {  // H threads per row
            const OffT b = off[v], e = off[v + 1], deg = e - b;
            if ((uint64_t)deg > kPrSmall) continue;
            if (deg == 0) {
                bool is_src = false;
#pragma unroll
                for (int s = 0; s < K; s++) is_src |= v == c.src[s];
                if (!is_src) continue;
            }
            ff acc[1][4];
            ms_run<K, kPrkBatch, 1, 1, 0>(a, b, e, half, acc);
            float x[4];
#pragma unroll
            for (int s = 0; s < 4; s++) x[s] = ms_value<OffT, K>(a, c, (uint32_t)v, deg, half * 4 + s, acc[0][s]);
            *reinterpret_cast<float4 *>(a.cout + v * K + 4 * half) = make_float4(x[0], x[1], x[2], x[3]);
        }
    });
}

// r0 = e_src per lane: contribution 1/deg(src) at the source, dangling 1 for
// an isolated source (as k_pr_init for one source).
template <class OffT, int K>
__global__ void k_prk_init(const OffT *off, const uint32_t *src, float *c, double *dang) {
    unsigned s = threadIdx.x;
    if (s >= (unsigned)K) return;
    uint32_t v = src[s];
    dang[s] = 0.0;
    if (v == 0xFFFFFFFFu) return;
    OffT deg = off[(uint64_t)v + 1] - off[v];
    if (deg == 0) dang[s] = 1.0;
    else c[(uint64_t)v * K + s] = 1.f / (float)deg;
}

// rank[x*K + s] -> out[s*n + v] for s < k (32 vertices x K sources per tile),
// x = newid[v] on a regrouped graph (else v).
template <int K>
__global__ void __launch_bounds__(kBlock) k_prk_out(const float *rank, uint64_t n, uint32_t k,
                                                    const uint32_t *newid, float *out) {
    __shared__ float t[32][K + 1];
    for (uint64_t v0 = (uint64_t)blockIdx.x * 32; v0 < n; v0 += (uint64_t)gridDim.x * 32) {
        for (int i = threadIdx.x; i < 32 * K; i += kBlock) {
            int vv = i / K, s = i % K;
            if (v0 + vv < n) t[vv][s] = rank[(newid ? (uint64_t)newid[v0 + vv] : v0 + vv) * K + s];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 32 * K; i += kBlock) {
            int s = i / 32, vv = i % 32;
            if ((uint32_t)s < k && v0 + vv < n) out[(uint64_t)s * n + v0 + vv] = t[vv][s];
        }
        __syncthreads();
    }
}

// Bin construction, in two passes over contiguous vertex ranges (one per
// CTA) so that each list keeps ascending row order.  counts[blk*4 + t]:
// rows of `mid`, rows of `big`, chunk items (word 2 unused).
template <class OffT>
__global__ void __launch_bounds__(kBlock) k_pr_bin_count(const OffT *off, uint64_t n, uint32_t mid, uint32_t chunk,
                                                         unsigned long long *counts) {
    uint64_t per = (n + gridDim.x - 1) / gridDim.x;
    uint64_t v0 = blockIdx.x * per, v1 = min(n, v0 + per);
    unsigned long long cm = 0, cb = 0, ci = 0;
    for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
        uint64_t deg = (uint64_t)(off[v + 1] - off[v]);
        if (deg <= kPrSmall) continue;
        if (deg <= mid) cm++;
        else if (deg <= chunk) cb++;
        else ci += (deg + chunk - 1) / chunk;
    }
    cm = block_reduce_sum(cm);
    cb = block_reduce_sum(cb);
    ci = block_reduce_sum(ci);
    if (threadIdx.x == 0) {
        counts[blockIdx.x * 4 + 0] = cm;
        counts[blockIdx.x * 4 + 1] = cb;
        counts[blockIdx.x * 4 + 2] = 0;
        counts[blockIdx.x * 4 + 3] = ci;
    }
}

template <class OffT>
__global__ void __launch_bounds__(kBlock) k_pr_bin_fill(const OffT *off, uint64_t n, uint32_t tmid, uint32_t chunk,
                                                        const unsigned long long *base, uint32_t *mid, uint32_t *big,
                                                        uint2 *items) {
    uint64_t per = (n + gridDim.x - 1) / gridDim.x;
    uint64_t v0 = blockIdx.x * per, v1 = min(n, v0 + per);
    unsigned long long bm = base[blockIdx.x * 4 + 0], bb = base[blockIdx.x * 4 + 1];
    unsigned long long bi = base[blockIdx.x * 4 + 3];
    for (uint64_t c0 = v0; c0 < v1; c0 += blockDim.x) {
        uint64_t v = c0 + threadIdx.x;
        uint64_t deg = v < v1 ? (uint64_t)(off[v + 1] - off[v]) : 0;
        unsigned long long fm = deg > kPrSmall && deg <= tmid, fb = deg > tmid && deg <= chunk;
        unsigned long long fi = deg > chunk ? (deg + chunk - 1) / chunk : 0;
        unsigned long long tm, tb, ti;
        unsigned long long pm = block_exclusive_scan(fm, tm);
        unsigned long long pb = block_exclusive_scan(fb, tb);
        unsigned long long pi = block_exclusive_scan(fi, ti);
        if (fm) mid[bm + pm] = (uint32_t)v;
        if (fb) big[bb + pb] = (uint32_t)v;
        for (unsigned long long i = 0; i < fi; i++) items[bi + pi + i] = make_uint2((uint32_t)v, (uint32_t)i);
        bm += tm;
        bb += tb;
        bi += ti;
    }
}

// Longest row of 8 lanes and edges per piece of a long row.  On a small graph
// an iteration is as long as its longest unit of work, so rows are cut finer
// there: pieces of m / 4096 edges (a power of two, 256 at least), 8 lanes a row
// up to 1/16 of that (32 at least).  8 sources, 20 iterations, with 4096 / finer
// pieces: 2^18 vertices 2.10 / 1.25 ms, 2^16 1.28 / 0.55, 2^14 0.99 / 0.25; one
// source: 0.83 / 0.89, 0.44 / 0.41, 0.30 / 0.22.  Values tuned below the built-in ones
// (256 and 4096) are limits besides; larger ones shrink in the same proportion.
void pr_limits(const ptg_tuning &t, uint64_t m, uint32_t &mid, uint32_t &chunk) {
    uint32_t fine = 256;
    while (fine < 4096 && (uint64_t)fine * 2 * 4096 <= m) fine *= 2;
    const uint32_t fine_mid = std::max(32u, fine / 16);
    chunk = t.pr_chunk <= 4096 ? std::min(t.pr_chunk, fine) : (uint32_t)((uint64_t)t.pr_chunk * fine / 4096);
    mid = t.pr_mid <= 256 ? std::min(t.pr_mid, fine_mid)
                          : std::max(fine_mid, (uint32_t)((uint64_t)t.pr_mid * fine / 4096));
}

template <class OffT>
void build_pr_bins(ptg_graph *g) {
    ptg_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const OffT *off = g->d_off.as<OffT>();
    const int nb = (int)std::min<uint64_t>(1024, std::max<uint64_t>(1, (g->n + kBlock - 1) / kBlock));
    DevBuf counts;
    counts.ensure((uint64_t)nb * 4 * 8);
    uint32_t mid, chunk;
    pr_limits(ctx->tuning, g->m, mid, chunk);
    launch(ctx, "k_pr_bin_count", k_pr_bin_count<OffT>, nb, kBlock, 0, st, off, g->n, mid, chunk,
           counts.as<unsigned long long>());
    std::vector<unsigned long long> h((size_t)nb * 4);
    PTG_CUDA_TRY(cudaMemcpyAsync(h.data(), counts.p, h.size() * 8, cudaMemcpyDeviceToHost, st));
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    unsigned long long tot[4] = {0, 0, 0, 0};
    for (int b = 0; b < nb; b++)
        for (int t = 0; t < 4; t++) {
            unsigned long long x = h[(size_t)b * 4 + t];
            h[(size_t)b * 4 + t] = tot[t];
            tot[t] += x;
        }
    PTG_CUDA_TRY(cudaMemcpyAsync(counts.p, h.data(), h.size() * 8, cudaMemcpyHostToDevice, st));
    g->d_pr_mid.ensure(std::max<unsigned long long>(tot[0], 1) * 4);
    g->d_pr_big.ensure(std::max<unsigned long long>(tot[1], 1) * 4);
    g->d_pr_items.ensure(std::max<unsigned long long>(tot[3], 1) * 8);
    launch(ctx, "k_pr_bin_fill", k_pr_bin_fill<OffT>, nb, kBlock, 0, st, off, g->n, mid, chunk,
           (const unsigned long long *)counts.p, g->d_pr_mid.as<uint32_t>(), g->d_pr_big.as<uint32_t>(),
           g->d_pr_items.as<uint2>());
    PTG_CUDA_TRY(cudaStreamSynchronize(st));
    g->n_pr_mid = tot[0];
    g->n_pr_big = tot[1];
    g->n_pr_items = tot[3];
    g->pr_mid = mid;
    g->pr_chunk = chunk;
    g->pr_bins_built = true;
}

// The bins of a graph as units of work for `warps` warps, with the workspace
// that an iteration's kernel needs (partial sums, their counters, three unit
// counters used in turn).  Small graphs take small units: every warp has some.
PrBins make_bins(ptg_graph *g, int sources, uint64_t warps, unsigned *&counters) {
    Workspace &ws = g->ctx->ws;
    PrBins b{};
    b.mid = g->d_pr_mid.as<uint32_t>();
    b.n_mid = g->n_pr_mid;
    b.big = g->d_pr_big.as<uint32_t>();
    b.n_big = g->n_pr_big;
    b.items = g->d_pr_items.as<uint2>();
    b.n_items = g->n_pr_items;
    b.chunk = g->pr_chunk;
    auto step = [&](uint64_t rows, uint64_t most, uint64_t unit) {  // rows per unit, a multiple of `unit`
        return (uint32_t)(std::min(most, std::max<uint64_t>(1, rows / (warps * 4 * unit))) * unit);
    };
    b.big_step = step(b.n_big, 8, 1);
    b.mid_step = step(b.n_mid, 8, 4);
    b.small_step = step(g->n, 16, 32);
    b.big_units = (b.n_big + b.big_step - 1) / b.big_step;
    b.mid_units = (b.n_mid + b.mid_step - 1) / b.mid_step;
    b.small_units = (g->n + b.small_step - 1) / b.small_step;
    const uint64_t rows = std::max<uint64_t>(1, b.big_units + b.mid_units);  // < 2^32 (ids are 32-bit)
    b.mid_share = ((b.mid_units << 32) + rows - 1) / rows;
    const uint64_t partial_bytes = std::max<uint64_t>(b.n_items, 1) * sources * sizeof(float2);
    constexpr uint64_t kCounters = 3 * kSlices * kSlicePad;
    ws.aux.ensure(partial_bytes + (b.n_items + kCounters) * 4);
    b.partial = ws.aux.as<float2>();
    counters = reinterpret_cast<unsigned *>(ws.aux.as<char>() + partial_bytes);
    b.left = counters + kCounters;
    PTG_CUDA_TRY(cudaMemsetAsync(counters, 0, (b.n_items + kCounters) * 4, g->ctx->stream));
    return b;
}

// Warps take units until there are none, so CTAs past those that an SM holds at
// once (ctas_per_sm) would only begin when the work is done: a tuning that asks
// for more gets as many as fit.
int pr_grid(ptg_graph *g, int ctas_per_sm, int sources, PrBins &bins) {
    const int per_sm = std::min(ctas_per_sm, (int)g->ctx->tuning.pr_ctas_per_sm);
    const uint64_t units = bins.n_items + bins.big_units + bins.mid_units + bins.small_units;
    const int grid = grid_for(units, kBlock / 32, g->ctx->sm_count * per_sm);
    // From 2^27 edges on the units are long enough for one counter, which then
    // balances best: 20 iterations at RMAT-24 28.9 ms (16 slices: 29.0), RMAT-23
    // 14.2 (15.0), RMAT-22 6.7 (6.3), RMAT-20 2.1 (1.5), RMAT-18 0.95 (0.63); of 8
    // sources, whose units are longer, 59.3 (8 slices: 60.2), 28.0 (30.6), 13.5
    // (13.6; 16 slices 15.0), 3.43 (3.29).
    bins.slices = std::min<unsigned>(g->m >= (1ull << 27) ? 1u : sources > 1 ? kSlices / 2 : kSlices, (unsigned)grid);
    return grid;
}

template <class OffT>
void pagerank_impl(ptg_graph *g, bool personalized, uint32_t src, double damping, uint32_t iters,
                   float *d_rank, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n, m = g->m;
    const int sms = ctx->sm_count;
    if (!g->pr_bins_built) build_pr_bins<OffT>(g);
    ws.aux2.ensure(2 * n * 4 + 64);                          // contrib ping-pong
    ws.bsum.ensure(1024 * 8);
    float *contrib[2] = {ws.aux2.as<float>(), ws.aux2.as<float>() + n};
    double *dang = ws.bsum.as<double>();  // three, used in turn: read, added to, cleared
    PTG_CUDA_TRY(cudaMemsetAsync(dang, 0, 64, st));
    int fill_grid = grid_for(n, kBlock, sms * 8);
    const OffT *off = g->d_off.as<OffT>();
    unsigned *counters;
    PrBins bins = make_bins(g, 1, (uint64_t)sms * kPrMinBlocks * (kBlock / 32), counters);
    const int grid = pr_grid(g, kPrMinBlocks, 1, bins);
    launch(ctx, "k_pr_init", k_pr_init<OffT>, fill_grid, kBlock, 0, st, off, n, personalized ? 1 : 0, src,
           contrib[0], &dang[0]);
    for (uint32_t it = 0; it < iters; it++) {
        PrArgs a;
        a.n = n;
        a.m = m;
        a.off = off;
        a.col = g->d_col.as<uint32_t>();
        a.contrib_in = contrib[it & 1];
        a.contrib_out = contrib[(it & 1) ^ 1];
        a.rank_out = (it + 1 == iters) ? d_rank : nullptr;
        a.dangling_in = &dang[it % 3];
        a.dangling_out = &dang[(it + 1) % 3];
        a.dangling_next = &dang[(it + 2) % 3];
        a.d = damping;
        a.teleport = (1.0 - damping) / (double)n;
        a.spread = damping / (double)n;
        a.personalized = personalized ? 1 : 0;
        a.src = src;
        bins.counter = counters + it % 3 * (kSlices * kSlicePad);
        bins.counter_next = counters + (it + 1) % 3 * (kSlices * kSlicePad);
        launch(ctx, "k_pr_iter", k_pr_iter<OffT>, grid, kBlock, 0, st, a, bins);
        rr.edges_relaxed += m;
    }
    PTG_CUDA_TRY(cudaGetLastError());
    rr.iterations = iters;
}

template <class OffT, int K>
void ppr_multi_impl(ptg_graph *g, const uint32_t *h_srcs, uint32_t k, float *d_rows, double damping,
                    uint32_t iters, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n;
    const int sms = ctx->sm_count;
    if (!g->pr_bins_built) build_pr_bins<OffT>(g);
    ws.aux2.ensure(2 * n * K * 4 + 64);                          // values ping-pong
    ws.bsum.ensure(1024 * 8);
    float *c[2] = {ws.aux2.as<float>(), ws.aux2.as<float>() + n * K};
    double *dang = ws.bsum.as<double>();                            // [3][K], used in turn
    uint32_t *d_src = reinterpret_cast<uint32_t *>(dang + 3 * K);  // [K]
    uint32_t lanes[K];
    for (int s = 0; s < K; s++) lanes[s] = (uint32_t)s < k ? h_srcs[s] : 0xFFFFFFFFu;
    PTG_CUDA_TRY(cudaMemsetAsync(dang, 0, 3 * K * 8, st));
    PTG_CUDA_TRY(cudaMemcpyAsync(d_src, lanes, sizeof(lanes), cudaMemcpyHostToDevice, st));
    map_sources_dev(g, d_src, K);
    PTG_CUDA_TRY(cudaMemsetAsync(c[0], 0, 2 * n * K * 4, st));  // both buffers (isolated vertices stay 0)
    const OffT *off = g->d_off.as<OffT>();
    unsigned *counters;
    PrBins bins = make_bins(g, K, (uint64_t)sms * kPrkMinBlocks * (kBlock / 32), counters);
    const int grid = pr_grid(g, kPrkMinBlocks, K, bins);
    launch(ctx, "k_prk_init", k_prk_init<OffT, K>, 1, 32, 0, st, off, (const uint32_t *)d_src, c[0], dang);
    for (uint32_t it = 0; it < iters; it++) {
        MsArgs a;
        a.n = n;
        a.off = off;
        a.col = g->d_col.as<uint32_t>();
        a.cin = c[it & 1];
        a.cout = c[(it & 1) ^ 1];
        a.dang_in = dang + (it % 3) * K;
        a.dang_out = dang + ((it + 1) % 3) * K;
        a.dang_next = dang + ((it + 2) % 3) * K;
        a.src = d_src;
        a.d = damping;
        a.last = it + 1 == iters;
        bins.counter = counters + it % 3 * (kSlices * kSlicePad);
        bins.counter_next = counters + (it + 1) % 3 * (kSlices * kSlicePad);
        launch(ctx, "k_prk_iter", k_prk_iter<OffT, K>, grid, kBlock, 0, st, a, bins);
        rr.edges_relaxed += g->m;
    }
    launch(ctx, "k_prk_out", k_prk_out<K>, grid_for((n + 31) / 32, 1, sms * 8), kBlock, 0, st,
           (const float *)c[iters & 1], n, k, (const uint32_t *)(g->relabeled ? g->d_newid.p : nullptr), d_rows);
    PTG_CUDA_TRY(cudaGetLastError());
    rr.iterations += iters;
}

}  // namespace

// Personalized PageRank of k <= 8 sources in one pass (4- or 8-wide values);
// each row of d_rows equals run_pagerank(personalized, that source) bit for bit.
void run_ppr_multi(ptg_graph *g, const uint32_t *h_srcs, uint32_t k, float *d_rows, double damping, uint32_t iters,
                   RunResult &rr) {
    PTG_REQUIRE(!g->out_of_core, PTG_ERR_UNSUPPORTED, "PageRank needs the graph resident in HBM");
    PTG_REQUIRE(g->symmetric, PTG_ERR_UNSUPPORTED, "pull PageRank needs a symmetric CSR (PTG_CSR_SYMMETRIC)");
    PTG_REQUIRE(k >= 1 && k <= 8, PTG_ERR_INVALID, "a multi-source PageRank pass holds 1..8 sources");
    PTG_REQUIRE(iters >= 1, PTG_ERR_INVALID, "PageRank needs at least one iteration");
    if (g->off64) {
        if (k <= 4) ppr_multi_impl<unsigned long long, 4>(g, h_srcs, k, d_rows, damping, iters, rr);
        else ppr_multi_impl<unsigned long long, 8>(g, h_srcs, k, d_rows, damping, iters, rr);
    } else {
        if (k <= 4) ppr_multi_impl<uint32_t, 4>(g, h_srcs, k, d_rows, damping, iters, rr);
        else ppr_multi_impl<uint32_t, 8>(g, h_srcs, k, d_rows, damping, iters, rr);
    }
}

// Degree bins of a resident graph, built now rather than on first use.
void pr_prepare_graph(ptg_graph *g) {
    if (g->out_of_core || !g->symmetric || g->pr_bins_built) return;
    if (g->off64) build_pr_bins<unsigned long long>(g);
    else build_pr_bins<uint32_t>(g);
}

void run_pagerank(ptg_graph *g, bool personalized, uint32_t src, double damping, uint32_t iters,
                  float *d_rank, RunResult &rr) {
    PTG_REQUIRE(!g->out_of_core, PTG_ERR_UNSUPPORTED, "PageRank needs the graph resident in HBM");
    PTG_REQUIRE(g->symmetric, PTG_ERR_UNSUPPORTED,
                "pull PageRank needs a symmetric CSR (PTG_CSR_SYMMETRIC)");
    float *rank = d_rank;
    if (g->relabeled) {
        // ranks in the stored vertex order, mapped to caller ids after
        if (personalized) src = map_source_host(g, src);
        g->ctx->ws.relab[0].ensure(g->n * 4);
        rank = g->ctx->ws.relab[0].as<float>();
    }
    if (g->off64) pagerank_impl<unsigned long long>(g, personalized, src, damping, iters, rank, rr);
    else pagerank_impl<uint32_t>(g, personalized, src, damping, iters, rank, rr);
    if (g->relabeled) unpermute_f32(g, rank, d_rank);
}

}  // namespace ptg

// For the tests: the limits that a graph of m edges gets.
extern "C" void ptg_internal_pr_limits(const ptg_tuning *t, uint64_t m, uint32_t *mid, uint32_t *chunk) {
    ptg::pr_limits(*t, m, *mid, *chunk);
}
