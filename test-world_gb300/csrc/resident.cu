// resident.cu - whole traversals of an in-HBM graph in one launch: BFS
// (direction-optimizing), SSSP (near/far buckets over integer atomicMin) and
// CC min-label propagation.
//
// Reference path replaced (ptGraph/main.cu): the host loops of
// bfsCaculateInOpt 1180-1418, ssspCaculateInOpt 678-889 and ccCaculateInOpt
// 222-440 with their relax and compaction kernels (gpu_kernels.cu:3-172).
//
// A search has a handful of levels (RMAT: 5-8 of BFS, 10-25 of SSSP), and
// with three to six launches, a compaction pass and a host decision each, a
// level cost 30-40 us before its edges were looked at.  Here one cooperative
// launch runs all levels: its CTAs meet at a grid barrier, read the level's
// counters and all take the same decision (push or pull, next bucket, end).
//
//  * The frontier is three lists written by the warps that find its vertices,
//    so there is no degree scan and no row search per edge: vertices of up to
//    kFewDeg and up to kSmallDeg edges, taken by 8 lanes each (16 or 4 of them
//    per warp and step: 8 edges in flight per lane either way, a 32-byte
//    sector at a time), and longer ones with a running count of their
//    kPiece-edge pieces, of which every warp takes an equal run.  (One item per
//    64 edges made the warp that finds a hub write thousands of items: 1.0 ms
//    in one level of an RMAT-24 search.)
//  * A found vertex is claimed with the result of an atomicOr on a bitmap, so
//    it is queued once.  Claimed vertices collect in a buffer of the warp's
//    own in shared memory and leave it 64 at a time: offsets read side by
//    side, one atomic on a list's tail per 64 vertices (one per find
//    serialised on that address).
//  * BFS pull rounds (each unvisited vertex looks for a parent in the frontier
//    bitmap) when the frontier's edges outweigh the unvisited ones (Beamer).
//  * SSSP parks vertices at or above the threshold in a bitmap; when the near
//    frontier is empty one pass over them takes those below the next threshold
//    and finds the smallest distance above it, from which an empty bucket goes
//    on.  Buckets whose edges cost less than the bucket itself double the
//    width.
//  * A heavy SSSP round pulls when the edges carry the same weight both ways:
//    only vertices above the frontier's least distance plus the least weight
//    can still improve, on RMAT-24 with 119 M edges in the round whose
//    frontier has 307 M.
//
// Phases hand data over through global memory across the grid barrier (its
// acquire makes earlier phases' stores visible to ordinary loads).  Within a
// phase a stale read is harmless by construction: distances only fall, a
// vertex improved during a phase is claimed for the next one, and claims are
// atomic.  Every wait at the barrier is bounded.
//
// What bounds it: a small graph's level is a chain of dependent reads and the
// barrier, 5-10 us; the heavy SSSP rounds of RMAT-24 probe 150-260 G targets/s,
// near what PageRank's gathers reach from L2 (one 32-byte sector each): a
// round of 307 M edges took 1170 us as a push and takes 710 as a pull.  Staging
// the edges ahead with cp.async and dropping candidates by the largest distance
// among the hubs changed neither.  Per search, before -> now: BFS on RMAT-16 214
// -> 83 us, on RMAT-24 590 -> 420 us; SSSP on RMAT-24 6.4-6.5 -> 3.2-3.7 ms (over
// the machines that it was measured on); a served mix of small graphs 8.8 -> 6.5
// ms (5.4 with PageRank's one launch per iteration).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ptg_device.cuh"

namespace ptg {
namespace {

typedef unsigned long long u64;

constexpr int kWarps = kBlock / 32;
constexpr uint32_t kFewDeg = 16;     // edges of a vertex that 8 lanes take two at a time
constexpr uint32_t kSmallDeg = 128;  // edges of a vertex that 8 lanes take (two steps of 8 each)
constexpr uint32_t kPiece = 256;     // edges of a longer vertex that a warp takes at a time
constexpr int kBuf = 320;       // claimed vertices a warp holds: 63 left over + 32 lanes x 8 edges
constexpr int kBuWords = 16;    // frontier bitmap words per warp and pull step, at most
constexpr unsigned kErrOverflow = 1u, kErrBarrier = 2u, kErrLimit = 4u;
// SSSP buckets with fewer edges than this (or than half the vertices) double
// the width of the next ones: such a bucket's two passes over the parked
// vertices and its barriers (15 us, 60 us with 8 M parked) outweigh its
// relaxations.  From width 6, with and without: RMAT-24 24 rounds and 3.48 ms a
// search against 49 and 3.62, RMAT-22 1.13 against 1.35 ms, RMAT-20 0.60 against
// 0.79, 4 K vertices 0.19 against 0.29.
constexpr u64 kWideEdges = 1ull << 21;

// Every thread takes the launch's decisions for itself, from words that it reads
// after a barrier.  A thread may be late with that read (another lane's kernels on
// its SM, a context switch), while others are on their way to the next barrier
// already, so no word that decides is written between the barrier before its read
// and the one after:
//   found, edges, few, items, bigs, least  the frontier's, by level % 3: a level reads
//       its own, adds to the next one's and clears the one after that, whose last
//       reader was the level before.  A bucket pass of SSSP fills the lists of the
//       present level (their tails and `least` are read by the round behind its
//       barrier only), but what it found it counts elsewhere:
//   bucket_found, bucket_edges, far_min    by pass % 3: a pass adds to its own, reads
//       those of the pass before and clears the next one's
//   cands                                  by level % 4: read by the next level, cleared
//       three levels on
//   pull_edges, pull_items, pull_bigs      by heavy round % 2: cleared behind the barrier
//       that the following heavy round counts up to
struct ResCtl {
    unsigned arrive, gen;           // grid barrier
    unsigned error;
    // per level (slot level % 3): vertices of up to kFewDeg edges, up to
    // kSmallDeg, and longer ones << 32 | their pieces
    u64 few[3], items[3], bigs[3];
    u64 found[3], edges[3];         // the frontier's vertices and edges
    u64 bucket_found[3], bucket_edges[3];  // SSSP: those that a bucket pass took, by turn
    u64 far_min[3];                 // SSSP: least distance that stays parked, by turn
    u64 cands[4];                   // unvisited vertices that a pull round looked at (level % 4)
    unsigned chunk[2];              // pull work counter, by level parity
    // SSSP: least distance of the frontier (slot level % 3); edges that a pull
    // round would look at and its lists (items, bigs), by turn
    unsigned least[3];
    u64 pull_edges[2], pull_items[2], pull_bigs[2];
    LevelMsg msg;                   // the outcome, where host memory cannot be mapped
};

struct ResArgs {
    uint64_t n, m;
    const void *off;
    const uint32_t *col, *w;
    uint32_t *value;                // result (BFS: by caller id; else by stored id)
    uint32_t *out;                  // SSSP on a regrouped graph: result by caller id (else nullptr)
    const uint32_t *perm, *newid;   // nullptr: stored in the caller's order
    uint32_t *bm[2], *vis, *far_bm;
    const uint32_t *nz;             // vertices with edges (BFS pull; nullptr: never pull)
    uint32_t *few[2], *q[2];        // vertices of 1..kFewDeg and ..kSmallDeg edges
    uint2 *big[2];                  // longer ones: (vertex, pieces before it)
    uint64_t qcap, bigcap;
    uint32_t src, base, delta, max_iters;
    float alpha, beta;
    int use_far;
    int can_pull;                   // SSSP: the same weight both ways on every edge
    uint32_t min_weight;
    ResCtl *ctl;
    LevelMsg *msg;                  // where the outcome goes (host-mapped, or ctl->msg)
    uint32_t seq;
    u64 barrier_polls;              // polls of the barrier before a CTA gives up
};


__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// All CTAs of the (cooperative) grid meet; false when one of them gave up.  Who
// passes knows that all others had reached it, so what was written before it is
// complete even when a CTA gives up at it.
__device__ bool grid_barrier(ResCtl *c, u64 limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (gridDim.x == 1) {
        __threadfence();
        __syncthreads();
        return true;
    }
    if (threadIdx.x == 0) {
        bool ok = true;
        __threadfence();
        const unsigned gen = *(volatile unsigned *)&c->gen;
        if (atomicAdd(&c->arrive, 1u) == gridDim.x - 1) {
            *(volatile unsigned *)&c->arrive = 0u;
            __threadfence();
            atomicExch(&c->gen, gen + 1u);
        } else {
            u64 polls = 0;
            while (ld_acquire(&c->gen) == gen) {
                if ((++polls & 1023u) == 0 && (*(volatile unsigned *)&c->error & kErrBarrier)) ok = false;
                if (polls > limit) {
                    atomicOr(&c->error, kErrBarrier);
                    ok = false;
                }
                if (!ok) break;
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// A warp's claimed vertices (shared memory) and what they add up to.
struct WarpBuf {
    uint32_t *v;
    uint32_t cnt;
    uint32_t least;  // SSSP: least improved distance below the threshold
    u64 found, edges;
};

// A frontier's lists and counters.
struct Frontier {
    uint32_t *few, *q;
    uint2 *big;
    u64 *nfew, *items, *bigs;
    unsigned *least;  // (may be null)
};

__device__ __forceinline__ Frontier frontier_of(const ResArgs &a, int buf, int slot) {
    return Frontier{a.few[buf],          a.q[buf],   a.big[buf], &a.ctl->few[slot], &a.ctl->items[slot],
                    &a.ctl->bigs[slot], &a.ctl->least[slot]};
}

// The last min(64, cnt) buffered vertices go to the frontier's lists: their
// offsets are read side by side, and one lane per list reserves the places in
// it at the same time (three reservations one after another made a flush as
// long as the relaxations that led to it).
template <class OffT>
__device__ void buf_flush(WarpBuf &b, const ResArgs &a, const Frontier &f) {
    const unsigned lane = lane_id();
    const uint32_t take = min(64u, b.cnt);
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    __syncwarp();
    uint32_t v[2];
    u64 deg[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const bool ok = lane + 32 * h < take;
        v[h] = ok ? b.v[b.cnt - take + lane + 32 * h] : 0u;
        deg[h] = ok ? (u64)(off[(uint64_t)v[h] + 1] - off[v[h]]) : 0ull;
        b.found += ok;
    }
    b.cnt -= take;
    b.edges += deg[0] + deg[1];
    unsigned few[2], mid[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        few[h] = __ballot_sync(0xffffffffu, deg[h] > 0 && deg[h] <= kFewDeg);
        mid[h] = __ballot_sync(0xffffffffu, deg[h] > kFewDeg && deg[h] <= kSmallDeg);
    }
    // longer vertices: entries and pieces counted together, in two halves of a word
    u64 p[2], incl = 0, bigs = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) p[h] = deg[h] > kSmallDeg ? (1ull << 32 | (deg[h] + kPiece - 1) / kPiece) : 0ull;
    if (__any_sync(0xffffffffu, (p[0] | p[1]) != 0)) {
        incl = p[0] + p[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        bigs = __shfl_sync(0xffffffffu, incl, 31);
    }
    const uint32_t nfew = __popc(few[0]) + __popc(few[1]), nmid = __popc(mid[0]) + __popc(mid[1]);
    u64 at = 0;
    if (lane < 3) {
        const u64 add = lane == 0 ? nfew : lane == 1 ? nmid : bigs;
        if (add) at = atomicAdd(lane == 0 ? f.nfew : lane == 1 ? f.items : f.bigs, add);
    }
    u64 at_few = __shfl_sync(0xffffffffu, at, 0), at_mid = __shfl_sync(0xffffffffu, at, 1);
    u64 at_big = __shfl_sync(0xffffffffu, at, 2) + incl - (p[0] + p[1]);
    // (a list cannot overflow: every vertex is listed once)
    const bool full = at_few + nfew > a.n || at_mid + nmid > a.qcap || (at_big + p[0] + p[1]) >> 32 > a.bigcap;
    if (__any_sync(0xffffffffu, full)) {
        if (lane == 0) atomicOr(&a.ctl->error, kErrOverflow);
        return;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if ((few[h] >> lane) & 1u) f.few[at_few + __popc(few[h] & lanemask_lt())] = v[h];
        if ((mid[h] >> lane) & 1u) f.q[at_mid + __popc(mid[h] & lanemask_lt())] = v[h];
        if (p[h]) f.big[at_big >> 32] = make_uint2(v[h], (uint32_t)at_big);
        at_few += __popc(few[h]);
        at_mid += __popc(mid[h]);
        at_big += p[h];
    }
}

// Buffers the lanes' claimed vertices (one each where `mine`).
__device__ __forceinline__ void buf_add(WarpBuf &b, bool mine, uint32_t v) {
    const unsigned mask = __ballot_sync(0xffffffffu, mine);
    if (mine) b.v[b.cnt + __popc(mask & lanemask_lt())] = v;
    b.cnt += __popc(mask);
}

// The phase's finds, added to the level's counters once per warp.
__device__ void buf_total(WarpBuf &b, u64 *found, u64 *edges) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        b.found += __shfl_xor_sync(0xffffffffu, b.found, o);
        b.edges += __shfl_xor_sync(0xffffffffu, b.edges, o);
    }
    if (lane_id() == 0 && b.found) {
        atomicAdd(found, b.found);
        atomicAdd(edges, b.edges);
    }
    b.found = b.edges = 0;
}

template <class OffT>
__device__ __forceinline__ void buf_finish(WarpBuf &b, const ResArgs &a, const Frontier &f, u64 *found, u64 *edges) {
    while (b.cnt) buf_flush<OffT>(b, a, f);
    if (found) buf_total(b, found, edges);
    else b.found = b.edges = 0;  // counted before
    if (f.least) {
        const uint32_t least = __reduce_min_sync(0xffffffffu, b.least);
        if (lane_id() == 0 && least != PTG_UNREACHED) atomicMin(f.least, least);
        b.least = PTG_UNREACHED;
    }
}

// Calls f(i, word of lane i) for the non-zero words of a warp's 32, all lanes
// together: lane l stands for bit l, so a word's vertices are read side by side.
template <class F>
__device__ __forceinline__ void for_words(uint32_t word, F &&f) {
    unsigned some = __ballot_sync(0xffffffffu, word != 0);
    while (some) {
        const int i = __ffs(some) - 1;
        some &= some - 1;
        f(i, __shfl_sync(0xffffffffu, word, i));
    }
}

// Queue of the set bits of a bitmap (bm == nullptr: of all n vertices).
template <class OffT>
__device__ void queue_bits(const ResArgs &a, const uint32_t *bm, const Frontier &f, WarpBuf &b) {
    const unsigned lane = lane_id();
    const uint64_t words = (a.n + 31) / 32, nwarps = (uint64_t)gridDim.x * kWarps;
    for (uint64_t w0 = ((uint64_t)blockIdx.x * kWarps + (threadIdx.x >> 5)) * 32; w0 < words; w0 += nwarps * 32) {
        const uint64_t wd = w0 + lane;
        uint32_t word = 0;
        if (wd < words) {
            const uint64_t left = a.n - wd * 32;
            word = bm ? bm[wd] : (left >= 32 ? 0xffffffffu : (1u << left) - 1u);
        }
        for_words(word, [&](int i, uint32_t bits) {
            buf_add(b, (bits >> lane) & 1u, (uint32_t)((w0 + i) * 32 + lane));
            while (b.cnt >= 64) buf_flush<OffT>(b, a, f);
        });
    }
    buf_finish<OffT>(b, a, f, nullptr, nullptr);
}

// Relaxes up to U edges per lane: targets v (PTG_UNREACHED: none), candidates
// nd.  MODE 0 BFS, 1 SSSP, 2 CC.
template <class OffT, int MODE, int U>
__device__ __forceinline__ void relax_edges(const ResArgs &a, const uint32_t (&v)[U], const uint32_t (&nd)[U],
                                            const uint32_t thr, uint32_t *bm_next, const Frontier &nx, WarpBuf &b) {
    bool claim[U];
    if (MODE == 0) {
        uint32_t seen[U];
#pragma unroll
        for (int i = 0; i < U; i++) seen[i] = v[i] != PTG_UNREACHED ? a.vis[v[i] >> 5] : 0xffffffffu;
#pragma unroll
        for (int i = 0; i < U; i++) claim[i] = !((seen[i] >> (v[i] & 31u)) & 1u);
#pragma unroll
        for (int i = 0; i < U; i++) {
            const uint32_t bit = 1u << (v[i] & 31u);
            if (claim[i]) seen[i] = atomicOr(&a.vis[v[i] >> 5], bit);
        }
#pragma unroll
        for (int i = 0; i < U; i++) {
            const uint32_t bit = 1u << (v[i] & 31u);
            claim[i] = claim[i] && !(seen[i] & bit);
            if (claim[i]) {
                a.value[a.perm ? a.perm[v[i]] : v[i]] = nd[i];
                if (a.nz) atomicOr(&bm_next[v[i] >> 5], bit);
            }
        }
    } else {
        uint32_t cur[U];
#pragma unroll
        for (int i = 0; i < U; i++) cur[i] = v[i] != PTG_UNREACHED ? a.value[v[i]] : 0u;
#pragma unroll
        for (int i = 0; i < U; i++) {
            claim[i] = nd[i] < cur[i];
            if (claim[i]) atomicMin(&a.value[v[i]], nd[i]);
            if (MODE == 1 && claim[i] && nd[i] < thr) b.least = min(b.least, nd[i]);
        }
        uint32_t old[U];
#pragma unroll
        for (int i = 0; i < U; i++) {
            const uint32_t bit = 1u << (v[i] & 31u);
            old[i] = 0xffffffffu;
            if (claim[i]) {
                if (nd[i] < thr) old[i] = atomicOr(&bm_next[v[i] >> 5], bit);
                else if (cur[i] == PTG_UNREACHED) atomicOr(&a.far_bm[v[i] >> 5], bit);
                // (a distance at or above the threshold was parked when it was written)
            }
        }
#pragma unroll
        for (int i = 0; i < U; i++) claim[i] = !((old[i] >> (v[i] & 31u)) & 1u);
    }
    bool any = false;
#pragma unroll
    for (int i = 0; i < U; i++) any |= claim[i];
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int i = 0; i < U; i++) buf_add(b, claim[i], v[i]);
        while (b.cnt >= 64) buf_flush<OffT>(b, a, nx);
    }
}

// Loads edge o of the row piece at `begin` (none at or past len): target and
// candidate value.  MODE 1 adds the weight.
template <class OffT, int MODE>
__device__ __forceinline__ void load_edge(const ResArgs &a, OffT begin, uint32_t len, uint32_t o, uint32_t val, u64 pol,
                                          uint32_t &v, uint32_t &nd) {
    v = o < len ? ld_edge(a.col + begin + o, pol) : PTG_UNREACHED;
    if (MODE == 1) nd = o < len ? val + ld_edge(a.w + begin + o, pol) : PTG_UNREACHED;
    else nd = val;
}

// The vertices of a list, 8 lanes each: PAR * 4 of them per warp and step, up
// to 8 / PAR edges of each per lane.  A warp loads 32 vertices side by side,
// or few enough that every warp has some.
template <class OffT, int MODE, int PAR>
__device__ __forceinline__ void push_list(const ResArgs &a, const uint32_t *q, u64 items, uint32_t level_val,
                                          uint32_t thr, uint32_t *bm_next, const Frontier &nx, WarpBuf &b, u64 pol) {
    constexpr int kEach = 8 / PAR, kStep = PAR * 4;
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const unsigned lane = lane_id(), sub = lane & 7u;
    const u64 warps = (u64)gridDim.x * kWarps, warp = (u64)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const u64 share = (items + warps - 1) / warps;
    const uint32_t per = share >= 32 ? 32u : (uint32_t)max((u64)4, (share + 3) / 4 * 4);
    for (u64 i0 = warp * per; i0 < items; i0 += warps * per) {
        const bool ok = lane < per && i0 + lane < items;
        const uint32_t u = ok ? q[i0 + lane] : 0u;
        const OffT begin = ok ? off[u] : (OffT)0;
        const uint32_t len = ok ? (uint32_t)(off[(uint64_t)u + 1] - begin) : 0u;
        const uint32_t val = MODE == 0 ? level_val + 1u : (ok ? a.value[u] : 0u);
        for (uint32_t s = 0; s < per; s += kStep) {
            OffT eb[PAR];
            uint32_t el[PAR], uv[PAR], most = 0;
#pragma unroll
            for (int p = 0; p < PAR; p++) {
                const uint32_t from = s + 4 * p + (lane >> 3);  // past 31: wraps to a lane, with no edges
                eb[p] = __shfl_sync(0xffffffffu, begin, from & 31u);
                el[p] = __shfl_sync(0xffffffffu, len, from & 31u);
                uv[p] = MODE == 0 ? val : __shfl_sync(0xffffffffu, val, from & 31u);
                if (from >= 32) el[p] = 0;
                most = max(most, el[p]);
            }
            most = __reduce_max_sync(0xffffffffu, most);
            for (uint32_t o = 0; o < most; o += 8 * kEach) {
                uint32_t v[8], nd[8];
#pragma unroll
                for (int i = 0; i < 8; i++)
                    load_edge<OffT, MODE>(a, eb[i / kEach], el[i / kEach], o + sub + 8u * (i % kEach), uv[i / kEach],
                                          pol, v[i], nd[i]);
                relax_edges<OffT, MODE, 8>(a, v, nd, thr, bm_next, nx, b);
            }
        }
    }
}

// One push phase over the frontier `f`; what it finds goes to `nx`.
template <class OffT, int MODE>
__device__ void push_phase(const ResArgs &a, const Frontier &f, uint32_t level_val, uint32_t thr, uint32_t *bm_next,
                           const Frontier &nx, WarpBuf &b, u64 *found, u64 *edges) {
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const unsigned lane = lane_id();
    const u64 warps = (u64)gridDim.x * kWarps, warp = (u64)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const u64 pol = l2_evict_first_policy();
    push_list<OffT, MODE, 4>(a, f.few, *f.nfew, level_val, thr, bm_next, nx, b, pol);
    push_list<OffT, MODE, 1>(a, f.q, *f.items, level_val, thr, bm_next, nx, b, pol);
    // longer vertices: an equal run of pieces per warp, one search for its
    // first, 32 vertices loaded side by side.  After the others: SSSP
    // distances that fall meanwhile reach the hubs' edges (hubs first: 8% more
    // relaxations on RMAT-24).
    const u64 bigs = *f.bigs, pieces = bigs & 0xffffffffull, count = bigs >> 32;
    u64 p = pieces * warp / warps;
    const u64 p1 = pieces * (warp + 1) / warps;
    if (p < p1) {
        u64 at = 0, hi = count;  // last entry with at most p pieces before it
        while (hi - at > 1) {
            const u64 mid = (at + hi) >> 1;
            if (f.big[mid].y <= p) at = mid;
            else hi = mid;
        }
        for (; p < p1 && at < count; at += 32) {
            const bool ok = at + lane < count;
            const uint2 e = ok ? f.big[at + lane] : make_uint2(0u, 0u);
            const OffT row = ok ? off[e.x] : (OffT)0, deg = ok ? off[(uint64_t)e.x + 1] - row : (OffT)0;
            const uint32_t val = MODE == 0 ? level_val + 1u : (ok ? a.value[e.x] : 0u);
            const uint32_t have = (uint32_t)min((u64)32, count - at);
            for (uint32_t j = 0; j < have && p < p1; j++) {
                const OffT ur = __shfl_sync(0xffffffffu, row, j), ud = __shfl_sync(0xffffffffu, deg, j);
                const uint32_t uv = __shfl_sync(0xffffffffu, val, j), us = __shfl_sync(0xffffffffu, e.y, j);
                for (; p < p1; p++) {
                    const u64 k = (p - us) * kPiece;
                    if (k >= (u64)ud) break;
                    const uint32_t len = (uint32_t)min((u64)kPiece, (u64)ud - k);
                    uint32_t v[8], nd[8];
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        load_edge<OffT, MODE>(a, ur + (OffT)k, len, lane + 32u * i, uv, pol, v[i], nd[i]);
                    relax_edges<OffT, MODE, 8>(a, v, nd, thr, bm_next, nx, b);
                }
            }
        }
    }
    buf_finish<OffT>(b, a, nx, found, edges);
}

// SSSP pull (symmetric graphs with the same weight both ways): candidates for
// a vertex over K edges of its row.  Any end below the threshold may give one:
// what is not in the frontier was relaxed before and improves nothing, and
// asking the frontier's bitmap first would be one more random read per edge
// (1060 us instead of 440 for 119 M edges, of which 6.3 M vertices with up to
// kFewDeg edges took 8 lanes each).
template <class OffT, int K>
__device__ __forceinline__ uint32_t pull_edges(const ResArgs &a, OffT begin, uint32_t len, uint32_t o, uint32_t step,
                                               uint32_t thr, u64 pol) {
    uint32_t c[K], w[K], best = PTG_UNREACHED;
#pragma unroll
    for (int i = 0; i < K; i++) {
        const bool ok = o + step * i < len;
        c[i] = ok ? ld_edge(a.col + begin + o + step * i, pol) : PTG_UNREACHED;
        w[i] = ok ? ld_edge(a.w + begin + o + step * i, pol) : 0u;
    }
#pragma unroll
    for (int i = 0; i < K; i++) c[i] = c[i] != PTG_UNREACHED ? a.value[c[i]] : PTG_UNREACHED;
#pragma unroll
    for (int i = 0; i < K; i++)
        if (c[i] < thr) best = min(best, c[i] + w[i]);
    return best;
}

// Vertices above `above` with up to kFewDeg edges, a lane each (the rows of a
// warp's neighbouring vertices are one run of memory, and grouped by degree
// they are equally long); longer ones are listed in `look`.
template <class OffT>
__device__ void sssp_pull_few(const ResArgs &a, uint32_t above, uint32_t thr, uint32_t *bm_next, const Frontier &nx,
                              WarpBuf &b, const Frontier &look, WarpBuf &longer) {
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const uint64_t nthreads = (uint64_t)gridDim.x * kBlock;
    const u64 pol = l2_evict_first_policy();
    for (uint64_t v0 = ((uint64_t)blockIdx.x * kBlock + threadIdx.x) & ~31ull; v0 < a.n; v0 += nthreads) {
        const uint64_t v = v0 + lane_id();
        OffT begin = 0;
        uint32_t len = 0;
        if (v < a.n && a.value[v] > above) {
            begin = off[v];
            len = (uint32_t)(off[v + 1] - begin);
        }
        buf_add(longer, len > kFewDeg, (uint32_t)v);
        while (longer.cnt >= 64) buf_flush<OffT>(longer, a, look);
        if (len > kFewDeg) len = 0;
        const uint32_t most = __reduce_max_sync(0xffffffffu, len);
        if (!most) continue;
        uint32_t best = PTG_UNREACHED;
        for (uint32_t o = 0; o < most; o += 4) best = min(best, pull_edges<OffT, 4>(a, begin, len, o, 1, thr, pol));
        const uint32_t t[1] = {best != PTG_UNREACHED ? (uint32_t)v : PTG_UNREACHED}, nd[1] = {best};
        relax_edges<OffT, 1, 1>(a, t, nd, thr, bm_next, nx, b);
    }
    buf_finish<OffT>(longer, a, look, nullptr, nullptr);
}

// The longer ones: 8 lanes each up to kSmallDeg edges, else a warp per piece
// (an equal run of pieces per warp, as in push_phase).
template <class OffT>
__device__ void sssp_pull_longer(const ResArgs &a, const Frontier &look, uint32_t thr, uint32_t *bm_next,
                                 const Frontier &nx, WarpBuf &b, u64 *found, u64 *edges) {
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const unsigned lane = lane_id(), sub = lane & 7u;
    const u64 warps = (u64)gridDim.x * kWarps, warp = (u64)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const u64 pol = l2_evict_first_policy();
    const u64 bigs = *look.bigs, pieces = bigs & 0xffffffffull, count = bigs >> 32;
    u64 p = pieces * warp / warps;
    const u64 p1 = pieces * (warp + 1) / warps;
    if (p < p1) {
        u64 at = 0, hi = count;  // last entry with at most p pieces before it
        while (hi - at > 1) {
            const u64 mid = (at + hi) >> 1;
            if (look.big[mid].y <= p) at = mid;
            else hi = mid;
        }
        for (; p < p1 && at < count; at++) {
            const uint2 e = look.big[at];
            const OffT row = off[e.x], deg = off[(uint64_t)e.x + 1] - row;
            uint32_t best = PTG_UNREACHED;
            for (; p < p1; p++) {
                const u64 k = (p - e.y) * kPiece;
                if (k >= (u64)deg) break;
                const uint32_t len = (uint32_t)min((u64)kPiece, (u64)deg - k);
                best = min(best, pull_edges<OffT, 8>(a, row + (OffT)k, len, lane, 32, thr, pol));
            }
            best = __reduce_min_sync(0xffffffffu, best);
            const uint32_t t[1] = {lane == 0 && best != PTG_UNREACHED ? e.x : PTG_UNREACHED}, nd[1] = {best};
            relax_edges<OffT, 1, 1>(a, t, nd, thr, bm_next, nx, b);
        }
    }
    const u64 items = *look.items;
    for (u64 i0 = warp * 4; i0 < items; i0 += warps * 4) {
        const u64 i = i0 + (lane >> 3);
        const uint32_t u = i < items ? look.q[i] : 0u;
        const OffT begin = i < items ? off[u] : (OffT)0;
        const uint32_t len = i < items ? (uint32_t)(off[(uint64_t)u + 1] - begin) : 0u;
        const uint32_t most = __reduce_max_sync(0xffffffffu, len);
        uint32_t best = PTG_UNREACHED;
        for (uint32_t o = 0; o < most; o += 64) best = min(best, pull_edges<OffT, 8>(a, begin, len, o + sub, 8, thr, pol));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        const uint32_t t[1] = {sub == 0 && best != PTG_UNREACHED ? u : PTG_UNREACHED}, nd[1] = {best};
        relax_edges<OffT, 1, 1>(a, t, nd, thr, bm_next, nx, b);
    }
    buf_finish<OffT>(b, a, nx, found, edges);
}

// One pull phase of BFS (symmetric graphs): a warp takes `step` bitmap words
// of vertices, lists the unvisited ones with edges, tests two per lane at a
// time (offsets, first four neighbours and their frontier bits in flight
// together) and walks the rest of a row four neighbours at a time; the words
// of the next frontier and of the visited bitmap are written with plain
// stores.  Counts what it finds; builds no queue.
template <class OffT>
__device__ void pull_phase(const ResArgs &a, const uint32_t *bm_cur, uint32_t *bm_next, uint32_t level_val,
                           unsigned *counter, bool late, uint32_t *list, uint32_t *mark, u64 *found, u64 *edges,
                           u64 *cands) {
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    const uint32_t *col = a.col;
    const uint32_t newval = level_val + 1u;
    const unsigned lane = lane_id();
    const uint64_t words = (a.n + 31) / 32;
    // small graphs: fewer words a step, so that every warp has work; with few
    // unvisited vertices left, 8 steps per trip to the counter (a warp's whole
    // share on RMAT-24: 30 us a round otherwise)
    const uint64_t share = words / ((uint64_t)gridDim.x * kWarps) + 1;
    const uint32_t step = share >= kBuWords ? (uint32_t)kBuWords : (uint32_t)share;
    const uint32_t run = late && step == kBuWords ? 8u : 1u;
    u64 nfound = 0, nedges = 0, ncands = 0;
    uint64_t cw0 = 0;
    for (uint32_t turn = run;; turn++, cw0 += step) {
        if (turn == run) {
            if (lane == 0) cw0 = (uint64_t)atomicAdd(counter, 1u) * step * run;
            cw0 = __shfl_sync(0xffffffffu, cw0, 0);
            turn = 0;
        }
        if (cw0 >= words) break;
        const uint64_t wd = cw0 + lane;
        const bool mine = lane < step && wd < words;
        uint32_t visw = 0, cand = 0;
        if (mine) {
            visw = a.vis[wd];
            cand = a.nz[wd] & ~visw;
        }
        const uint32_t cnt = __popc(cand);
        uint32_t pre = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= (unsigned)o) pre += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
        uint32_t pos = pre - cnt;
        ncands += total;
        while (cand) {
            const int bit = __ffs(cand) - 1;
            cand &= cand - 1;
            list[pos++] = (uint32_t)(wd * 32 + bit);
        }
        mark[lane] = 0;
        __syncwarp();
        for (uint32_t i = lane; i < total; i += 64) {
            const bool has2 = i + 32 < total;
            const uint32_t v0 = list[i], v1 = has2 ? list[i + 32] : v0;
            const OffT b0 = off[v0], e0 = off[(uint64_t)v0 + 1];
            const OffT b1 = has2 ? off[v1] : (OffT)0, e1 = has2 ? off[(uint64_t)v1 + 1] : (OffT)0;
            uint32_t c[8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                c[j] = b0 + (OffT)j < e0 ? col[b0 + j] : PTG_UNREACHED;
                c[4 + j] = b1 + (OffT)j < e1 ? col[b1 + j] : PTG_UNREACHED;
            }
            bool f[2] = {false, false};
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (c[j] != PTG_UNREACHED) f[j >> 2] |= bit_test(bm_cur, c[j]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (h == 1 && !has2) break;
                const uint32_t v = h ? v1 : v0;
                const OffT b = h ? b1 : b0, e = h ? e1 : e0;
                bool hit = f[h];
                for (OffT k = b + 4; k < e && !hit; k += 4) {
                    const uint32_t c0 = col[k];
                    const uint32_t c1 = k + 1 < e ? col[k + 1] : c0;
                    const uint32_t c2 = k + 2 < e ? col[k + 2] : c0;
                    const uint32_t c3 = k + 3 < e ? col[k + 3] : c0;
                    hit = bit_test(bm_cur, c0) | bit_test(bm_cur, c1) | bit_test(bm_cur, c2) | bit_test(bm_cur, c3);
                }
                if (hit) {
                    atomicOr(&mark[(v >> 5) - (uint32_t)cw0], 1u << (v & 31u));
                    a.value[a.perm ? a.perm[v] : v] = newval;
                    nedges += (u64)(e - b);
                    nfound++;
                }
            }
        }
        __syncwarp();
        if (mine) {
            const uint32_t f = mark[lane];
            bm_next[wd] = f;
            if (f) a.vis[wd] = visw | f;
        }
        __syncwarp();
    }
    if (lane == 0 && ncands) atomicAdd(cands, ncands);
    WarpBuf b{nullptr, 0, PTG_UNREACHED, nfound, nedges};
    buf_total(b, found, edges);
}

// 4 CTAs per SM: the rounds wait for reads, so warps count.  Push, pull and bucket
// code share the 64 registers that leaves, and SSSP spills 144 bytes (stores; 180
// of loads; 224 and 316 with 64-bit offsets), CC 28 and BFS 40.
template <class OffT, int MODE>
__global__ void __launch_bounds__(kBlock, 4) k_traverse(ResArgs a) {
    __shared__ uint32_t s_buf[kWarps][kBuf];
    __shared__ uint32_t s_list[MODE == 0 ? kWarps : 1][MODE == 0 ? kBuWords * 32 : 1];
    __shared__ uint32_t s_mark[MODE == 0 ? kWarps : 1][32];
    __shared__ uint32_t s_look[MODE == 1 ? kWarps : 1][96];
    const OffT *off = reinterpret_cast<const OffT *>(a.off);
    ResCtl *ctl = a.ctl;
    const unsigned wid = threadIdx.x >> 5;
    const uint64_t tid = (uint64_t)blockIdx.x * kBlock + threadIdx.x, nthreads = (uint64_t)gridDim.x * kBlock;
    const uint64_t words = (a.n + 31) / 32;
    const bool leader = tid == 0;
    WarpBuf buf{s_buf[wid], 0, PTG_UNREACHED, 0, 0};

    // ---- initial state ----
    for (uint64_t i = tid; i < a.n; i += nthreads) a.value[i] = MODE == 2 ? (uint32_t)i : PTG_UNREACHED;
    for (uint64_t i = tid; i < words; i += nthreads) {
        a.bm[0][i] = 0u;
        a.bm[1][i] = 0u;
        if (MODE == 0) a.vis[i] = 0u;
        if (MODE == 1 && a.use_far) a.far_bm[i] = 0u;
    }
    if (leader) {
        for (int i = 0; i < 3; i++) ctl->few[i] = ctl->items[i] = ctl->bigs[i] = ctl->found[i] = ctl->edges[i] = 0;
        for (int i = 0; i < 3; i++) ctl->far_min[i] = ~0ull, ctl->bucket_found[i] = ctl->bucket_edges[i] = 0;
        ctl->chunk[0] = ctl->chunk[1] = 0;
        for (int i = 0; i < 4; i++) ctl->cands[i] = 0;
        for (int i = 0; i < 3; i++) ctl->least[i] = PTG_UNREACHED;
        for (int i = 0; i < 2; i++) ctl->pull_edges[i] = ctl->pull_items[i] = ctl->pull_bigs[i] = 0;
        ctl->error = 0;
    }
    if (!grid_barrier(ctl, a.barrier_polls)) return;
    bool queued = MODE != 2;  // the current frontier is in the queue (else only in its bitmap, or all vertices)
    if (MODE != 2) {
        if (blockIdx.x == 0) {
            const uint32_t s = a.newid ? a.newid[a.src] : a.src;
            const u64 deg = (u64)(off[(uint64_t)s + 1] - off[s]);
            if (threadIdx.x == 0) {
                a.value[MODE == 0 && a.perm ? a.src : s] = a.base;
                if (MODE == 0) {
                    a.vis[s >> 5] = 1u << (s & 31u);
                    a.bm[0][s >> 5] = 1u << (s & 31u);
                }
                ctl->least[0] = a.base;
                if (deg > kSmallDeg) {
                    a.big[0][0] = make_uint2(s, 0u);
                    ctl->bigs[0] = 1ull << 32 | (deg + kPiece - 1) / kPiece;
                } else {
                    (deg > kFewDeg ? a.q : a.few)[0][0] = s;
                    (deg > kFewDeg ? ctl->items : ctl->few)[0] = deg ? 1 : 0;
                }
                ctl->found[0] = 1;
                ctl->edges[0] = deg;
            }
        }
        if (!grid_barrier(ctl, a.barrier_polls)) return;
    }

    uint64_t m_unvisited = a.m, edges_done = 0;
    u64 front_E = 0;
    uint32_t iterations = 0, pulls = 0, level = 0, far_turn = 0, pull_turn = 0, late_pulls = 0;
    uint32_t thr = PTG_UNREACHED, steps = 0;
    u64 delta = a.delta, bucket_E = 0;
    if (MODE == 1 && a.use_far) thr = bucket_end(a.base, a.delta);
    bool bottom_up = false, limit = false, scanned = false;
    int cur = 0;
    while (true) {
        // a sign of life for the host, which bounds its wait (a path of 10^8
        // vertices has as many levels); seldom, as a store to host memory holds up
        // the next fence
        if (leader && (++steps & 63u) == 0) ((volatile LevelMsg *)a.msg)->frontier_E = steps;
        const int slot = level % 3, next = (level + 1) % 3, later = (level + 2) % 3;
        // (after a bucket pass: what it took, the round before had found nothing)
        u64 F = scanned ? ctl->bucket_found[(far_turn + 2) % 3] : ctl->found[slot];
        u64 E = scanned ? ctl->bucket_edges[(far_turn + 2) % 3] : ctl->edges[slot];
        const Frontier front = frontier_of(a, cur, slot);
        if (MODE == 2 && level == 0) F = a.n, E = a.m;
        if (F == 0) {
            if (MODE != 1 || !a.use_far || thr == PTG_UNREACHED) break;
            // next bucket: parked vertices below the threshold were settled by
            // the bucket that ends; of the others, those below the next
            // threshold are its frontier.  A bucket without any is tried once
            // more from the least parked distance, which this pass finds too.
            u64 from = thr;
            if (scanned) {
                from = ctl->far_min[(far_turn + 2) % 3];
                if (from == ~0ull) break;
            } else {
                // a bucket with few edges costs its passes over the parked
                // vertices, not its relaxations: wider ones from here on
                if (bucket_E < max(kWideEdges, (u64)a.n / 2)) delta *= 2;
                bucket_E = 0;
            }
            scanned = true;
            const uint32_t to = bucket_end(from, delta);
            if (leader) {
                const int after = (far_turn + 1) % 3;
                ctl->far_min[after] = ~0ull;
                ctl->bucket_found[after] = ctl->bucket_edges[after] = 0;
            }
            uint32_t best = PTG_UNREACHED;
            for (uint64_t w0 = (tid >> 5) * 32; w0 < words; w0 += nthreads) {
                const uint64_t wd = w0 + lane_id();
                uint32_t word = wd < words ? a.far_bm[wd] : 0u;
                const uint32_t had = word;
                // four words' distances in flight: 48 us a pass on RMAT-24, 75
                // with one after the other
                for (int i = 0; i < 32; i += 4) {
                    uint32_t bits[4], d[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) bits[j] = __shfl_sync(0xffffffffu, had, i + j);
                    if (!(bits[0] | bits[1] | bits[2] | bits[3])) continue;
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        d[j] = (bits[j] >> lane_id()) & 1u ? a.value[(w0 + i + j) * 32 + lane_id()] : 0u;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const bool near = ((bits[j] >> lane_id()) & 1u) && d[j] >= thr && d[j] < to;
                        if (near) buf.least = min(buf.least, d[j]);
                        else if (d[j] >= thr) best = min(best, d[j]);
                        buf_add(buf, near, (uint32_t)((w0 + i + j) * 32 + lane_id()));
                        const uint32_t stay = __ballot_sync(0xffffffffu, d[j] >= thr && !near);
                        if ((int)lane_id() == i + j) word = stay;
                    }
                    while (buf.cnt >= 64) buf_flush<OffT>(buf, a, front);
                }
                if (word != had) a.far_bm[wd] = word;
            }
            best = __reduce_min_sync(0xffffffffu, best);
            if (lane_id() == 0 && best != PTG_UNREACHED) atomicMin(&ctl->far_min[far_turn % 3], (u64)best);
            buf_finish<OffT>(buf, a, front, &ctl->bucket_found[far_turn % 3], &ctl->bucket_edges[far_turn % 3]);
            thr = to;
            far_turn++;
            if (!grid_barrier(ctl, a.barrier_polls)) return;
            continue;
        }
        scanned = false;
        if (iterations >= a.max_iters) {
            limit = true;
            break;
        }
        iterations++;
        if (leader) {  // the level after next starts from zero (its slot was read two barriers ago)
            ctl->few[later] = ctl->items[later] = ctl->bigs[later] = ctl->found[later] = ctl->edges[later] = 0;
            ctl->chunk[(level + 1) & 1] = 0;
            ctl->cands[(level + 1) & 3] = 0;
            ctl->least[later] = PTG_UNREACHED;
        }
        if (MODE == 0 && a.nz) {
            const u64 seen_E = level ? E : 0;  // the seed level runs top-down
            if (!bottom_up && (double)seen_E > (double)m_unvisited / a.alpha) bottom_up = true;
            else if (bottom_up && (double)F < (double)a.n / a.beta) {
                // back to push, unless the unvisited vertices have few edges
                // left: a pull round over those is 21-25 us on RMAT-24 where
                // listing 900 K vertices and pushing took 104 us (31 us with
                // 3221 vertices), so for a few levels
                if (m_unvisited * 64 > a.m || ++late_pulls > 4) bottom_up = false;
            }
            m_unvisited = m_unvisited > seen_E ? m_unvisited - seen_E : 0;
        }
        uint32_t *bm_cur = a.bm[cur], *bm_next = a.bm[cur ^ 1];
        bool sssp_pull = false;
        u64 pull_E = 0;
        uint32_t above = 0;
        int turn = 0;
        if (MODE == 1) {
            front_E += E;
            // A heavy round may look at fewer edges from the other side: only
            // vertices above the frontier's least distance plus the least
            // weight can improve.  Their edges are counted first, 35 us on RMAT-24
            // (not when those of all vertices that were in no frontier are too
            // many already).  An edge costs both ways about the same, listing
            // the vertices a quarter of a heavy round: RMAT-24's rounds pull
            // 119 M edges instead of 307 M in 730 us (1170), 32 M instead of
            // 56 M in 350 us (430), and push 46 M against 45 M.
            const u64 most = E / 4 * 3;
            if (a.can_pull && E > max((u64)kSsspPullEdges, (u64)a.m / 16) && (front_E > a.m || a.m - front_E < most)) {
                const uint32_t least = ctl->least[slot];
                above = least + min(a.min_weight, PTG_UNREACHED - 1 - least);
                turn = pull_turn++ & 1;
                u64 sum = 0;
                for (uint64_t v = tid; v < a.n; v += nthreads * 4) {
                    uint32_t d[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) d[i] = v + i * nthreads < a.n ? a.value[v + i * nthreads] : 0u;
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (d[i] > above) sum += (u64)(off[v + i * nthreads + 1] - off[v + i * nthreads]);
                }
                sum = block_reduce_sum(sum);
                if (threadIdx.x == 0 && sum) atomicAdd(&ctl->pull_edges[turn], sum);
                if (!grid_barrier(ctl, a.barrier_polls)) return;
                pull_E = ctl->pull_edges[turn];
                sssp_pull = pull_E < most;
                if (leader) ctl->pull_edges[turn ^ 1] = ctl->pull_items[turn ^ 1] = ctl->pull_bigs[turn ^ 1] = 0;
            }
        }
        if (MODE == 1 && sssp_pull) {
            pulls++;
            edges_done += pull_E;
            bucket_E += E;
            for (uint64_t i = tid; i < words; i += nthreads) bm_cur[i] = 0u;
            // its lists go where the frontier's were
            const Frontier look{a.few[cur], a.q[cur], a.big[cur], &ctl->pull_items[turn] /* (none) */,
                                &ctl->pull_items[turn], &ctl->pull_bigs[turn], nullptr};
            const Frontier nx = frontier_of(a, cur ^ 1, next);
            WarpBuf longer{s_look[wid], 0, PTG_UNREACHED, 0, 0};
            sssp_pull_few<OffT>(a, above, thr, bm_next, nx, buf, look, longer);
            if (!grid_barrier(ctl, a.barrier_polls)) return;
            sssp_pull_longer<OffT>(a, look, thr, bm_next, nx, buf, &ctl->found[next], &ctl->edges[next]);
        } else if (MODE == 0 && bottom_up) {
            // few unvisited vertices left: what the last pull round looked at and did not find
            const bool late = level && !queued && (ctl->cands[(level + 3) & 3] - F) * 64 < a.n;
            pulls++;
            pull_phase<OffT>(a, bm_cur, bm_next, a.base + level, &ctl->chunk[level & 1], late, s_list[wid], s_mark[wid],
                             &ctl->found[next], &ctl->edges[next], &ctl->cands[level & 3]);
            queued = false;
        } else {
            if (!queued) {
                // the frontier came from a pull round (or is every vertex):
                // its queue, and a clear bitmap for the next one
                queue_bits<OffT>(a, MODE == 2 ? nullptr : bm_cur, front, buf);
                for (uint64_t i = tid; i < words; i += nthreads) bm_next[i] = 0u;
                if (!grid_barrier(ctl, a.barrier_polls)) return;
                queued = true;
            }
            edges_done += E;
            bucket_E += E;
            // this level's bitmap is read by nothing any more: clear for the level after next
            for (uint64_t i = tid; i < words; i += nthreads) bm_cur[i] = 0u;
            push_phase<OffT, MODE>(a, front, a.base + level, thr, bm_next,
                                   frontier_of(a, cur ^ 1, next), buf,
                                   &ctl->found[next], &ctl->edges[next]);
        }
        if (!grid_barrier(ctl, a.barrier_polls)) return;
        cur ^= 1;
        level++;
    }
    if (MODE == 1 && a.out) {  // the values by caller id
        for (uint64_t v = tid; v < a.n; v += nthreads) a.out[v] = a.value[a.newid[v]];
        if (!grid_barrier(ctl, a.barrier_polls)) return;
    }
    if (leader) {  // everything was written before the last barrier
        volatile LevelMsg *m = a.msg;
        m->F = iterations;
        m->pad = pulls;
        m->error = *(volatile unsigned *)&ctl->error | (limit ? kErrLimit : 0u);
        m->E = edges_done;
        __threadfence_system();
        m->seq = a.seq;
    }
}

template <class OffT, int MODE>
void launch_traverse(ptg_ctx *ctx, const char *name, ResArgs &a) {
    // 4 CTAs of 256 threads with 64 registers fill an SM's register file; the
    // query makes sure that a cooperative grid fits
    static const int per_sm = [] {
        int x = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x, k_traverse<OffT, MODE>, kBlock, 0) == cudaSuccess ? x : 0;
    }();
    PTG_REQUIRE(per_sm >= 1, PTG_ERR_CUDA, "the traversal kernel does not fit an SM");
    // A small graph's level costs its chain of dependent reads and a barrier
    // over the grid: a CTA per 2048 edges up to 1.5 per SM, and from there one
    // per 16 K edges up to what the tuning allows (4 per SM).  BFS / SSSP of
    // RMAT graphs: 65 K vertices 87 / 280 us with 222 CTAs, 118 / 258 with
    // 608; 32 K vertices 94 / 228 us with 228, 125 / 389 with 28.
    const int sms = ctx->sm_count, most = sms * std::min(per_sm, (int)ctx->tuning.expand_ctas_per_sm);
    const uint64_t work = std::max(a.m, a.n);
    const int grid = std::min(most, std::min(grid_for(work, 2048, most), std::max(sms + sms / 2, grid_for(work, 16384, most))));
    cudaStream_t st = ctx->stream;
    void *args[] = {&a};
    ctx->prof.begin(name, st);
    PTG_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_traverse<OffT, MODE>, dim3(grid), dim3(kBlock), args, 0, st));
    ctx->prof.end(st);
}

// Bitmap of vertices with at least one edge (pull rounds never look at the
// others: on a symmetric graph they are unreachable).
template <class OffT>
__global__ void k_nonzero_bits(const OffT *off, uint64_t n, uint32_t *nz) {
    uint64_t words = (n + 31) / 32;
    for (uint64_t wd = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; wd < words;
         wd += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t bits = 0;
        for (int b = 0; b < 32; b++) {
            uint64_t v = wd * 32 + b;
            if (v < n && off[v + 1] > off[v]) bits |= 1u << b;
        }
        nz[wd] = bits;
    }
}

template <class OffT>
void resident_impl(ptg_graph *g, TravKind kind, ResArgs &a) {
    ptg_ctx *ctx = g->ctx;
    if (kind == TRAV_BFS) launch_traverse<OffT, 0>(ctx, "k_traverse_bfs", a);
    else if (kind == TRAV_SSSP) launch_traverse<OffT, 1>(ctx, "k_traverse_sssp", a);
    else launch_traverse<OffT, 2>(ctx, "k_traverse_cc", a);
}

}  // namespace

// Built once per graph.
void build_nonzero_bits(ptg_graph *g) {
    if (g->d_nzbm.p) return;
    const uint64_t words = (g->n + 31) / 32;
    g->d_nzbm.ensure(words * 4);
    const int grid = grid_for(words, kBlock, g->ctx->sm_count * 8);
    if (g->off64)
        launch(g->ctx, "k_nonzero_bits", k_nonzero_bits<unsigned long long>, grid, kBlock, 0, g->ctx->stream,
               g->d_off.as<unsigned long long>(), g->n, g->d_nzbm.as<uint32_t>());
    else
        launch(g->ctx, "k_nonzero_bits", k_nonzero_bits<uint32_t>, grid, kBlock, 0, g->ctx->stream,
               g->d_off.as<uint32_t>(), g->n, g->d_nzbm.as<uint32_t>());
}

// A traversal of an in-HBM graph.  d_value: BFS levels by caller id; SSSP
// distances by caller id; CC labels (vertex ids of the stored order) by
// stored id.  delta: SSSP bucket width (0: label-correcting rounds).
void run_resident(ptg_graph *g, TravKind kind, uint32_t src, uint32_t *d_value, uint32_t base, uint32_t delta,
                  bool allow_pull, uint32_t max_iters, RunResult &rr) {
    ptg_ctx *ctx = g->ctx;
    Workspace &ws = ctx->ws;
    cudaStream_t st = ctx->stream;
    const uint64_t n = g->n, m = g->m, words = (n + 31) / 32;
    ResArgs a{};
    a.qcap = std::min(n, m / kFewDeg + 1);
    a.bigcap = std::min(n, m / kSmallDeg + 1);
    const uint64_t few_bytes = (n * 4 + 15) / 16 * 16, list_bytes = few_bytes + (a.qcap * 4 + 15) / 16 * 16;
    for (int i = 0; i < 2; i++) {
        ws.q[i].ensure(list_bytes + a.bigcap * sizeof(uint2));
        ws.bm[i].ensure(words * 4);
        a.few[i] = ws.q[i].as<uint32_t>();
        a.q[i] = reinterpret_cast<uint32_t *>(ws.q[i].as<char>() + few_bytes);
        a.big[i] = reinterpret_cast<uint2 *>(ws.q[i].as<char>() + list_bytes);
        a.bm[i] = ws.bm[i].as<uint32_t>();
    }
    if (!ws.res.p) {  // the barrier's words start at zero once; every launch leaves them ready for the next
        ws.res.ensure(sizeof(ResCtl));
        PTG_CUDA_TRY(cudaMemsetAsync(ws.res.p, 0, sizeof(ResCtl), st));
    }
    ensure_level_msg(ws);
    a.ctl = ws.res.as<ResCtl>();
    a.msg = ws.d_msg ? ws.d_msg : &a.ctl->msg;
    a.seq = ++ws.msg_seq;
    a.n = n;
    a.m = m;
    a.off = g->d_off.p;
    a.col = g->d_col.as<uint32_t>();
    a.w = g->d_w.as<uint32_t>();
    a.value = d_value;
    a.src = src;
    a.base = base;
    a.delta = delta;
    a.max_iters = max_iters;
    a.barrier_polls = ctx->barrier_polls;
    a.alpha = ctx->tuning.bfs_alpha;
    a.beta = ctx->tuning.bfs_beta;
    a.use_far = kind == TRAV_SSSP && delta != 0;
    if (g->relabeled) {
        a.newid = g->d_newid.as<uint32_t>();
        if (kind == TRAV_BFS) a.perm = g->d_perm.as<uint32_t>();
        if (kind == TRAV_SSSP) {  // distances are compared: by stored id, mapped at the end
            ws.relab[0].ensure(n * 4);
            a.value = ws.relab[0].as<uint32_t>();
            a.out = d_value;
        }
    }
    if (kind == TRAV_BFS) {
        ws.vis.ensure(words * 4);
        a.vis = ws.vis.as<uint32_t>();
        if (allow_pull) {
            build_nonzero_bits(g);
            a.nz = g->d_nzbm.as<uint32_t>();
        }
    }
    if (a.use_far) {
        ws.farbm.ensure(words * 4);
        a.far_bm = ws.farbm.as<uint32_t>();
    }
    if (kind == TRAV_SSSP && allow_pull) {
        a.can_pull = 1;
        a.min_weight = g->min_weight;
    }
    LevelMsg done{};
    try {
        if (g->off64) resident_impl<unsigned long long>(g, kind, a);
        else resident_impl<uint32_t>(g, kind, a);
        if (ws.d_msg) {
            done = wait_level_msg(ctx, st);
        } else {
            PTG_CUDA_TRY(cudaMemcpyAsync(&done, a.msg, sizeof(done), cudaMemcpyDeviceToHost, st));
            PTG_CUDA_TRY(cudaStreamSynchronize(st));
        }
        PTG_REQUIRE(done.seq == a.seq, PTG_ERR_TIMEOUT, "a traversal's blocks did not all reach a barrier");
    } catch (const Error &) {
        // did the launch end at a barrier?  (Its CTAs publish nothing then.)
        unsigned error = 0;
        const bool gave_up = cudaMemcpyAsync(&error, &a.ctl->error, sizeof(error), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
                             cudaStreamSynchronize(st) == cudaSuccess && (error & kErrBarrier);
        ws.res.release();  // a barrier that was left half-way is not used again
        PTG_REQUIRE(!gave_up, PTG_ERR_TIMEOUT, "a traversal's blocks did not all reach a barrier");
        throw;
    }
    PTG_REQUIRE(!(done.error & kErrOverflow), PTG_ERR_CUDA, "frontier overflow in relax");
    PTG_REQUIRE(!done.error, PTG_ERR_TIMEOUT, "iteration limit reached");
    rr.iterations += done.F;
    rr.bottom_up_rounds += done.pad;
    rr.edges_relaxed = done.E;
}

}  // namespace ptg
