// bd_bfs.cu -- the B200 direction-optimizing BFS (hybrid_bfs) and its C ABI.
//
// Data layout in HBM for one handle (n vertices, arcs = 2m):
//   depth   int32[n]      -1 = unvisited
//   parent  int64[n]      written once per reached vertex; the reference's
//                         -deg / -1 encoding of unreached vertices is filled
//                         in lazily (finalize_parents_kernel) when read
//   vis[2]  uint32[n/32]  visited bitmaps; a bottom-up step reads vis[cur]
//                         (frozen) and writes whole words of vis[cur^1]
//   qs[2]   uint32[n]     frontier queue of vertices with degree < large_deg
//   ql[2], qlb[2]         frontier vertices with degree >= large_deg, with the
//                         prefix sum of their chunk counts (work units of
//                         `chunk` edges spread over all warps)
//   ctrl                  Ctrl block: barrier, Beamer state, step counters
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "bd_bfs_device.cuh"
#include "bd_device_util.cuh"
#include "bd_internal.h"

namespace bd {

namespace {

constexpr int64_t kRecCap = 1 << 15;
constexpr long long kDefaultSpin = 4000000;  // ~2 s of polling

using namespace dev;

// Per-thread accumulators of one step, reduced once per CTA at its end.
struct Local {
    unsigned long long found;
    unsigned long long degsum;
};

// What a step needs of the traversal state, in registers.
struct StepView {
    int dir;
    int level;
    int vis_cur;
    int q_cur;
    int bu_sparse;
    long long f_small;
    long long f_large;
    long long f_chunks;
    long long barrier;
};

__device__ __forceinline__ StepView view_of(const LevelState &s)
{
    StepView v;
    v.dir = s.dir;
    v.bu_sparse = s.bu_sparse;
    v.level = s.level;
    v.vis_cur = s.vis_cur;
    v.q_cur = s.q_cur;
    v.barrier = s.barrier;
    v.f_small = s.f_small;
    v.f_large = s.f_large;
    v.f_chunks = s.f_chunks;
    return v;
}

// Visited-bit lookups.  A plain (L1-cacheable) load is correct here: the
// bitmap a bottom-up step reads is not written during that step, and every
// CTA passes the grid barrier's acquire before the step, after which weak
// loads observe all writes made before the barrier (PTX memory model).
__device__ __forceinline__ uint32_t ld_bits(const uint32_t *p) { return *p; }

// Warp-collective: reserves `count` large-queue slots and `chunks` chunk ids
// for this lane with one atomic for the whole warp.  Slots and chunk ids are
// handed out in the same lane order, so chunk bases stay sorted by slot.
__device__ __forceinline__ void warp_reserve_large(Acc *acc, unsigned count,
                                                   unsigned long long chunks,
                                                   unsigned long long &pos,
                                                   unsigned long long &cbase)
{
    const unsigned ci = warp_incl_scan(count);
    const unsigned long long hi = warp_incl_scan(chunks);
    const unsigned ct = __shfl_sync(kFull, ci, 31);
    const unsigned long long ht = __shfl_sync(kFull, hi, 31);
    unsigned long long old = 0;
    if (lane_id() == 0 && ct) {
        old = atomicAdd(&acc->large_packed, ((unsigned long long)ct << kLargeShift) | ht);
    }
    old = __shfl_sync(kFull, old, 0);
    pos = (old >> kLargeShift) + (ci - count);
    cbase = (old & kChunkMask) + (hi - chunks);
}

// Warp-collective append of up to K discoveries per lane with one atomic
// for all the small-degree ones.
template <int K>
__device__ __forceinline__ void warp_append_k(const BfsParams &p, Acc *acc, int qout,
                                              const bool (&has)[K], const uint32_t (&v)[K],
                                              const int64_t (&deg)[K], Local &loc)
{
    const int lane = lane_id();
    unsigned sm[K];
    bool large[K];
    unsigned total = 0, any_large = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (has[k]) {
            loc.found += 1;
            loc.degsum += (unsigned long long)deg[k];
        }
        large[k] = has[k] && deg[k] >= (int64_t)p.large_deg;
        sm[k] = __ballot_sync(kFull, has[k] && !large[k]);
        total += __popc(sm[k]);
        any_large |= __ballot_sync(kFull, large[k]);
    }
    if (total) {
        unsigned long long base = 0;
        if (lane == 0) { base = atomicAdd(&acc->small_cnt, (unsigned long long)total); }
        base = __shfl_sync(kFull, base, 0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (has[k] && !large[k]) { p.qs[qout][base + __popc(sm[k] & lanemask_lt())] = v[k]; }
            base += __popc(sm[k]);
        }
    }
    if (any_large) {
        unsigned count = 0;
        unsigned long long chunks = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (large[k]) {
                count += 1;
                chunks += (unsigned long long)((deg[k] + p.chunk - 1) / p.chunk);
            }
        }
        unsigned long long pos, cbase;
        warp_reserve_large(acc, count, chunks, pos, cbase);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (large[k]) {
                p.ql[qout][pos] = v[k];
                p.qlb[qout][pos] = cbase;
                pos += 1;
                cbase += (unsigned long long)((deg[k] + p.chunk - 1) / p.chunk);
            }
        }
    }
}

__device__ __forceinline__ int64_t degree_of(const BfsParams &p, uint32_t v)
{
    return __ldg(&p.off[v + 1]) - __ldg(&p.off[v]);
}

// The warps that share a step (the grid's, or CTA 0's) and its counters.
struct Team {
    long long gw, nw;  // this warp among nw
    Acc *acc;
};

constexpr int kILP = 4;

// Top-down claims of a batch of kILP neighbours per lane (hybrid_bfs.cc:83-96):
// visited-bit filter, then the atomicOr that sets the bit decides the single
// winner, which writes depth and parent and joins the next frontier.  Every
// stage issues its kILP memory operations back to back.  The filter reads
// through L1: the barrier before the step emptied it, a bit set since then only
// costs an atomic, and most arcs of a late level lead to vertices visited levels
// ago (top-down at scale 20, six roots: 2.93 ms through L2, 1.75 ms).  (Claiming by atomicCAS
// on the depth word and setting the bit afterwards took a second atomic per
// winner and a scattered sector per loser.)
__device__ __forceinline__ void td_claim_batch(const BfsParams &p, Acc *acc, uint32_t *vis,
                                               int qout, int new_level, const bool (&ok)[kILP],
                                               const uint32_t (&v)[kILP],
                                               const uint32_t (&src)[kILP], Local &loc)
{
    uint32_t w[kILP];
#pragma unroll
    for (int i = 0; i < kILP; ++i) { w[i] = ok[i] ? __ldca(&vis[v[i] >> 5]) : 0xFFFFFFFFu; }
    bool won[kILP];
#pragma unroll
    for (int i = 0; i < kILP; ++i) {
        const uint32_t bit = 1u << (v[i] & 31);
        won[i] = !(w[i] & bit);  // arcs past the list read as visited
        if (won[i]) { w[i] = atomicOr(&vis[v[i] >> 5], bit); }
    }
    int64_t deg[kILP];
#pragma unroll
    for (int i = 0; i < kILP; ++i) {
        won[i] = won[i] && !((w[i] >> (v[i] & 31)) & 1u);
        deg[i] = 0;
        if (won[i]) {
            p.depth[v[i]] = new_level;
            p.parent[v[i]] = (int64_t)src[i];
            deg[i] = degree_of(p, v[i]);
        }
    }
    warp_append_k<kILP>(p, acc, qout, won, v, deg, loc);
}

// Processes arcs [b, e) of vertex u with all 32 lanes (coalesced reads).
__device__ __forceinline__ void td_edges_warp(const BfsParams &p, Acc *acc, uint32_t *vis,
                                              int qout, int new_level, uint32_t u, int64_t b,
                                              int64_t e, Local &loc)
{
    const int lane = lane_id();
    for (int64_t base = b; base < e; base += 32 * kILP) {
        uint32_t v[kILP], src[kILP];
        bool ok[kILP];
#pragma unroll
        for (int i = 0; i < kILP; ++i) {
            const int64_t k = base + i * 32 + lane;
            ok[i] = k < e;
            v[i] = ok[i] ? __ldg(&p.adj[k]) : 0u;
            src[i] = u;
        }
        td_claim_batch(p, acc, vis, qout, new_level, ok, v, src, loc);
    }
}

struct WarpScratch {
    int32_t incl[32];
    uint32_t u[32];
    int64_t beg[32];
};

// Bounds of the levels CTA 0 runs alone (solo_run).
template <int BLOCK>
constexpr int kSoloCap = BLOCK / 8 * 5;
template <int BLOCK>
constexpr long long kSoloArcs = 5 * BLOCK;
template <int BLOCK>
constexpr long long kSoloBu = 8 * BLOCK;
template <int BLOCK>
constexpr long long kSoloBuArcs = 64 * BLOCK;
template <int BLOCK>
constexpr long long kSoloBuFew = 16 * BLOCK;  // above half of kSoloBu vertices

// Two queues of vertices: id, low word of the list start, and its high 16 bits
// with the degree (65535: that or more), which becomes the position of the list's
// first arc when the level is run (below 2^16, as kSoloArcs is).
template <int BLOCK>
struct SoloQueues {
    uint32_t v[2][kSoloCap<BLOCK>];
    uint32_t lo[2][kSoloCap<BLOCK>];
    uint32_t hi[2][kSoloCap<BLOCK>];
};

template <int BLOCK>
struct SharedState {
    union {
        WarpScratch warp[BLOCK / 32];   // the grid's top-down steps
        SoloQueues<BLOCK> queues;       // CTA 0's narrow levels
    };
    unsigned long long red_found[BLOCK / 32];
    unsigned long long red_deg[BLOCK / 32];
    LevelState st;       // this CTA's copy of the traversal state
    PolicyBlob pol;      // the learned policy's weights, staged once
    int rule_dir;
    int consult;         // the learned policy decides the next step
    // CTA 0's narrow levels
    BfsParams par;       // the launch's parameters, for code that is not inlined
    Acc acc;             // counters (queue entries past the shared queue too)
    unsigned queued;     // entries of the queue being filled
    unsigned warp_sum[BLOCK / 32];
};

template <int BLOCK>
__device__ void td_step(const BfsParams &p, const StepView &sv, const Team &team,
                        SharedState<BLOCK> &sh, Local &loc)
{
    const int lane = lane_id();
    const int warp = threadIdx.x >> 5;
    const long long gw = team.gw, nw = team.nw;
    const int qin = sv.q_cur, qout = sv.q_cur ^ 1;
    uint32_t *vis = p.vis[sv.vis_cur];
    Acc *acc = team.acc;
    const int new_level = sv.level + 1;

    // Phase A: chunks of large-degree frontier vertices.  Warp gw takes a
    // contiguous range of chunk ids, so every warp gets the same number of
    // edges (within one chunk); one binary search finds the range's first
    // vertex, then the walk moves forward.
    const long long nl = sv.f_large;
    const long long nch = sv.f_chunks;
    if (nch > 0) {
        // (x counts parts of chunks where there are too few chunks for the warps)
        const int cut = split_chunks(nch, p.chunk, nw);
        const int64_t part = split_part(p.chunk, cut);
        const long long per = ((nch << cut) + nw - 1) / nw;
        const long long x0 = gw * per, x1 = min(nch << cut, x0 + per);
        const long long c0 = x0 >> cut;
        if (x0 < x1) {
            long long lo = 0, hi = nl - 1;  // last i with qlb[i] <= c0
            while (lo < hi) {
                long long mid = (lo + hi + 1) >> 1;
                if ((long long)__ldcg(&p.qlb[qin][mid]) <= c0) { lo = mid; } else { hi = mid - 1; }
            }
            long long i = lo;
            long long ibase = (long long)__ldcg(&p.qlb[qin][i]);
            long long inext = i + 1 < nl ? (long long)__ldcg(&p.qlb[qin][i + 1]) : nch;
            for (long long x = x0; x < x1; ++x) {
                const long long c = x >> cut;
                while (c >= inext) {
                    ++i;
                    ibase = inext;
                    inext = i + 1 < nl ? (long long)__ldcg(&p.qlb[qin][i + 1]) : nch;
                }
                const uint32_t u = __ldcg(&p.ql[qin][i]);
                const int64_t ub = __ldg(&p.off[u]), ue = __ldg(&p.off[u + 1]);
                const int64_t cb = ub + (c - ibase) * (int64_t)p.chunk;
                const int64_t b = cb + (x & ((1ll << cut) - 1)) * part;
                const int64_t e = min(min(ue, cb + (int64_t)p.chunk), b + part);
                td_edges_warp(p, acc, vis, qout, new_level, u, b, e, loc);
            }
        }
    }

    // Phase B: small-degree frontier vertices, up to 32 per warp; their arcs are
    // laid end to end and dealt to the lanes 32 at a time.
    WarpScratch &ws = sh.warp[warp];
    const int group = split_group(sv.f_small, average(sh.st.f_degsum, sh.st.f_count), nw);
    for (long long g = gw; g << group < sv.f_small; g += nw) {
        const long long idx = (g << group) + lane;
        uint32_t u = 0;
        int64_t beg = 0;
        int32_t deg = 0;
        if (lane >> group == 0 && idx < sv.f_small) {
            u = __ldcg(&p.qs[qin][idx]);
            beg = __ldg(&p.off[u]);
            deg = (int32_t)(__ldg(&p.off[u + 1]) - beg);
        }
        const int32_t incl = warp_incl_scan(deg);
        const int32_t total = __shfl_sync(kFull, incl, 31);
        ws.incl[lane] = incl;
        ws.u[lane] = u;
        ws.beg[lane] = beg;
        __syncwarp();
        for (int32_t base = 0; base < total; base += 32 * kILP) {
            uint32_t v[kILP], src[kILP];
            bool ok[kILP];
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                const int32_t e = base + i * 32 + lane;
                ok[i] = e < total;
                v[i] = 0;
                src[i] = 0;
                if (ok[i]) {
                    int lo = 0, hi = 31;  // first owner with incl > e
                    while (lo < hi) {
                        int mid = (lo + hi) >> 1;
                        if (ws.incl[mid] > e) { hi = mid; } else { lo = mid + 1; }
                    }
                    const int32_t excl = lo ? ws.incl[lo - 1] : 0;
                    src[i] = ws.u[lo];
                    v[i] = __ldg(&p.adj[ws.beg[lo] + (e - excl)]);
                }
            }
            td_claim_batch(p, acc, vis, qout, new_level, ok, v, src, loc);
        }
        __syncwarp();
    }
}

// Bottom-up step (hybrid_bfs.cc:111-143).  A warp works on K consecutive
// bitmap words (32 K vertices) at a time, so K independent load chains are
// in flight per lane.  Unvisited lanes scan their own neighbour lists (the
// first bu_prefix arcs, P arcs per word per round), stopping at the first
// visited neighbour; lists longer than that are finished by the whole warp,
// 32 arcs per ballot (warp-ballot early exit).  Reads only the frozen bitmap
// vis[cur]; writes whole words of vis[cur^1].
template <int BLOCK, int K>
__device__ void bu_step(const BfsParams &p, const StepView &sv, const Team &team, Local &loc)
{
    constexpr int P = K >= 4 ? 2 : 4;
    const int lane = lane_id();
    const long long gw = team.gw, nw = team.nw;
    const uint32_t *vin = p.vis[sv.vis_cur];
    uint32_t *vout = p.vis[sv.vis_cur ^ 1];
    const int qout = sv.q_cur ^ 1;
    Acc *acc = team.acc;
    const int new_level = sv.level + 1;

    // Warp gw owns groups gw, gw + nw, gw + 2 nw, ... of K words.  It loads
    // 32 / K of its groups at once (one word per lane), passes full groups
    // through, and works only on the groups with unvisited vertices: late
    // levels, where most words are full, cost a bitmap sweep.
    constexpr int GPB = 32 / K;
    constexpr unsigned kGroupMask = (1u << K) - 1u;
    for (long long t0 = 0; (gw + t0 * nw) * K < p.words; t0 += GPB) {
        const int j = lane / K;
        const long long wl = (gw + (t0 + j) * nw) * K + lane % K;
        const uint32_t mw = wl < p.words ? __ldcg(&vin[wl]) : kFull;
        const unsigned openm = __ballot_sync(kFull, mw != kFull);
        if (!((openm >> (j * K)) & kGroupMask) && wl < p.words) { vout[wl] = kFull; }
        unsigned groups = 0;
#pragma unroll
        for (int g = 0; g < GPB; ++g) {
            if ((openm >> (g * K)) & kGroupMask) { groups |= 1u << g; }
        }
        while (groups) {
            const int g = __ffs(groups) - 1;
            groups &= groups - 1;
            const long long w0 = (gw + (t0 + g) * nw) * K;
            uint32_t word[K];
#pragma unroll
            for (int k = 0; k < K; ++k) { word[k] = __shfl_sync(kFull, mw, g * K + k); }
            // Per word only the list start, its length and the parent are kept
            // (open / fnd hold the flags, one bit per word), so that K = 4 fits
            // the 64 registers of a full SM.
            const uint32_t v0 = (uint32_t)(w0 * 32 + lane);
            unsigned open = 0, fnd = 0;
            uint32_t par[K], len[K];  // length: 2^32 - 1 stands for that or more
            int64_t beg[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                par[k] = len[k] = 0;
                beg[k] = 0;
                if (!((word[k] >> lane) & 1u)) {
                    open |= 1u << k;
                    beg[k] = __ldg(&p.off[v0 + 32 * k]);
                    len[k] = (uint32_t)min(__ldg(&p.off[v0 + 32 * k + 1]) - beg[k], (int64_t)kFull);
                }
            }
            // per-lane scan of the first bu_prefix arcs, P arcs per word per round
            const uint32_t lim = (uint32_t)(p.bu_prefix + P - 1) / P * P;
            for (uint32_t r = 0; r < lim; r += P) {
                uint32_t x[K][P], hit[K][P];
#pragma unroll
                for (int k = 0; k < K; ++k) {
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        x[k][j] = (open >> k) & 1u && r + j < len[k] ? __ldg(&p.adj[beg[k] + r + j]) : 0u;
                    }
                }
#pragma unroll
                for (int k = 0; k < K; ++k) {
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        hit[k][j] = (open >> k) & 1u && r + j < len[k]
                                        ? (ld_bits(&vin[x[k][j] >> 5]) >> (x[k][j] & 31)) & 1u
                                        : 0u;
                    }
                }
                bool more = false;
#pragma unroll
                for (int k = 0; k < K; ++k) {
#pragma unroll
                    for (int j = 0; j < P; ++j) {
                        if (hit[k][j] && (open >> k) & 1u) {
                            fnd |= 1u << k;
                            open &= ~(1u << k);
                            par[k] = x[k][j];
                        }
                    }
                    more |= (open >> k) & 1u && r + P < len[k];
                }
                if (!__any_sync(kFull, more)) { break; }
            }
            bool found[K];
            uint32_t v[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                v[k] = v0 + 32 * k;
                unsigned pending = __ballot_sync(kFull, (open >> k) & 1u && len[k] > lim);
                while (pending) {
                    const int owner = __ffs(pending) - 1;
                    pending &= pending - 1;
                    const int64_t first = __shfl_sync(kFull, beg[k], owner), b = first + lim;
                    const uint32_t l = __shfl_sync(kFull, len[k], owner);
                    // (the list's end is not read again: that read stood before every
                    // scan, 10 to 20 % of a level of few words)
                    const int64_t e = l != kFull
                                          ? first + l
                                          : __ldg(&p.off[__shfl_sync(kFull, v[k], owner) + 1]);
                    for (int64_t base = b; base < e; base += 32) {
                        const int64_t kk = base + lane;
                        bool hit = false;
                        uint32_t xx = 0;
                        if (kk < e) {
                            xx = __ldg(&p.adj[kk]);
                            hit = (ld_bits(&vin[xx >> 5]) >> (xx & 31)) & 1u;
                        }
                        const unsigned hm = __ballot_sync(kFull, hit);
                        if (hm) {
                            const uint32_t hx = __shfl_sync(kFull, xx, __ffs(hm) - 1);
                            if (lane == owner) {
                                fnd |= 1u << k;
                                par[k] = hx;
                            }
                            break;
                        }
                    }
                }
                found[k] = (fnd >> k) & 1u;
                const unsigned fm = __ballot_sync(kFull, found[k]);
                if (lane == 0 && w0 + k < p.words) { vout[w0 + k] = word[k] | fm; }
                if (found[k]) {
                    p.depth[v[k]] = new_level;
                    p.parent[v[k]] = (int64_t)par[k];
                }
            }
            int64_t deg[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                deg[k] = len[k] == kFull ? degree_of(p, v[k]) : (int64_t)len[k];
            }
            warp_append_k<K>(p, acc, qout, found, v, deg, loc);
        }
    }
}

// Bottom-up step, lane-owned words (hybrid_bfs.cc:111-143).  Each lane owns
// one bitmap word (32 vertices) and walks its unvisited vertices on its own:
// a lane that finds a parent moves straight to its next vertex instead of
// waiting for the warp's slowest list.  P arcs are probed per iteration.
// Lists longer than kLongList are left to the whole warp (ballot scan) after
// the per-lane walk.  Reads only the frozen bitmap vis[cur]; writes whole
// words of vis[cur^1].
constexpr int64_t kLongList = 256;

template <int BLOCK>
__device__ void bu_step_lanes(const BfsParams &p, const StepView &sv, const Team &team, Local &loc)
{
    constexpr int P = 4;
    const int lane = lane_id();
    const long long gw = team.gw, nw = team.nw;
    const uint32_t *vin = p.vis[sv.vis_cur];
    uint32_t *vout = p.vis[sv.vis_cur ^ 1];
    const int qout = sv.q_cur ^ 1;
    Acc *acc = team.acc;
    const int new_level = sv.level + 1;

    for (long long base = gw * 32; base < p.words; base += nw * 32) {
        const long long w = base + lane;
        const bool mine = w < p.words;
        const uint32_t word = mine ? __ldcg(&vin[w]) : kFull;
        uint32_t todo = ~word;     // unvisited vertices of this lane's word
        uint32_t found = 0;        // ... that found a parent
        uint32_t longs = 0;        // ... with lists left to the warp
        int64_t e = 0, end = 0;
        int cur = -1;
        unsigned long long degsum = 0;
        while (__any_sync(kFull, todo != 0 || cur >= 0)) {
            if (cur < 0 && todo) {
                cur = __ffs(todo) - 1;
                todo &= todo - 1;
                const uint32_t v = (uint32_t)(w * 32 + cur);
                e = __ldg(&p.off[v]);
                end = __ldg(&p.off[v + 1]);
                if (end - e > kLongList) {
                    longs |= 1u << cur;
                    cur = -1;
                }
            }
            if (cur >= 0) {
                uint32_t x[P], bits[P];
#pragma unroll
                for (int j = 0; j < P; ++j) { x[j] = (e + j < end) ? __ldg(&p.adj[e + j]) : 0u; }
#pragma unroll
                for (int j = 0; j < P; ++j) { bits[j] = (e + j < end) ? ld_bits(&vin[x[j] >> 5]) : 0u; }
                int hit = -1;
#pragma unroll
                for (int j = P - 1; j >= 0; --j) {
                    if ((e + j < end) && ((bits[j] >> (x[j] & 31)) & 1u)) { hit = j; }
                }
                if (hit >= 0) {
                    const uint32_t v = (uint32_t)(w * 32 + cur);
                    found |= 1u << cur;
                    p.depth[v] = new_level;
                    p.parent[v] = (int64_t)x[hit];
                    degsum += (unsigned long long)(end - __ldg(&p.off[v]));
                    cur = -1;
                } else {
                    e += P;
                    if (e >= end) { cur = -1; }
                }
            }
        }
        // long lists: the whole warp, one vertex at a time, 32 arcs a ballot
        unsigned owners = __ballot_sync(kFull, longs != 0);
        while (owners) {
            const int owner = __ffs(owners) - 1;
            uint32_t ol = __shfl_sync(kFull, longs, owner);
            const long long ow = __shfl_sync(kFull, w, owner);
            while (ol) {
                const int bit = __ffs(ol) - 1;
                ol &= ol - 1;
                const uint32_t v = (uint32_t)(ow * 32 + bit);
                const int64_t b = __ldg(&p.off[v]), en = __ldg(&p.off[v + 1]);
                for (int64_t kb = b; kb < en; kb += 32) {
                    const int64_t k = kb + lane;
                    bool hit = false;
                    uint32_t xx = 0;
                    if (k < en) {
                        xx = __ldg(&p.adj[k]);
                        hit = (ld_bits(&vin[xx >> 5]) >> (xx & 31)) & 1u;
                    }
                    const unsigned hm = __ballot_sync(kFull, hit);
                    if (hm) {
                        const uint32_t hx = __shfl_sync(kFull, xx, __ffs(hm) - 1);
                        if (lane == owner) {
                            found |= 1u << bit;
                            p.depth[v] = new_level;
                            p.parent[v] = (int64_t)hx;
                            degsum += (unsigned long long)(en - b);
                        }
                        break;
                    }
                }
            }
            owners &= owners - 1;
        }
        if (mine) { vout[w] = word | found; }
        // append this lane's discoveries: one atomic per warp for the small
        // ones, one per large vertex (rare)
        uint32_t small = 0, large = 0;
        for (uint32_t f = found; f; f &= f - 1) {
            const int bit = __ffs(f) - 1;
            const uint32_t v = (uint32_t)(w * 32 + bit);
            if (__ldg(&p.off[v + 1]) - __ldg(&p.off[v]) >= (int64_t)p.large_deg) {
                large |= 1u << bit;
            } else {
                small |= 1u << bit;
            }
        }
        const unsigned cnt = __popc(small);
        const unsigned incl = warp_incl_scan(cnt);
        const unsigned total = __shfl_sync(kFull, incl, 31);
        if (total) {
            unsigned long long start = 0;
            if (lane == 0) { start = atomicAdd(&acc->small_cnt, (unsigned long long)total); }
            start = __shfl_sync(kFull, start, 0) + (incl - cnt);
            for (uint32_t f = small; f; f &= f - 1) {
                p.qs[qout][start++] = (uint32_t)(w * 32 + (__ffs(f) - 1));
            }
        }
        if (__any_sync(kFull, large != 0)) {
            unsigned long long chunks = 0;
            for (uint32_t f = large; f; f &= f - 1) {
                const uint32_t v = (uint32_t)(w * 32 + (__ffs(f) - 1));
                const int64_t d = __ldg(&p.off[v + 1]) - __ldg(&p.off[v]);
                chunks += (unsigned long long)((d + p.chunk - 1) / p.chunk);
            }
            unsigned long long pos, cbase;
            warp_reserve_large(acc, __popc(large), chunks, pos, cbase);
            for (uint32_t f = large; f; f &= f - 1) {
                const uint32_t v = (uint32_t)(w * 32 + (__ffs(f) - 1));
                const int64_t d = __ldg(&p.off[v + 1]) - __ldg(&p.off[v]);
                p.ql[qout][pos] = v;
                p.qlb[qout][pos] = cbase;
                pos += 1;
                cbase += (unsigned long long)((d + p.chunk - 1) / p.chunk);
            }
        }
        loc.found += __popc(found);
        loc.degsum += degsum;
    }
}

// Beamer's rule (hybrid_bfs.cc:152-191) for the step about to run, given the
// frontier in the state.  Updates the Beamer state like the reference loop
// does when it commits to that direction.
__device__ int beamer_choose(LevelState &c, const BfsParams &p, bool commit)
{
    if (c.in_bu) { return kDirBU; }
    // scout > etc / alpha, without the division where the product fits
    const bool pull = c.etc >= 0 && ((c.scout | p.alpha) >> 31) == 0 ? c.scout * p.alpha > c.etc
                                                                     : c.scout > c.etc / p.alpha;
    if (pull) {
        if (commit) {
            c.in_bu = 1;
            c.awake = c.f_count;  // queue_.combined_size()
        }
        return kDirBU;
    }
    if (commit) { c.etc -= c.scout; }
    return kDirTD;
}

// After a step of direction `dir` found `found` vertices of degree sum
// `degsum`: the reference's bookkeeping (scout after top-down, the awake
// test of the bottom-up do-while, scout = 1 on leaving it).
__device__ void beamer_after_step(LevelState &c, const BfsParams &p, int dir, long long found,
                                  long long degsum)
{
    if (dir == kDirTD) {
        c.scout = degsum;
    } else if (c.in_bu) {
        c.old_awake = c.awake;
        c.awake = found;
        if (!(c.awake >= c.old_awake || c.awake > p.n / p.beta)) {
            c.in_bu = 0;
            c.scout = 1;
        }
    }
}

// Whether the learned policy is consulted for the step after state c: it is
// installed, the BFS goes on, and the frontier's degree sum over the
// unexplored one lies in the band the policy was trained to decide in
// (outside it the rule decides and the network is not run).
__device__ __forceinline__ bool policy_applies(const LevelState &c, const BfsParams &p)
{
    return p.alg == BD_ALG_LEARNED && p.policy != nullptr && c.f_count != 0 &&
           policy_in_band(p.policy, c.f_degsum, 2 * p.m - c.visited_degsum);
}

// The rule's direction for the next step (committed into the Beamer state
// unless the learned policy will decide).  One thread.
__device__ int rule_direction(LevelState &c, const BfsParams &p)
{
    if (c.f_count == 0) { return kDirDone; }
    if (p.alg == BD_ALG_TOP_DOWN) { return kDirTD; }
    if (p.alg == BD_ALG_BOTTOM_UP) { return kDirBU; }
    return beamer_choose(c, p, !policy_applies(c, p));
}

// The learned policy's pick over the rule's (NaN gap: a feature outside the
// trusted range, the rule decides); keeps the rule's state consistent with
// the step actually taken.  One thread.
__device__ int apply_policy(LevelState &c, const PolicyBlob *w, int rule, float gap)
{
    int d = rule;
    if (isfinite(gap) && fabsf(gap) >= w->margin) { d = gap > 0.f ? kDirBU : kDirTD; }
    if (d != rule) { c.policy_overrides += 1; }
    if (d == kDirTD) {
        c.in_bu = 0;
        c.etc -= c.scout;
    } else if (!c.in_bu) {
        c.in_bu = 1;
        c.awake = c.f_count;
    }
    return d;
}

// Picks c.dir for the next step: thread 0 applies the rule (in the branch that
// advanced the state), warp 0 runs the policy network where it applies.
__device__ __forceinline__ void decide_rule(LevelState &c, const BfsParams &p, int &rule_dir,
                                            int &consult)
{
    consult = policy_applies(c, p);
    rule_dir = rule_direction(c, p);
    if (!consult) { c.dir = rule_dir; }
}

// After decide_rule and a block barrier; every thread of the block.  Ends with
// the decision visible to the block.
template <typename Shared>
__device__ __forceinline__ void decide_policy(const BfsParams &p, Shared &sh)
{
    if (!sh.consult) { return; }
    if (threadIdx.x < 32) {
        LevelState &c = sh.st;
        const float gap = policy_gap_warp(&sh.pol, c.f_count, c.f_degsum, 2 * p.m - c.visited_degsum,
                                          c.level, p.n, p.m, c.prev_dir, c.prev_ns);
        if (threadIdx.x == 0) { c.dir = apply_policy(c, &sh.pol, sh.rule_dir, gap); }
    }
    __syncthreads();
}

// Advances the state over the step that just ended, from that step's
// counters a and its end time.  One thread per CTA; every CTA computes the
// same result.
__device__ void advance(LevelState &c, const BfsParams &p, const Acc &a, long long t_end)
{
    const long long found = (long long)a.found;
    const long long degsum = (long long)a.degsum;
    const unsigned long long lp = a.large_packed;
    const long long ns = t_end - c.t_last;
    const int dir = c.dir;
    c.visited_degsum += degsum;
    c.reached += found;
    // once fewer than half of the live vertices are unvisited, bottom-up
    // work per bitmap word is sparse: switch to the lane-owned layout
    c.bu_sparse = 2 * (p.n_live - c.reached) < p.n_live;
    c.f_count = found;
    c.f_degsum = degsum;
    c.f_small = (long long)a.small_cnt;
    c.f_large = (long long)(lp >> kLargeShift);
    c.f_chunks = (long long)(lp & kChunkMask);
    c.prev_dir = dir;
    c.prev_ns = ns;
    c.t_last = t_end;
    if (dir == kDirTD) { c.td_steps += 1; } else { c.bu_steps += 1; }
    c.level += 1;
    c.q_cur ^= 1;
    if (dir == kDirBU) { c.vis_cur ^= 1; }
    beamer_after_step(c, p, dir, found, degsum);
    c.step += 1;
}

// Sums the block's step counters into acc->found / degsum (any memory) from
// thread 0.  Ends after a block barrier; the sums are thread 0's.
template <int BLOCK>
__device__ __forceinline__ void block_totals(SharedState<BLOCK> &sh, Local &loc,
                                             unsigned long long &tf, unsigned long long &td)
{
    const int lane = lane_id();
    const int warp = threadIdx.x >> 5;
    const unsigned long long f = warp_sum(loc.found);
    const unsigned long long d = warp_sum(loc.degsum);
    if (lane == 0) {
        sh.red_found[warp] = f;
        sh.red_deg[warp] = d;
    }
    loc.found = 0;
    loc.degsum = 0;
    __syncthreads();
    tf = td = 0;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < BLOCK / 32; ++i) {
            tf += sh.red_found[i];
            td += sh.red_deg[i];
        }
    }
}

// The step record of the step that just ended (before advance).
__device__ __forceinline__ void record_step(const BfsParams &p, const LevelState &st,
                                            long long found, long long t_end)
{
    if (st.step >= p.rec_cap) { return; }
    bd_step r;
    r.dir = st.dir;
    r.level = st.level;
    r.frontier = st.f_count;
    r.frontier_edges = st.f_degsum;
    r.unexplored_edges = 2 * p.m - st.visited_degsum;
    r.found = found;
    r.ns = t_end - st.t_last;
    p.rec[st.step] = r;
}

// Grid barrier number b: arrival (one release-add) and polling until every CTA
// has arrived, at most p.spin_limit polls; running out sets
// ctrl->error = BD_ERR_TIMEOUT.  Thread 0 of each CTA.  False after an error.
// solo: CTA 0 arrives only after levels of its own, or a long list of sources;
// the bound then holds for each of these (p.spin_limit polls in which ctrl->beat
// does not change), as it does for a level of the grid.
__device__ __forceinline__ bool arrive_wait(const BfsParams &p, long long b, bool solo)
{
    Ctrl *c = p.ctrl;
    red_release_add64(&c->bar, 1ull);
    const unsigned long long target = (unsigned long long)(b + 1) * p.expected_ctas;
    long long it = 0;
    // During CTA 0's narrow levels the others poll relaxed: an acquire load
    // empties the SM's L1, and CTA 0 shares its SM (its reads, spilled registers
    // among them, then went to L2: 4.1 us a level instead of 2.6).  At the end of
    // a grid step the waits are short, and a poll that is itself the acquire
    // saves a round trip (0.4 us a level).
    unsigned long long beat = solo ? ld_relaxed64(&c->beat) : 0ull;
    while (solo && ld_relaxed64(&c->bar) < target) {
        if (++it > p.spin_limit) {
            const unsigned long long now = ld_relaxed64(&c->beat);
            if (now == beat) {
                atomicExch(&c->error, (int)BD_ERR_TIMEOUT);
                return false;
            }
            beat = now;
            it = 0;
        }
        __nanosleep(64);
    }
    while (ld_acquire64(&c->bar) < target) {
        if (++it > p.spin_limit) {
            atomicExch(&c->error, (int)BD_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(32);
    }
    return __ldcg(&c->error) == 0;
}

// CTA 0's part of a barrier's counter ring: the next barrier's slot.
__device__ __forceinline__ void clear_next_acc(Ctrl *c, long long b)
{
    Acc *z = &c->acc[(b + 1) % 3];
    z->found = z->degsum = z->small_cnt = z->large_packed = z->t_end = 0;
}

// The end of a step: block reduction of the counters, the grid barrier, then
// every CTA advances its copy of the state from the step's counters and decides
// the next direction.  A timeout ends this CTA's loop.
template <int BLOCK>
__device__ void end_step(const BfsParams &p, const StepView &sv, SharedState<BLOCK> &sh,
                         Local &loc)
{
    Ctrl *c = p.ctrl;
    unsigned long long tf, td;
    block_totals<BLOCK>(sh, loc, tf, td);
    if (threadIdx.x == 0) {
        Acc *acc = &c->acc[sv.barrier % 3];
        if (tf) { atomicAdd(&acc->found, tf); }
        if (td) { atomicAdd(&acc->degsum, td); }
        if (blockIdx.x == 0) { clear_next_acc(c, sv.barrier); }
        atomicMax(&acc->t_end, (unsigned long long)globaltimer());
        LevelState &st = sh.st;
        if (arrive_wait(p, sv.barrier, false)) {
            // 16 bytes a request: all CTAs read this one line at once
            const ulonglong2 *from = reinterpret_cast<const ulonglong2 *>(acc);
            const ulonglong2 w0 = __ldcg(&from[0]), w1 = __ldcg(&from[1]);
            const long long t_end = (long long)__ldcg(&acc->t_end);
            Acc a;
            a.found = w0.x;
            a.degsum = w0.y;
            a.small_cnt = w1.x;
            a.large_packed = w1.y;
            if (blockIdx.x == 0) { record_step(p, st, (long long)a.found, t_end); }
            advance(st, p, a, t_end);
        } else {
            st.f_count = 0;  // leave the loop
        }
        st.barrier += 1;
        decide_rule(st, p, sh.rule_dir, sh.consult);
    }
    __syncthreads();
    decide_policy(p, sh);
}

// K bitmap words per warp step: 1, 2, 4 (warp-shared words) or 32 (one word
// per lane).
template <int BLOCK, int K>
__device__ __forceinline__ void bu_layout(const BfsParams &p, const StepView &sv, const Team &team,
                                          Local &loc)
{
    if constexpr (K == 32) {
        bu_step_lanes<BLOCK>(p, sv, team, loc);
    } else {
        bu_step<BLOCK, K>(p, sv, team, loc);
    }
}

// ---------------------------------------------------------------------------
// Narrow levels: CTA 0 alone
// ---------------------------------------------------------------------------
// A level of a few thousand arcs does not need the grid, and pays for it: the
// grid barrier with its counters, and the round trips of a queue in global
// memory.  CTA 0 therefore runs such levels by itself while the other CTAs wait
// at one grid barrier.  Its queue lies in shared memory with each vertex's list
// start, so a level is a chain of three round trips (arc; visited word; claim
// with offsets) and a few block barriers.
//
// Levels of a 1021 x 1031 grid by frontier size, 512 threads, medians in us of
// levels all on the whole grid and of levels all in one CTA: up to 16 vertices 4.9
// and 2.8, 32 to 64 5.1 and 3.1, 100 to 160 5.2 and 4.2, 180 to 240 5.7 and 4.9, 260
// to 319 5.8 and 5.6, 321 to 380 5.8 and 6.2, 400 to 480 5.9 and 6.8, 560 to 640 5.9
// and 10.1 (one SM's requests then bound it).  So the line lies at kSoloCap
// vertices, which is also what keeps the queues within the memory of the grid's own
// scratch (a CTA that holds more shared memory leaves less L1 for the bottom-up
// steps), and at kSoloArcs arcs.
//
// Bottom-up levels run here in graphs of at most kSoloBu vertices while the lists of
// the unvisited ones hold at most kSoloBuArcs arcs, or kSoloBuFew: the grid is better
// at many arcs the more words there are to share, but in a hub numbering 32 vertices
// of the highest degrees make one word and one warp's work.  Six searches bottom-up throughout in
// ms, all steps on the grid, up to kSoloBuArcs and up to kSoloBuFew in CTA 0:
// 1024 vertices, 16 edges each 0.67, 0.35, 0.69; 4096, 4 each 0.65, 0.77, 0.63 in
// file order and 2.10, 0.82, 2.06 in hub order; grid 60 x 60 3.72, 3.34, 2.97.
// Levels before CTA 0 meets the others once, so that none polls for long.
constexpr int kSoloLevels = 128;

extern __shared__ __align__(16) unsigned char bfs_shared[];  // a SharedState

template <int BLOCK>
__device__ __forceinline__ bool solo_applies(const LevelState &st, const BfsParams &p)
{
    if (st.dir == kDirTD) {
        return st.f_count <= kSoloCap<BLOCK> && st.f_degsum <= kSoloArcs<BLOCK>;
    }
    const long long arcs = 2 * p.n <= kSoloBu<BLOCK> || p.perm ? kSoloBuArcs<BLOCK>
                                                               : kSoloBuFew<BLOCK>;
    return st.dir == kDirBU && p.n <= kSoloBu<BLOCK> && 2 * p.m - st.visited_degsum <= arcs;
}

__device__ __forceinline__ uint32_t solo_hi(int64_t beg, int64_t deg)
{
    return ((uint32_t)((uint64_t)beg >> 32) << 16) | (uint32_t)min(deg, (int64_t)0xFFFF);
}

// Warp-collective: appends up to K vertices per lane to shared queue q; past its
// end they go to the global queues (qout).
template <int BLOCK, int K>
__device__ __forceinline__ void solo_append(const BfsParams &p, SharedState<BLOCK> &sh,
                                            SoloQueues<BLOCK> &sq, int q, int qout,
                                            const bool (&has)[K], const uint32_t (&v)[K],
                                            const int64_t (&beg)[K], const int64_t (&deg)[K],
                                            Local &loc)
{
    unsigned m[K], total = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        m[k] = __ballot_sync(kFull, has[k]);
        total += __popc(m[k]);
    }
    if (!total) { return; }
    unsigned base = 0;
    if (lane_id() == 0) { base = atomicAdd(&sh.queued, total); }
    base = __shfl_sync(kFull, base, 0);
    bool over[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const unsigned pos = base + __popc(m[k] & lanemask_lt());
        base += __popc(m[k]);
        over[k] = has[k] && pos >= (unsigned)kSoloCap<BLOCK>;
        if (has[k]) {
            loc.found += 1;
            loc.degsum += (unsigned long long)deg[k];
            if (!over[k]) {
                sq.v[q][pos] = v[k];
                sq.lo[q][pos] = (uint32_t)beg[k];
                sq.hi[q][pos] = solo_hi(beg[k], deg[k]);
            }
        }
    }
    if (base > (unsigned)kSoloCap<BLOCK>) {
        Local none{0, 0};
        warp_append_k<K>(p, &sh.acc, qout, over, v, deg, none);
    }
}

// The frontier of the state, from the global queues into shared queue q.
template <int BLOCK>
__device__ void solo_load(const BfsParams &p, SharedState<BLOCK> &sh, SoloQueues<BLOCK> &sq, int q)
{
    const LevelState &st = sh.st;
    const int small = (int)st.f_small, count = (int)st.f_count;
    for (int i = threadIdx.x; i < count; i += BLOCK) {
        const uint32_t v = i < small ? __ldcg(&p.qs[st.q_cur][i]) : __ldcg(&p.ql[st.q_cur][i - small]);
        const int64_t b = __ldg(&p.off[v]);
        sq.v[q][i] = v;
        sq.lo[q][i] = (uint32_t)b;
        sq.hi[q][i] = solo_hi(b, __ldg(&p.off[v + 1]) - b);
    }
}

// Shared queue q into the global queues of the state's frontier, beside what
// has gone there already.
template <int BLOCK>
__device__ void solo_flush(const BfsParams &p, SharedState<BLOCK> &sh, SoloQueues<BLOCK> &sq, int q)
{
    const int count = (int)min(sh.queued, (unsigned)kSoloCap<BLOCK>);
    Local none{0, 0};
    for (int i0 = 0; i0 < count; i0 += BLOCK) {
        const int i = i0 + threadIdx.x;
        const bool has[1] = {i < count};
        const uint32_t v[1] = {has[0] ? sq.v[q][i] : 0u};
        int64_t deg[1] = {has[0] ? (int64_t)(sq.hi[q][i] & 0xFFFFu) : 0};
        if (deg[0] == 0xFFFF) { deg[0] = degree_of(p, v[0]); }
        warp_append_k<1>(p, &sh.acc, sh.st.q_cur, has, v, deg, none);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        LevelState &st = sh.st;
        st.f_small = (long long)sh.acc.small_cnt;
        st.f_large = (long long)(sh.acc.large_packed >> kLargeShift);
        st.f_chunks = (long long)(sh.acc.large_packed & kChunkMask);
    }
}

// Degrees in the low halves of hi[q] become positions of the lists' first arcs.
template <int BLOCK>
__device__ void solo_scan(SharedState<BLOCK> &sh, SoloQueues<BLOCK> &sq, int q, int count)
{
    constexpr int E = (kSoloCap<BLOCK> + BLOCK - 1) / BLOCK;  // consecutive entries per thread
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t h[E];
    unsigned sum = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const int i = (int)threadIdx.x * E + k;
        h[k] = i < count ? sq.hi[q][i] : 0u;
        sum += h[k] & 0xFFFFu;
    }
    const unsigned incl = warp_incl_scan(sum);
    if (lane == 31) { sh.warp_sum[warp] = incl; }
    __syncthreads();
    const unsigned w = lane < BLOCK / 32 ? sh.warp_sum[lane] : 0u;
    const unsigned wi = warp_incl_scan(w);
    unsigned at = incl - sum + (warp ? __shfl_sync(kFull, wi, warp - 1) : 0u);
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const int i = (int)threadIdx.x * E + k;
        if (i < count) { sq.hi[q][i] = (h[k] & 0xFFFF0000u) | at; }
        at += h[k] & 0xFFFFu;
    }
    __syncthreads();
}

// A top-down level from shared queue q into q ^ 1.  The arcs of all lists, laid
// end to end, are dealt to the threads, ILP at a time with each stage's reads
// issued together; an unvisited neighbour is claimed by the atomicOr on its
// visited word (its old value names the one winner), and its offsets are read
// with the claim rather than after it.
template <int BLOCK, int ILP>
__device__ __forceinline__ void solo_td(const BfsParams &p, SharedState<BLOCK> &sh, SoloQueues<BLOCK> &sq, int q,
                        Local &loc)
{
    const LevelState &st = sh.st;
    const int count = (int)st.f_count, arcs = (int)st.f_degsum, new_level = st.level + 1;
    const int qout = st.q_cur ^ 1;
    uint32_t *vis = p.vis[st.vis_cur];
    int top = 1;  // first step of the searches: the largest power of two below count
    while (top * 2 < count) { top *= 2; }
    // whole warps: the appends are warp-collective
    for (int e0 = (int)threadIdx.x & ~31; e0 < arcs; e0 += BLOCK * ILP) {
        bool won[ILP];
        int e[ILP], at[ILP];
        uint32_t v[ILP], src[ILP];
        int64_t beg[ILP], deg[ILP];
#pragma unroll
        for (int i = 0; i < ILP; ++i) {
            e[i] = e0 + i * BLOCK + lane_id();
            won[i] = e[i] < arcs;
            at[i] = 0;  // last list that starts at or before arc e
        }
        for (int d = top; d > 0; d >>= 1) {
#pragma unroll
            for (int i = 0; i < ILP; ++i) {
                const int t = at[i] + d;
                if (t < count && (int)(sq.hi[q][t] & 0xFFFFu) <= e[i]) { at[i] = t; }
            }
        }
#pragma unroll
        for (int i = 0; i < ILP; ++i) {
            const uint32_t h = sq.hi[q][at[i]];
            const int64_t b = ((int64_t)(h >> 16) << 32) | sq.lo[q][at[i]];
            src[i] = sq.v[q][at[i]];
            v[i] = won[i] ? __ldg(&p.adj[b + (e[i] - (int)(h & 0xFFFFu))]) : 0u;
        }
        uint32_t old[ILP];
#pragma unroll
        for (int i = 0; i < ILP; ++i) { old[i] = won[i] ? __ldcg(&vis[v[i] >> 5]) : 0xFFFFFFFFu; }
#pragma unroll
        for (int i = 0; i < ILP; ++i) {
            won[i] = !((old[i] >> (v[i] & 31)) & 1u);
            beg[i] = deg[i] = 0;
            if (won[i]) {
                old[i] = atomicOr(&vis[v[i] >> 5], 1u << (v[i] & 31));
                beg[i] = __ldg(&p.off[v[i]]);
                deg[i] = __ldg(&p.off[v[i] + 1]) - beg[i];
            }
        }
#pragma unroll
        for (int i = 0; i < ILP; ++i) {
            won[i] = won[i] && !((old[i] >> (v[i] & 31)) & 1u);
            if (won[i]) {
                p.depth[v[i]] = new_level;
                p.parent[v[i]] = (int64_t)src[i];
            }
        }
        solo_append<BLOCK, ILP>(p, sh, sq, q ^ 1, qout, won, v, beg, deg, loc);
    }
}

// The source frontier (hybrid_bfs.cc:158-163 for one source; any number of
// sources start as one frontier) into shared queue 0, and the first decision.
template <int BLOCK>
__device__ void solo_init(const BfsParams &p, SharedState<BLOCK> &sh, SoloQueues<BLOCK> &sq,
                          Local &loc)
{
    for (int64_t i0 = (int64_t)(threadIdx.x & ~31u); i0 < p.source_count; i0 += BLOCK) {
        if (threadIdx.x == 0 && i0) { st_relaxed64(&p.ctrl->beat, globaltimer()); }
        const int64_t i = i0 + lane_id();
        bool has[1] = {i < p.source_count};
        uint32_t v[1] = {0u};
        int64_t beg[1] = {0}, deg[1] = {0};
        if (has[0]) {
            const int64_t s = p.sources ? __ldg(&p.sources[i]) : p.source;
            v[0] = p.perm ? __ldg(&p.perm[s]) : (uint32_t)s;
            beg[0] = __ldg(&p.off[v[0]]);
            deg[0] = __ldg(&p.off[v[0] + 1]) - beg[0];
            has[0] = atomicCAS(&p.depth[v[0]], -1, 0) == -1;  // else a repeated source
        }
        if (has[0]) {
            p.parent[v[0]] = (int64_t)v[0];
            atomicOr(&p.vis[0][v[0] >> 5], 1u << (v[0] & 31));
        }
        solo_append<BLOCK, 1>(p, sh, sq, 0, 0, has, v, beg, deg, loc);
    }
    unsigned long long tf, td;
    block_totals<BLOCK>(sh, loc, tf, td);
    if (threadIdx.x == 0) {
        LevelState &st = sh.st;
        st.f_count = (long long)tf;
        st.f_degsum = (long long)td;
        st.visited_degsum = (long long)td;
        st.reached = (long long)tf;
        st.etc = 2 * p.m;             // edges_to_check = num_edges * 2
        st.scout = (long long)td;     // scout_count = out_degree(source)
        st.prev_dir = kDirTD;
        st.t_last = globaltimer();
        decide_rule(st, p, sh.rule_dir, sh.consult);
    }
    __syncthreads();
    decide_policy(p, sh);
}

// CTA 0: the source setup (init), then levels as long as they are narrow.  Not
// inlined: beside it the grid's steps would spill registers (12 % slower
// bottom-up and top-down levels at scales 19 and 22).
template <int BLOCK>
__device__ __noinline__ void solo_run(bool init)
{
    SharedState<BLOCK> &sh = *reinterpret_cast<SharedState<BLOCK> *>(bfs_shared);
    const BfsParams &p = sh.par;
    SoloQueues<BLOCK> &sq = sh.queues;
    Local loc{0, 0};
    int q = 0;
    bool shared_queue = init;  // the frontier is in queue q (else in the global queues)
    if (threadIdx.x == 0) {
        sh.queued = 0;
        sh.acc.small_cnt = sh.acc.large_packed = 0;
    }
    __syncthreads();
    if (init) { solo_init<BLOCK>(p, sh, sq, loc); }
    for (int l = 0; l < kSoloLevels && solo_applies<BLOCK>(sh.st, p); ++l) {
        if (sh.st.dir == kDirTD) {
            if (!shared_queue) {
                solo_load<BLOCK>(p, sh, sq, q);
                __syncthreads();
            }
            solo_scan<BLOCK>(sh, sq, q, (int)sh.st.f_count);
            if (threadIdx.x == 0) { sh.queued = 0; }
            __syncthreads();
            if (sh.st.f_degsum <= BLOCK) {  // one arc a thread: four slots would issue for nothing
                solo_td<BLOCK, 1>(p, sh, sq, q, loc);
            } else {
                solo_td<BLOCK, kILP>(p, sh, sq, q, loc);
            }
            q ^= 1;
            shared_queue = true;
        } else {
            if (threadIdx.x == 0) {
                sh.queued = 0;
                sh.acc.small_cnt = sh.acc.large_packed = 0;
            }
            __syncthreads();
            const StepView sv = view_of(sh.st);
            const Team team{(long long)(threadIdx.x >> 5), BLOCK / 32, &sh.acc};
            bu_step<BLOCK, 1>(p, sv, team, loc);
            shared_queue = false;
        }
        unsigned long long tf, td;
        block_totals<BLOCK>(sh, loc, tf, td);
        if (threadIdx.x == 0) {
            LevelState &st = sh.st;
            const long long t_end = globaltimer();
            Acc a;
            a.found = tf;
            a.degsum = td;
            a.small_cnt = sh.acc.small_cnt;
            a.large_packed = sh.acc.large_packed;
            st_relaxed64(&p.ctrl->beat, t_end);
            record_step(p, st, (long long)tf, t_end);
            advance(st, p, a, t_end);
            decide_rule(st, p, sh.rule_dir, sh.consult);
            // what lies in the global queues counts for this frontier only (the
            // policy may still change the direction, not the size: past the
            // shared queue a top-down level is the grid's either way)
            if (!shared_queue || st.f_count <= kSoloCap<BLOCK>) {
                sh.acc.small_cnt = sh.acc.large_packed = 0;
            }
        }
        __syncthreads();
        decide_policy(p, sh);
    }
    if (shared_queue && sh.st.dir != kDirDone) { solo_flush<BLOCK>(p, sh, sq, q); }
}

// KD: bottom-up layout while most live vertices are unvisited; KS: after.
template <int BLOCK, int MINB, int KD, int KS>
__global__ void __launch_bounds__(BLOCK, MINB) bfs_persistent_kernel(
    const __grid_constant__ BfsParams p)
{
    SharedState<BLOCK> &sh = *reinterpret_cast<SharedState<BLOCK> *>(bfs_shared);
    Ctrl *c = p.ctrl;
    if (p.policy) {
        const float *src = reinterpret_cast<const float *>(p.policy);
        float *dst = reinterpret_cast<float *>(&sh.pol);
        for (int i = threadIdx.x; i < (int)(sizeof(PolicyBlob) / sizeof(float)); i += BLOCK) {
            dst[i] = src[i];
        }
    }
    if (threadIdx.x == 0) {
        memset(&sh.st, 0, sizeof(LevelState));
        sh.par = p;
        sh.st.barrier = c->barrier;
        // an earlier launch of the call timed out: its barrier count is void
        sh.consult = __ldcg(&c->error);
    }
    __syncthreads();
    if (sh.consult) { return; }
    // consecutive ranks on different CTAs: a narrow level's few work items then
    // spread over the SMs instead of filling some
    const Team grid{(long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x,
                    (long long)gridDim.x * (BLOCK / 32), nullptr};
    bool init = true;
    Local loc{0, 0};
    do {
        if (init || solo_applies<BLOCK>(sh.st, p)) {
            // CTA 0 alone; the others take the state it publishes
            if (blockIdx.x == 0) { solo_run<BLOCK>(init); }
            init = false;
            __syncthreads();
            if (threadIdx.x == 0) {
                const long long b = sh.st.barrier;
                if (blockIdx.x == 0) {
                    c->pub[b & 1] = sh.st;
                    clear_next_acc(c, b);
                }
                if (arrive_wait(p, b, blockIdx.x != 0)) {
                    if (blockIdx.x != 0) {
                        const long long *from = reinterpret_cast<const long long *>(&c->pub[b & 1]);
                        long long *to = reinterpret_cast<long long *>(&sh.st);
#pragma unroll
                        for (int i = 0; i < (int)(sizeof(LevelState) / 8); ++i) {
                            to[i] = __ldcg(&from[i]);
                        }
                    }
                } else {
                    sh.st.dir = kDirDone;
                }
                sh.st.barrier = b + 1;
            }
            __syncthreads();
            continue;
        }
        const StepView sv = view_of(sh.st);
        Team team = grid;
        team.acc = &c->acc[sv.barrier % 3];
        if (sv.dir == kDirTD) {
            td_step<BLOCK>(p, sv, team, sh, loc);
        } else {
            if (sv.bu_sparse) {
                bu_layout<BLOCK, KS>(p, sv, team, loc);
            } else {
                bu_layout<BLOCK, KD>(p, sv, team, loc);
            }
        }
        end_step<BLOCK>(p, sv, sh, loc);
    } while (sh.st.dir != kDirDone);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c->st = sh.st;
        c->barrier = sh.st.barrier;
        if (p.result) {
            p.result[0] = sh.st.visited_degsum / 2;
            p.result[1] = sh.st.reached;
        }
    }
}

// ---------------------------------------------------------------------------
// Deterministic tree: parent(v) = min{u in N(v) : depth[u] == depth[v]-1}
// ---------------------------------------------------------------------------
// Bound by the arcs' 4 bytes and the depth gathers.  A warp takes 32 vertices and
// deals their lists, laid end to end, to its lanes, four arcs each with the loads
// issued together; the best neighbour of each vertex is kept by a shared-memory
// minimum, which starts from the parent the search found (any of them is one level
// up), so an arc to a larger id is dropped before its depth is gathered.  Lists of
// more than kMinLong arcs are left as chunks to min_parent_long_kernel: a warp that
// walked a hub's list by itself took 163 us at scale 16, where the search takes 60.
constexpr int64_t kMinLong = 512;  // also the chunk length

struct MinScratch {
    int32_t incl[32];
    uint32_t best[32];
    int32_t up[32];  // depth of a parent
    int64_t beg[32];
};

__global__ void __launch_bounds__(256) min_parent_kernel(const int64_t *off, const uint32_t *adj,
                                                         int64_t n, const int32_t *depth,
                                                         int64_t *parent, bool seeded, uint2 *chunks,
                                                         unsigned long long *count)
{
    __shared__ MinScratch scratch[8];
    MinScratch &ws = scratch[threadIdx.x >> 5];
    const int lane = lane_id();
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long w = gw; w < (n + 31) / 32; w += nw) {
        const int64_t v = w * 32 + lane;
        const int32_t dv = v < n ? depth[v] : -1;
        int64_t beg = 0, deg = 0;
        uint32_t first = 0xFFFFFFFFu;
        if (dv > 0) {
            beg = off[v];
            deg = off[v + 1] - beg;
            if (seeded) { first = (uint32_t)parent[v]; }
        }
        const bool longer = deg > kMinLong;
        if (longer && !seeded) { parent[v] = (int64_t)first; }
        unsigned owners = __ballot_sync(kFull, longer);
        while (owners) {
            const int o = __ffs(owners) - 1;
            owners &= owners - 1;
            const long long k = (__shfl_sync(kFull, deg, o) + kMinLong - 1) / kMinLong;
            unsigned long long at = 0;
            if (lane == 0) { at = atomicAdd(count, (unsigned long long)k); }
            at = __shfl_sync(kFull, at, 0);
            for (long long i = lane; i < k; i += 32) {
                chunks[at + i] = make_uint2((uint32_t)(w * 32 + o), (uint32_t)i);
            }
        }
        const int32_t len = longer ? 0 : (int32_t)deg;
        const int32_t incl = warp_incl_scan(len);
        const int32_t total = __shfl_sync(kFull, incl, 31);
        if (total == 0) { continue; }
        ws.incl[lane] = incl;
        ws.best[lane] = first;
        ws.up[lane] = dv - 1;
        ws.beg[lane] = beg;
        __syncwarp();
        for (int32_t base = 0; base < total; base += 32 * kILP) {
            int at[kILP];
            uint32_t u[kILP];
            bool in[kILP];
#pragma unroll
            for (int i = 0; i < kILP; ++i) { at[i] = 0; }  // lists that end at or before arc e
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
#pragma unroll
                for (int i = 0; i < kILP; ++i) {
                    if (ws.incl[at[i] + d - 1] <= base + i * 32 + lane) { at[i] += d; }
                }
            }
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                const int32_t e = base + i * 32 + lane;
                in[i] = e < total;
                u[i] = 0;
                if (in[i]) {
                    u[i] = __ldg(&adj[ws.beg[at[i]] + (e - (at[i] ? ws.incl[at[i] - 1] : 0))]);
                }
            }
            int32_t du[kILP];
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                in[i] = in[i] && u[i] < *(volatile uint32_t *)&ws.best[at[i]];
                du[i] = in[i] ? __ldg(&depth[u[i]]) : 0;
            }
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                if (in[i] && du[i] == ws.up[at[i]]) { atomicMin(&ws.best[at[i]], u[i]); }
            }
        }
        __syncwarp();
        const uint32_t best = ws.best[lane];
        if (len > 0 && (!seeded || best != first)) { parent[v] = (int64_t)best; }
        __syncwarp();
    }
}

// The chunks min_parent_kernel listed, one per warp at a time.  The last block
// clears the count for the next launch.
__global__ void __launch_bounds__(256) min_parent_long_kernel(const int64_t *off,
                                                              const uint32_t *adj,
                                                              const int32_t *depth,
                                                              int64_t *parent, const uint2 *chunks,
                                                              unsigned long long *count)
{
    const int lane = lane_id();
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long total = (long long)__ldcg(&count[0]);
    for (long long c = gw; c < total; c += nw) {
        const uint2 q = __ldg(&chunks[c]);
        const int64_t b = __ldg(&off[q.x]) + (int64_t)q.y * kMinLong;
        const int64_t e = min(__ldg(&off[q.x + 1]), b + kMinLong);
        const int32_t up = __ldg(&depth[q.x]) - 1;
        // chunks of the same vertex lower it meanwhile: any value is a bound
        const uint32_t bound = (uint32_t)__ldcg(&parent[q.x]);
        uint32_t best = bound;
        for (int64_t base = b; base < e; base += 32 * kILP) {
            uint32_t u[kILP];
            int32_t du[kILP];
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                const int64_t k = base + i * 32 + lane;
                u[i] = k < e ? __ldg(&adj[k]) : 0xFFFFFFFFu;
            }
#pragma unroll
            for (int i = 0; i < kILP; ++i) { du[i] = u[i] < best ? __ldg(&depth[u[i]]) : -2; }
#pragma unroll
            for (int i = 0; i < kILP; ++i) {
                if (du[i] == up && u[i] < best) { best = u[i]; }
            }
        }
        best = __reduce_min_sync(kFull, best);
        if (lane == 0 && best < bound) {
            atomicMin(reinterpret_cast<long long *>(&parent[q.x]), (long long)best);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&count[1], 1ull) == gridDim.x - 1) {
        count[0] = 0;
        count[1] = 0;
    }
}

// The reference's encoding of unreached vertices (hybrid_bfs.cc:433-443).
__global__ void finalize_parents_kernel(const int64_t *off, int64_t n, const int32_t *depth,
                                        int64_t *parent)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        if (depth[v] < 0) {
            const int64_t d = off[v + 1] - off[v];
            parent[v] = d != 0 ? -d : -1;
        }
    }
}

// Depths and parents in the caller's arrays and numbering, with the reference's
// encoding of unreached vertices.  HUB (BD_ORDER_HUB): the traversal arrays are
// indexed, and parents named, by traversal id.  A thread takes V consecutive
// vertices with each stage's reads issued together (V = 4: 16-byte accesses to the
// caller's arrays, which have to be aligned for them): bound by the random sectors
// of depth, parent and numbering, which one vertex a thread left waiting on one
// chain of four reads.
template <bool HUB, int V>
__global__ void __launch_bounds__(256) outputs_kernel(const uint32_t *perm, const uint32_t *iperm,
                                                      const int64_t *off, int64_t n,
                                                      const int32_t *depth, const int64_t *parent,
                                                      int32_t *out_depth, int64_t *out_parent)
{
    static_assert(V == 1 || V == 4, "one vertex or four");
    for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * V; v < n;
         v += (int64_t)gridDim.x * blockDim.x * V) {
        int64_t t[V];
        if constexpr (HUB && V == 4) {
            const uint4 q = __ldg(reinterpret_cast<const uint4 *>(perm + v));
            t[0] = q.x;
            t[1] = q.y;
            t[2] = q.z;
            t[3] = q.w;
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i) { t[i] = HUB ? (int64_t)__ldg(&perm[v + i]) : v + i; }
        }
        int32_t d[V];
        int64_t par[V];
        bool all = true;
#pragma unroll
        for (int i = 0; i < V; ++i) { d[i] = __ldg(&depth[t[i]]); }
#pragma unroll
        for (int i = 0; i < V; ++i) {
            par[i] = d[i] >= 0 ? __ldg(&parent[t[i]]) : 0;
            all = all && d[i] >= 0;
        }
        if constexpr (HUB) {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                if (d[i] >= 0) { par[i] = (int64_t)__ldg(&iperm[par[i]]); }
            }
        }
        if (!all) {
            int64_t o[V + 1];
#pragma unroll
            for (int i = 0; i <= V; ++i) { o[i] = __ldg(&off[v + i]); }
#pragma unroll
            for (int i = 0; i < V; ++i) {
                if (d[i] < 0) { par[i] = o[i + 1] != o[i] ? o[i] - o[i + 1] : -1; }
            }
        }
        if constexpr (V == 4) {
            *reinterpret_cast<int4 *>(out_depth + v) = make_int4(d[0], d[1], d[2], d[3]);
            *reinterpret_cast<longlong2 *>(out_parent + v) = make_longlong2(par[0], par[1]);
            *reinterpret_cast<longlong2 *>(out_parent + v + 2) = make_longlong2(par[2], par[3]);
        } else {
            out_depth[v] = d[0];
            out_parent[v] = par[0];
        }
    }
}

// clear(): no vertex visited but the isolated ones.
__global__ void clear_kernel(int64_t n, const uint32_t *isolated, int32_t *depth, uint32_t *vis)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    int4 *d4 = reinterpret_cast<int4 *>(depth);  // cudaMalloc aligns to 256
    for (int64_t i = t; i < n / 4; i += nt) { d4[i] = make_int4(-1, -1, -1, -1); }
    if (t < (n & 3)) { depth[(n & ~(int64_t)3) + t] = -1; }
    for (int64_t w = t; w < (n + 31) / 32; w += nt) { vis[w] = isolated[w]; }
}

int grid_for(int64_t items, int threads = 256)
{
    int64_t b = (items + threads - 1) / threads;
    if (b < 1) { b = 1; }
    if (b > 148 * 32) { b = 148 * 32; }
    return (int)b;
}

// outputs_kernel for a graph's layout and the caller's arrays.
cudaError_t launch_outputs(const bd_graph *g, const int32_t *depth, const int64_t *parent,
                           int32_t *out_depth, int64_t *out_parent, cudaStream_t s)
{
    const int64_t n = g->n;
    const bool wide = n % 4 == 0 && (reinterpret_cast<uintptr_t>(out_depth) |
                                     reinterpret_cast<uintptr_t>(out_parent)) % 16 == 0;
    auto fn = g->d_perm ? (wide ? outputs_kernel<true, 4> : outputs_kernel<true, 1>)
                        : (wide ? outputs_kernel<false, 4> : outputs_kernel<false, 1>);
    fn<<<grid_for(wide ? n / 4 : n), 256, 0, s>>>(g->d_perm, g->d_iperm, g->d_off, n, depth, parent,
                                                  out_depth, out_parent);
    return cudaGetLastError();
}

using KernelFn = void (*)(BfsParams);

struct KernelChoice {
    KernelFn fn;
    int block;
    size_t smem;  // dynamic shared memory
};

KernelChoice pick_kernel(int block, int kd = 4, int ks = 4)
{
#define BD_KC(B, M, D, S) \
    if (block == B && kd == D && ks == S) { return {bfs_persistent_kernel<B, M, D, S>, B, sizeof(SharedState<B>)}; }
#define BD_KC_B(B, M)                                                                  \
    BD_KC(B, M, 1, 1) BD_KC(B, M, 2, 2) BD_KC(B, M, 4, 4) BD_KC(B, M, 32, 32)          \
    BD_KC(B, M, 2, 32) BD_KC(B, M, 4, 32)
    BD_KC_B(256, 4) BD_KC_B(512, 2) BD_KC_B(1024, 1)
#undef BD_KC_B
#undef BD_KC
    return {nullptr, 0, 0};
}

// Allows the kernel its shared memory and returns the CTAs of the device that
// can be resident at once (0 after an error).
int co_resident_ctas(const KernelChoice &kc, int device)
{
    int per_sm = 0, sms = 0;
    if (cudaFuncSetAttribute((const void *)kc.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kc.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)kc.fn, kc.block,
                                                      kc.smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        return 0;
    }
    return per_sm * sms;
}

}  // namespace

}  // namespace bd

using namespace bd;

struct bd_bfs {
    bd_graph *g = nullptr;
    bd_bfs_opts opts{};
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int32_t *depth = nullptr;
    int64_t *parent = nullptr;
    uint32_t *vis[2] = {nullptr, nullptr};
    uint32_t *qs[2] = {nullptr, nullptr};
    uint32_t *ql[2] = {nullptr, nullptr};
    unsigned long long *qlb[2] = {nullptr, nullptr};
    Ctrl *ctrl = nullptr;
    bd_step *rec = nullptr;
    int64_t *d_sources = nullptr;
    int64_t sources_cap = 0;
    // run_many: a pair of events and of results per root, kept for the next call
    std::vector<cudaEvent_t> events;
    int64_t *d_results = nullptr;
    int64_t results_cap = 0;
    CtrlHead *head = nullptr;  // pinned: where a run's outcome is read back to
    PolicyBlob *policy = nullptr;  // device copy, or null
    KernelChoice kernel{nullptr, 0, 0};
    int grid = 0;
    MinParentScratch min_scratch;  // opts.min_parent
    CheckScratch check;
    bool ctrl_valid = false;  // no launch has failed since the control block was zeroed
    int64_t cap_large = 0;
    // BD_ORDER_HUB graphs: depths and parents in the caller's numbering,
    // filled from the traversal arrays when first read after a run
    int32_t *out_depth = nullptr;
    int64_t *out_parent = nullptr;
    bool cleared = false;
    bool ran = false;
    bool parents_final = false;  // caller-visible depths and parents are up to date
    bool rows_by_run = false;    // the last run queued wrote out_depth and out_parent itself
    bool min_due = false;        // its smallest-parent pass went over the caller's rows only
    int64_t last_source = -1;
    CtrlHead last{};
};

namespace bd {

bd_status bfs_install_policy(bd_bfs *b, const PolicyBlob *blob)
{
    BD_CUDA(cudaSetDevice(b->device));
    if (!blob) {
        cudaFree(b->policy);
        b->policy = nullptr;
        return BD_OK;
    }
    if (!b->policy) { BD_CUDA(cudaMalloc(&b->policy, sizeof(PolicyBlob))); }
    BD_CUDA(cudaMemcpy(b->policy, blob, sizeof(PolicyBlob), cudaMemcpyHostToDevice));
    return BD_OK;
}

namespace {

BfsParams make_params(bd_bfs *b)
{
    BfsParams p{};
    p.off = traversal_off(b->g);
    p.adj = traversal_adj(b->g);
    p.n = b->g->n;
    p.m = b->g->m;
    p.depth = b->depth;
    p.parent = b->parent;
    p.vis[0] = b->vis[0];
    p.vis[1] = b->vis[1];
    p.words = bitmap_words(b->g->n);
    p.n_live = b->g->n_live;
    for (int i = 0; i < 2; ++i) {
        p.qs[i] = b->qs[i];
        p.ql[i] = b->ql[i];
        p.qlb[i] = b->qlb[i];
    }
    p.ctrl = b->ctrl;
    p.rec = b->rec;
    p.rec_cap = kRecCap;
    p.alg = b->opts.alg;
    p.alpha = b->opts.alpha;
    p.beta = b->opts.beta;
    p.large_deg = (uint32_t)b->opts.large_degree;
    p.chunk = (uint32_t)b->opts.chunk_edges;
    p.bu_prefix = b->opts.bu_prefix;
    p.spin_limit = b->opts.spin_limit;
    p.expected_ctas = (unsigned)(b->grid + b->opts.test_extra_ctas);
    p.policy = b->policy;
    p.perm = b->g->d_perm;
    return p;
}

bd_status enqueue_clear(bd_bfs *b)
{
    const int64_t n = b->g->n;
    clear_kernel<<<grid_for(n, 512), 256, 0, b->stream>>>(n, traversal_isolated(b->g), b->depth,
                                                          b->vis[0]);
    BD_CUDA(cudaGetLastError());
    return BD_OK;
}

bd_status ensure_sources(bd_bfs *b, int64_t count)
{
    if (count <= b->sources_cap) { return BD_OK; }
    cudaFree(b->d_sources);
    b->d_sources = nullptr;
    b->sources_cap = 0;
    BD_CUDA(cudaMalloc(&b->d_sources, sizeof(int64_t) * count));
    b->sources_cap = count;
    return BD_OK;
}

// Enqueues the persistent kernel (+ min-parent pass) for `count` sources in
// d_sources, or for the one source given (count 1).  m_c and n_c go to result
// (device) if given.  With out_depth / out_parent (device, n entries each) the results are also written there
// in the caller's ids and the reference's encoding, inside the timed region.
bd_status enqueue_bfs(bd_bfs *b, int64_t count, int64_t source, cudaEvent_t start,
                      cudaEvent_t stop, int64_t *result = nullptr, int32_t *out_depth = nullptr,
                      int64_t *out_parent = nullptr)
{
    BfsParams p = make_params(b);
    p.sources = count > 1 ? b->d_sources : nullptr;
    p.source = source;
    p.source_count = count;
    p.result = result;
    if (!b->ctrl_valid) {
        BD_CUDA(cudaMemsetAsync(b->ctrl, 0, sizeof(Ctrl), b->stream));
        b->ctrl_valid = true;
    }
    // The timed region starts with the source setup, as run_beamer's does
    // (hybrid_bfs.cc:158-160); clear() stays outside it.
    if (start) { BD_CUDA(cudaEventRecord(start, b->stream)); }
    void *args[] = {&p};
    BD_CUDA(cudaLaunchCooperativeKernel((const void *)b->kernel.fn, dim3(b->grid),
                                        dim3(b->kernel.block), args, b->kernel.smem, b->stream));
    if (out_depth) {
        BD_CUDA(launch_outputs(b->g, b->depth, b->parent, out_depth, out_parent, b->stream));
        if (b->opts.min_parent) {
            BD_CUDA(launch_min_parent(b->g, b->min_scratch, out_depth, out_parent, b->stream));
        }
    } else if (b->opts.min_parent) {
        // the smallest parent in the caller's numbering: on a hub graph, map
        // the outputs back first, then pick parents on the caller's CSR
        int32_t *depth = b->depth;
        int64_t *parent = b->parent;
        if (b->out_depth) {
            BD_CUDA(launch_outputs(b->g, depth, parent, b->out_depth, b->out_parent, b->stream));
            depth = b->out_depth;
            parent = b->out_parent;
        }
        BD_CUDA(launch_min_parent(b->g, b->min_scratch, depth, parent, b->stream));
    }
    b->rows_by_run = !out_depth && b->opts.min_parent && b->out_depth;
    b->min_due = out_depth && b->opts.min_parent;
    if (stop) { BD_CUDA(cudaEventRecord(stop, b->stream)); }
    return BD_OK;
}

// Queues the read-back of a run's outcome behind it; the caller waits for the
// stream once, for this and whatever else it queued.
bd_status enqueue_collect(bd_bfs *b)
{
    BD_CUDA(cudaMemcpyAsync(b->head, b->ctrl, sizeof(CtrlHead), cudaMemcpyDeviceToHost, b->stream));
    return BD_OK;
}

bd_status collect(bd_bfs *b, bd_run_stats *stats, double ms)
{
    b->last = *b->head;
    b->ran = true;
    b->cleared = false;
    // (a min-parent run on a hub graph does, unless its rows went to the caller)
    b->parents_final = b->rows_by_run;
    if (b->last.error) {
        b->ctrl_valid = false;
        return (bd_status)b->last.error;
    }
    if (stats) {
        stats->ms = ms;
        stats->num_steps = b->last.st.step;
        stats->reached = b->last.st.reached;
        stats->traversed_edges = b->last.st.visited_degsum / 2;
        stats->top_down_steps = b->last.st.td_steps;
        stats->bottom_up_steps = b->last.st.bu_steps;
    }
    return BD_OK;
}

bd_status run_sources(bd_bfs *b, const int64_t *sources, int64_t count, bd_run_stats *stats)
{
    if (!b || !sources || count <= 0) { return BD_ERR_INVALID; }
    for (int64_t i = 0; i < count; ++i) {
        if (sources[i] < 0 || sources[i] >= b->g->n) { return BD_ERR_RANGE; }
    }
    BD_CUDA(cudaSetDevice(b->device));
    if (!b->cleared) { BD_TRY(enqueue_clear(b)); }
    if (count > 1) {
        BD_TRY(ensure_sources(b, count));
        BD_CUDA(cudaMemcpyAsync(b->d_sources, sources, sizeof(int64_t) * count,
                                cudaMemcpyHostToDevice, b->stream));
    }
    BD_TRY(enqueue_bfs(b, count, sources[0], b->ev0, b->ev1));
    BD_TRY(enqueue_collect(b));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    float ms = 0.f;
    BD_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
    b->last_source = count == 1 ? sources[0] : -1;
    return collect(b, stats, (double)ms);
}

// Makes the caller-visible depths and parents current (queued on the handle's
// stream): the reference's -deg / -1 encoding of unreached vertices, on a hub graph the mapping
// back to the caller's numbering, and the smallest parents where the run left them to do.
bd_status finalize_parents(bd_bfs *b)
{
    if (!b->ran) { return BD_ERR_STATE; }
    if (b->parents_final) { return BD_OK; }
    const int64_t n = b->g->n;
    if (b->out_depth) {
        BD_CUDA(launch_outputs(b->g, b->depth, b->parent, b->out_depth, b->out_parent, b->stream));
    } else {
        finalize_parents_kernel<<<grid_for(n), 256, 0, b->stream>>>(b->g->d_off, n, b->depth,
                                                                  b->parent);
    }
    BD_CUDA(cudaGetLastError());
    if (b->min_due) {
        BD_CUDA(launch_min_parent(b->g, b->min_scratch, b->out_depth ? b->out_depth : b->depth,
                                  b->out_parent ? b->out_parent : b->parent, b->stream));
    }
    b->parents_final = true;  // in stream order
    return BD_OK;
}

void bfs_free(bd_bfs *b)
{
    if (!b) { return; }
    cudaSetDevice(b->device);
    if (b->stream) { cudaStreamSynchronize(b->stream); }
    cudaFree(b->depth);
    cudaFree(b->parent);
    cudaFree(b->out_depth);
    cudaFree(b->out_parent);
    for (int i = 0; i < 2; ++i) {
        cudaFree(b->vis[i]);
        cudaFree(b->qs[i]);
        cudaFree(b->ql[i]);
        cudaFree(b->qlb[i]);
    }
    cudaFree(b->ctrl);
    cudaFree(b->rec);
    cudaFree(b->d_sources);
    cudaFree(b->d_results);
    for (cudaEvent_t e : b->events) { cudaEventDestroy(e); }
    if (b->head) { cudaFreeHost(b->head); }
    cudaFree(b->policy);
    min_parent_free(&b->min_scratch);
    check_free(&b->check);
    if (b->ev0) { cudaEventDestroy(b->ev0); }
    if (b->ev1) { cudaEventDestroy(b->ev1); }
    if (b->stream) { cudaStreamDestroy(b->stream); }
    delete b;
}

}  // namespace

cudaError_t min_parent_alloc(const bd_graph *g, MinParentScratch *s, cudaStream_t stream)
{
    if (g->max_degree <= kMinLong) { return cudaSuccess; }  // nothing is ever listed
    // a list of more than kMinLong arcs has less than 2 arcs / kMinLong chunks
    cudaError_t e = cudaMalloc(&s->chunks, sizeof(uint2) * (2 * g->arcs / kMinLong));
    if (e == cudaSuccess) { e = cudaMalloc(&s->count, sizeof(unsigned long long) * 2); }
    if (e == cudaSuccess) { e = cudaMemsetAsync(s->count, 0, sizeof(unsigned long long) * 2, stream); }
    return e;
}

void min_parent_free(MinParentScratch *s)
{
    cudaFree(s->chunks);
    cudaFree(s->count);
    *s = MinParentScratch{};
}

cudaError_t launch_min_parent(const bd_graph *g, const MinParentScratch &s, const int32_t *depth,
                              int64_t *parent, cudaStream_t stream)
{
    min_parent_kernel<<<grid_for(bitmap_words(g->n) * 32), 256, 0, stream>>>(
        g->d_off, g->d_adj, g->n, depth, parent, g->symmetric, s.chunks, s.count);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !s.chunks) { return e; }
    min_parent_long_kernel<<<148 * 4, 256, 0, stream>>>(g->d_off, g->d_adj, depth, parent, s.chunks,
                                                        s.count);
    return cudaGetLastError();
}

}  // namespace bd

extern "C" {

void bd_bfs_default_opts(bd_bfs_opts *o)
{
    if (!o) { return; }
    memset(o, 0, sizeof(*o));
    o->alg = BD_ALG_BEAMER;
    o->alpha = 15;
    o->beta = 18;
}

bd_status bd_bfs_create(bd_graph *g, const bd_bfs_opts *opts, bd_bfs **out)
{
    if (!g || !out) { return BD_ERR_INVALID; }
    bd_bfs_opts o;
    bd_bfs_default_opts(&o);
    if (opts) { o = *opts; }
    if (o.alg < BD_ALG_BEAMER || o.alg > BD_ALG_LEARNED || o.alpha <= 0 || o.beta <= 0) {
        return BD_ERR_INVALID;
    }
    if (o.block_size == 0) { o.block_size = 512; }
    if (o.block_size != 256 && o.block_size != 512 && o.block_size != 1024) { return BD_ERR_INVALID; }
    if (o.bu_words == 0) { o.bu_words = 4; }
    if (o.bu_sparse_words == 0) { o.bu_sparse_words = o.bu_words == 1 ? 1 : 32; }
    if (o.large_degree <= 0) { o.large_degree = 32; }
    if (o.large_degree > (1 << 20)) { return BD_ERR_INVALID; }
    if (o.chunk_edges <= 0) { o.chunk_edges = 256; }
    if (o.bu_prefix <= 0) { o.bu_prefix = 32; }
    if (o.spin_limit <= 0) { o.spin_limit = kDefaultSpin; }
    if (o.test_extra_ctas < 0) { return BD_ERR_INVALID; }
    BD_TRY(ensure_device());
    auto *b = new bd_bfs();
    b->g = g;
    b->opts = o;
    b->device = current_device();
    const int64_t n = g->n;
    const int64_t words = bitmap_words(n);
    b->cap_large = std::min<int64_t>(n, g->arcs / o.large_degree + 1);
    auto fail = [&](bd_status st) { bfs_free(b); return st; };
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess) {
        return fail(BD_ERR_CUDA);
    }
    bool ok = cudaMalloc(&b->depth, sizeof(int32_t) * n) == cudaSuccess &&
              cudaMalloc(&b->parent, sizeof(int64_t) * n) == cudaSuccess &&
              (!g->d_perm || (cudaMalloc(&b->out_depth, sizeof(int32_t) * n) == cudaSuccess &&
                              cudaMalloc(&b->out_parent, sizeof(int64_t) * n) == cudaSuccess)) &&
              cudaMalloc(&b->ctrl, sizeof(Ctrl)) == cudaSuccess &&
              cudaHostAlloc(&b->head, sizeof(CtrlHead), cudaHostAllocDefault) == cudaSuccess &&
              cudaMalloc(&b->rec, sizeof(bd_step) * kRecCap) == cudaSuccess &&
              (!o.min_parent || min_parent_alloc(g, &b->min_scratch, b->stream) == cudaSuccess);
    for (int i = 0; i < 2 && ok; ++i) {
        ok = cudaMalloc(&b->vis[i], sizeof(uint32_t) * words) == cudaSuccess &&
             cudaMalloc(&b->qs[i], sizeof(uint32_t) * n) == cudaSuccess &&
             cudaMalloc(&b->ql[i], sizeof(uint32_t) * b->cap_large) == cudaSuccess &&
             cudaMalloc(&b->qlb[i], sizeof(unsigned long long) * b->cap_large) == cudaSuccess;
    }
    if (!ok) { return fail(BD_ERR_OOM); }
    b->kernel = pick_kernel(o.block_size, o.bu_words, o.bu_sparse_words);
    if (!b->kernel.fn) { return fail(BD_ERR_INVALID); }
    b->grid = co_resident_ctas(b->kernel, b->device);
    if (b->grid < 1) { return fail(BD_ERR_CUDA); }
    *out = b;
    return BD_OK;
}

bd_status bd_bfs_clear(bd_bfs *b)
{
    if (!b) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(b->device));
    BD_TRY(enqueue_clear(b));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    b->cleared = true;
    b->ran = false;
    return BD_OK;
}

bd_status bd_bfs_run(bd_bfs *b, int64_t source, bd_run_stats *stats)
{
    return run_sources(b, &source, 1, stats);
}

bd_status bd_bfs_run_multi(bd_bfs *b, const int64_t *sources, int64_t count, bd_run_stats *stats)
{
    return run_sources(b, sources, count, stats);
}

static bd_status run_with_alg(bd_bfs *b, int alg, int64_t alpha, int64_t beta, int64_t source,
                              bd_run_stats *stats)
{
    if (!b) { return BD_ERR_INVALID; }
    if (alpha <= 0 || beta <= 0) { return BD_ERR_INVALID; }
    bd_bfs_opts saved = b->opts;
    b->opts.alg = alg;
    b->opts.alpha = alpha;
    b->opts.beta = beta;
    bd_status st = run_sources(b, &source, 1, stats);
    b->opts = saved;
    return st;
}

bd_status bd_bfs_run_beamer(bd_bfs *b, int64_t source, int64_t alpha, int64_t beta,
                            bd_run_stats *stats)
{
    return run_with_alg(b, BD_ALG_BEAMER, alpha, beta, source, stats);
}

bd_status bd_bfs_run_top_down(bd_bfs *b, int64_t source, bd_run_stats *stats)
{
    if (!b) { return BD_ERR_INVALID; }
    return run_with_alg(b, BD_ALG_TOP_DOWN, b->opts.alpha, b->opts.beta, source, stats);
}

bd_status bd_bfs_run_bottom_up(bd_bfs *b, int64_t source, bd_run_stats *stats)
{
    if (!b) { return BD_ERR_INVALID; }
    return run_with_alg(b, BD_ALG_BOTTOM_UP, b->opts.alpha, b->opts.beta, source, stats);
}

}  // extern "C"

namespace bd {
namespace {

constexpr int64_t kKeptEvents = 2050;  // a handle keeps events for 1024 roots

// Events and result slots for k roots.
bd_status ensure_many(bd_bfs *b, int64_t k)
{
    while ((int64_t)b->events.size() < 2 * k + 2) {
        cudaEvent_t e = nullptr;
        BD_CUDA(cudaEventCreate(&e));
        b->events.push_back(e);
    }
    if (k <= b->results_cap) { return BD_OK; }
    cudaFree(b->d_results);
    b->d_results = nullptr;
    b->results_cap = 0;
    BD_CUDA(cudaMalloc(&b->d_results, sizeof(int64_t) * 2 * k));
    b->results_cap = k;
    return BD_OK;
}

bd_status run_many(bd_bfs *b, const int64_t *sources, int64_t k, int32_t *d_depth,
                   int64_t *d_parent, double *ms_out, int64_t *edges_out, int64_t *reached_out,
                   double *e2e_ms)
{
    if (!b || !sources || k <= 0) { return BD_ERR_INVALID; }
    for (int64_t i = 0; i < k; ++i) {
        if (sources[i] < 0 || sources[i] >= b->g->n) { return BD_ERR_RANGE; }
    }
    BD_CUDA(cudaSetDevice(b->device));
    bd_status st = ensure_many(b, k);
    if (st != BD_OK) { return st; }
    const std::vector<cudaEvent_t> &ev = b->events;  // 2 per root, then the call's 2
    int64_t *d_edges = b->d_results;
    std::vector<int64_t> host_edges(2 * k);
    cudaEventRecord(ev[2 * k], b->stream);
    const int64_t n = b->g->n;
    for (int64_t i = 0; i < k && st == BD_OK; ++i) {
        st = enqueue_clear(b);
        if (st == BD_OK) {
            st = enqueue_bfs(b, 1, sources[i], ev[2 * i], ev[2 * i + 1], d_edges + 2 * i,
                             d_depth ? d_depth + i * n : nullptr,
                             d_depth ? d_parent + i * n : nullptr);
        }
    }
    if (st == BD_OK &&
        (cudaMemcpyAsync(host_edges.data(), d_edges, sizeof(int64_t) * 2 * k, cudaMemcpyDeviceToHost,
                         b->stream) != cudaSuccess ||
         cudaEventRecord(ev[2 * k + 1], b->stream) != cudaSuccess ||
         enqueue_collect(b) != BD_OK || cudaStreamSynchronize(b->stream) != cudaSuccess)) {
        st = BD_ERR_CUDA;
    }
    if (st == BD_OK) {
        float w = 0.f;
        cudaEventElapsedTime(&w, ev[2 * k], ev[2 * k + 1]);
        if (e2e_ms) { *e2e_ms = (double)w; }
        for (int64_t i = 0; i < k; ++i) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]);
            if (ms_out) { ms_out[i] = (double)ms; }
            if (edges_out) { edges_out[i] = host_edges[2 * i]; }
            if (reached_out) { reached_out[i] = host_edges[2 * i + 1]; }
        }
        b->last_source = sources[k - 1];
        st = collect(b, nullptr, 0.0);
    }
    while ((int64_t)b->events.size() > kKeptEvents) {
        cudaEventDestroy(b->events.back());
        b->events.pop_back();
    }
    return st;
}

}  // namespace
}  // namespace bd

extern "C" {

bd_status bd_bfs_run_many(bd_bfs *b, const int64_t *sources, int64_t k, double *ms_out,
                          int64_t *edges_out, int64_t *reached_out, double *e2e_ms)
{
    return run_many(b, sources, k, nullptr, nullptr, ms_out, edges_out, reached_out, e2e_ms);
}

bd_status bd_bfs_run_many_into(bd_bfs *b, const int64_t *sources, int64_t k, int32_t *d_depth,
                               int64_t *d_parent, double *ms_out, int64_t *edges_out,
                               int64_t *reached_out, double *e2e_ms)
{
    if (!d_depth || !d_parent) { return BD_ERR_INVALID; }
    return run_many(b, sources, k, d_depth, d_parent, ms_out, edges_out, reached_out, e2e_ms);
}

bd_status bd_bfs_get_depths(bd_bfs *b, int32_t *depth)
{
    if (!b || !depth) { return BD_ERR_INVALID; }
    if (!b->ran) { return BD_ERR_STATE; }
    BD_CUDA(cudaSetDevice(b->device));
    BD_TRY(finalize_parents(b));
    BD_CUDA(cudaMemcpyAsync(depth, b->out_depth ? b->out_depth : b->depth,
                            sizeof(int32_t) * b->g->n, cudaMemcpyDeviceToHost, b->stream));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    return BD_OK;
}

bd_status bd_bfs_get_parents(bd_bfs *b, int64_t *parent)
{
    if (!b || !parent) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(b->device));
    BD_TRY(finalize_parents(b));
    BD_CUDA(cudaMemcpyAsync(parent, b->out_parent ? b->out_parent : b->parent,
                            sizeof(int64_t) * b->g->n, cudaMemcpyDeviceToHost, b->stream));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    return BD_OK;
}

bd_status bd_bfs_device_ptrs(bd_bfs *b, const int32_t **depth, const int64_t **parent)
{
    if (!b) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(b->device));
    BD_TRY(finalize_parents(b));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    if (depth) { *depth = b->out_depth ? b->out_depth : b->depth; }
    if (parent) { *parent = b->out_parent ? b->out_parent : b->parent; }
    return BD_OK;
}

bd_status bd_bfs_count_traversed_edges(bd_bfs *b, int64_t *out)
{
    if (!b || !out) { return BD_ERR_INVALID; }
    if (!b->ran) { return BD_ERR_STATE; }
    *out = b->last.st.visited_degsum / 2;
    return BD_OK;
}

// hybrid_bfs::check (hybrid_bfs.cc:281-379), on the device (bd_check.cu),
// of the parents the last run left in HBM.
bd_status bd_bfs_check(bd_bfs *b, int64_t source, int32_t *ok)
{
    if (!b || !ok) { return BD_ERR_INVALID; }
    if (source < 0 || source >= b->g->n) { return BD_ERR_RANGE; }
    const int64_t *parent = nullptr;
    BD_TRY(bd_bfs_device_ptrs(b, nullptr, &parent));
    return check_parents_device(b->g, source, parent, ok, nullptr, &b->check);
}

bd_status bd_bfs_get_steps(bd_bfs *b, bd_step *steps, int64_t capacity, int64_t *count)
{
    if (!b || !count || capacity < 0 || (!steps && capacity)) { return BD_ERR_INVALID; }
    if (!b->ran) { return BD_ERR_STATE; }
    int64_t have = std::min<int64_t>(b->last.st.step, kRecCap);
    int64_t take = std::min(have, capacity);
    if (take) {
        BD_CUDA(cudaSetDevice(b->device));
        BD_CUDA(cudaMemcpy(steps, b->rec, sizeof(bd_step) * take, cudaMemcpyDeviceToHost));
    }
    *count = have;
    return BD_OK;
}

bd_status bd_bfs_destroy(bd_bfs *b)
{
    if (!b) { return BD_ERR_INVALID; }
    bfs_free(b);
    return BD_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free entry point (bd_bfs_run_noalloc).
//
// For callers that must not allocate device memory while they run a BFS:
// a service whose device memory is fully carved up in advance by its own
// pool allocator (a cudaMalloc there fails or fragments the pool), or code
// that cannot afford the device-wide synchronisation cudaMalloc / cudaFree
// may cause.  The caller passes the CSR and the output arrays; every
// temporary (control block, the two visited bitmaps, the frontier queues)
// lives in one file-scope device array of fixed size, so graphs are limited
// to BD_NOALLOC_MAX_VERTICES vertices.  Each GPU that loads this library
// holds that array (about 7.2 MB) until the process exits.
// ---------------------------------------------------------------------------
namespace bd {
namespace {

constexpr int64_t kNaMaxVertices = BD_NOALLOC_MAX_VERTICES;
constexpr int64_t kNaWords = kNaMaxVertices / 32;
constexpr int64_t kNaLarge = 1 << 17;  // slots for large-degree frontier vertices
constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kNaOffCtrl = 0;
constexpr size_t kNaOffLive = align256(kNaOffCtrl + sizeof(Ctrl));  // vertices of nonzero degree
constexpr size_t kNaOffVis = align256(kNaOffLive + sizeof(unsigned long long));
constexpr size_t kNaOffQs = align256(kNaOffVis + 2 * sizeof(uint32_t) * kNaWords);
constexpr size_t kNaOffQl = align256(kNaOffQs + 2 * sizeof(uint32_t) * kNaMaxVertices);
constexpr size_t kNaOffQlb = align256(kNaOffQl + 2 * sizeof(uint32_t) * kNaLarge);
constexpr size_t kNaBytes = align256(kNaOffQlb + 2 * sizeof(unsigned long long) * kNaLarge);

// The scratch array.  Host code must not use this name as an address: it
// gets the device address from cudaGetSymbolAddress (noalloc_scratch_base).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
unsigned char *g_na_base[kNaMaxDevices] = {};
int g_na_grid[kNaMaxDevices] = {};

// Once per device, with that device current: the device address of the
// scratch array and the co-resident grid size of the persistent kernel.
bd_status noalloc_setup(int dev, unsigned char **base, int *grid)
{
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_base[dev]) {
        void *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess) { return cuda_fail(e, "cudaGetSymbolAddress", __FILE__, __LINE__); }
        const int ctas = co_resident_ctas(pick_kernel(512), dev);
        if (ctas < 1) { return cuda_fail(cudaGetLastError(), "occupancy", __FILE__, __LINE__); }
        g_na_grid[dev] = ctas;
        g_na_base[dev] = static_cast<unsigned char *>(ptr);
    }
    *base = g_na_base[dev];
    *grid = g_na_grid[dev];
    return BD_OK;
}

// depth = -1; vis[0] = degree-zero and padding bits; the count of vertices of
// nonzero degree added into *live (zeroed before).
__global__ void noalloc_prepare_kernel(const int64_t *off, int64_t n, int32_t *depth,
                                       uint32_t *vis0, unsigned long long *live)
{
    const int64_t words = (n + 31) / 32;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t v = t; v < n; v += stride) { depth[v] = -1; }
    unsigned long long nz = 0;
    for (int64_t w = t; w < words; w += stride) {
        uint32_t b = 0;
        for (int k = 0; k < 32; ++k) {
            const int64_t v = w * 32 + k;
            if (v >= n || off[v + 1] == off[v]) { b |= 1u << k; }
        }
        vis0[w] = b;
        nz += 32 - __popc(b);
    }
    nz = dev::warp_sum(nz);
    if (dev::lane_id() == 0 && nz) { atomicAdd(live, nz); }
}

}  // namespace
}  // namespace bd

extern "C" bd_status bd_bfs_run_noalloc(const int64_t *d_offsets, const uint32_t *d_adjacency,
                                        int64_t num_vertices, int64_t num_arcs, int64_t source,
                                        int64_t alpha, int64_t beta, int32_t *d_depth,
                                        int64_t *d_parent, void *stream,
                                        int64_t *traversed_edges)
{
    using namespace bd;
    if (!d_offsets || (!d_adjacency && num_arcs) || !d_depth || !d_parent || num_vertices <= 0 ||
        num_arcs < 0 || alpha <= 0 || beta <= 0) {
        return BD_ERR_INVALID;
    }
    if (num_vertices > kNaMaxVertices || num_arcs > ((int64_t)1 << 34)) { return BD_ERR_LIMIT; }
    if (source < 0 || source >= num_vertices) { return BD_ERR_RANGE; }
    int dev = 0, major = 0;
    BD_CUDA(cudaGetDevice(&dev));
    BD_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10 || dev >= kNaMaxDevices) { return BD_ERR_NODEV; }
    unsigned char *base = nullptr;
    int grid = 0;
    BD_TRY(noalloc_setup(dev, &base, &grid));
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    BfsParams p{};
    p.off = d_offsets;
    p.adj = d_adjacency;
    p.n = num_vertices;
    p.m = num_arcs / 2;
    p.depth = d_depth;
    p.parent = d_parent;
    p.words = bitmap_words(num_vertices);
    Ctrl *ctrl = reinterpret_cast<Ctrl *>(base + kNaOffCtrl);
    unsigned long long *live = reinterpret_cast<unsigned long long *>(base + kNaOffLive);
    for (int i = 0; i < 2; ++i) {
        p.vis[i] = reinterpret_cast<uint32_t *>(base + kNaOffVis) + i * kNaWords;
        p.qs[i] = reinterpret_cast<uint32_t *>(base + kNaOffQs) + i * kNaMaxVertices;
        p.ql[i] = reinterpret_cast<uint32_t *>(base + kNaOffQl) + i * kNaLarge;
        p.qlb[i] = reinterpret_cast<unsigned long long *>(base + kNaOffQlb) + i * kNaLarge;
    }
    p.ctrl = ctrl;
    p.rec = nullptr;
    p.rec_cap = 0;
    p.alg = BD_ALG_BEAMER;
    p.alpha = alpha;
    p.beta = beta;
    // The regular handle's defaults (bd_bfs_create), except that the
    // large-degree threshold rises above them on graphs of more than
    // 32 x kNaLarge arcs: at most num_arcs / large_deg vertices qualify, and
    // the array holds kNaLarge of them.
    p.large_deg = (uint32_t)std::max<int64_t>(32, num_arcs / kNaLarge + 1);
    p.chunk = 256;
    p.bu_prefix = 32;
    p.spin_limit = kDefaultSpin;
    p.expected_ctas = (unsigned)grid;
    p.policy = nullptr;
    p.source = source;
    p.source_count = 1;

    // The control block, live count and vis[0] are rewritten
    // here; the queues and vis[1] are written before they are read within a
    // run.  The live count (vertices of nonzero degree) decides the
    // bottom-up layout switch, so it is read back before the launch.
    BD_CUDA(cudaMemsetAsync(base + kNaOffCtrl, 0,
                            kNaOffLive + sizeof(unsigned long long) - kNaOffCtrl, s));
    noalloc_prepare_kernel<<<grid_for(std::max<int64_t>(num_vertices, 1)), 256, 0, s>>>(
        d_offsets, num_vertices, d_depth, p.vis[0], live);
    BD_CUDA(cudaGetLastError());
    unsigned long long n_live = 0;
    BD_CUDA(cudaMemcpyAsync(&n_live, live, sizeof(n_live), cudaMemcpyDeviceToHost, s));
    BD_CUDA(cudaStreamSynchronize(s));
    p.n_live = (int64_t)n_live;
    KernelChoice kc = pick_kernel(512);
    void *args[] = {&p};
    BD_CUDA(cudaLaunchCooperativeKernel((const void *)kc.fn, dim3(grid), dim3(kc.block), args,
                                        kc.smem, s));
    finalize_parents_kernel<<<grid_for(num_vertices), 256, 0, s>>>(d_offsets, num_vertices, d_depth,
                                                                   d_parent);
    BD_CUDA(cudaGetLastError());
    CtrlHead host{};
    BD_CUDA(cudaMemcpyAsync(&host, ctrl, sizeof(CtrlHead), cudaMemcpyDeviceToHost, s));
    BD_CUDA(cudaStreamSynchronize(s));
    if (host.error) { return (bd_status)host.error; }
    if (traversed_edges) { *traversed_edges = host.st.visited_degsum / 2; }
    return BD_OK;
}
