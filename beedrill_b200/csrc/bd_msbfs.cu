// bd_msbfs.cu -- batched traversal: up to 64 BFSs at once, one bit lane of a
// uint64 per root ("multi-source BFS"), in one persistent cooperative launch.
//
// The reference runs its trials one root at a time (hybrid_bfs_main.cc:252-302);
// every root re-reads the whole graph.  Here R <= 64 roots share each pass
// over the adjacency: vertex v carries reach[v] (lanes delivered to it so
// far, this step's deliveries included) and F[v] (lanes whose frontier holds
// it), and a level updates all lanes with 64-bit ORs.  Results per lane are exactly
// those of a single-source BFS from that lane's root: depths equal, parents
// one level up (each (vertex, lane) gets the first neighbour that delivered
// the lane's bit).
//
// Steps, chosen per level on the device (Beamer-style rule over the batch):
//   push  frontier vertices OR their lanes into their neighbours' reach
//         word (atomicOr; the returned old word identifies the one writer
//         that delivered each new lane, which becomes that lane's parent),
//         then into the next frontier word;
//   pull  each vertex not yet reached by every lane ORs its neighbours'
//         frontier words until it has all the lanes it still needs that
//         some frontier holds (the lanes delivered by the step before).
//
// Layout in HBM (n vertices, R lanes):
//   reach   uint64[n]      lanes delivered to v so far: one load tells a
//                          push which lanes v still lacks; after the run,
//                          the lanes that reached v
//   F[3]    uint64[n]      frontier words, three buffers: step s reads
//                          F[s%3], writes F[(s+1)%3], clears F[(s+2)%3]
//   Q[3]                   the vertex lists of those frontiers (degree bins)
//   done    uint32[n/32]   vertices every lane has reached, and isolated ones:
//                          pull steps skip them by the word
//   drec    16 B [n][16]   delivery records: {lane mask lo, hi, provider,
//                          level}, one store for all the lanes one
//                          neighbour delivered at one level, push or pull
//                          (drec_cnt[n] counts them)
//   depth   int32[n][R]    per-lane rows, vertex-major (a vertex's lanes share
//   parent  uint32[n][R]   sectors): deliveries past a vertex's 16 records
// The kernel leaves F zero when it ends (it clears the last
// frontier's words), so a call needs no memsets of them.
#include <algorithm>
#include <cstring>
#include <vector>

#include "bd_device_util.cuh"
#include "bd_internal.h"
#include "bd_policy.cuh"

namespace bd {
namespace {

using namespace dev;
using ull = unsigned long long;

constexpr int kPush = 0, kPull = 1, kMsDone = 2;
constexpr int kLargeShift = 38;
constexpr ull kChunkMask = (1ull << kLargeShift) - 1;
constexpr int64_t kMsRecCap = 1 << 14;
constexpr long long kMsDefaultSpin = 4000000;
constexpr unsigned kRecSlots = 16;  // delivery records per vertex

// Counters of one step, in a ring of three slots (step s uses s % 3; CTA 0
// clears (s + 1) % 3 during step s, after every CTA has read it).
struct alignas(16) MsAcc {
    ull vertices;    // vertices entering the next frontier
    ull degsum;      // their degree sum
    ull lanes;       // new (vertex, lane) pairs
    ull small_cnt;
    ull large_packed;
    ull done_degsum; // degree sum of vertices that just got every lane
    ull t_end;       // max over CTAs of their arrival time
    ull lanes_or;    // lanes delivered in the step (the next frontier's lanes)
    ull work;        // pull steps: next bitmap word to hand out
    ull deferred;    // pull steps: chunks of long lists left for all warps
};

// State between steps: written first by the init kernel, then kept by every
// CTA as an identical copy in shared memory (advanced by the same function
// of the same counters), written back by CTA 0 at the end.
struct MsState {
    int dir, level, step, prev_dir;
    long long f_count, f_degsum, f_small, f_large, f_chunks;
    long long p_small, p_large;  // lists of the frontier read by the previous step
    long long arcs_left;         // 2m - degree sum of vertices reached by all lanes
    long long lanes_total;
    long long t_last, push_steps, pull_steps;
    long long prev_ns, policy_overrides;
    ull active;                  // lanes the frontier about to be expanded holds
    long long bars;              // grid barriers passed
};

// The control block; its head is what the host reads after a run.
struct alignas(16) MsCtrlHead {
    ull bar;       // barrier arrivals; barrier b is complete at (b + 1) * CTAs
    int error, pad0;
    ull t_start;   // min over CTAs of their start time
    MsState st;
};
struct MsCtrl : MsCtrlHead {
    MsAcc acc[3];
};

// Pinned host memory of a call: the group's sources (64 each), the per-lane counts
// (128 each) and the head of the control block.
struct MsHostIo {
    MsCtrlHead head;
    int64_t *sources;
    ull *counts;
};

struct MsParams {
    const int64_t *off;
    const uint32_t *adj;
    uint32_t *done;   // bit v: every lane reached v, or v is isolated (no lane can)
    int64_t n, m;
    ull *reach;       // lanes delivered to v so far (the handle's seen array)
    ull *F[3];
    uint32_t *qs[3];
    uint32_t *ql[3];
    ull *qlb[3];
    int32_t *depth;     // per-lane rows, used when a vertex runs out of records
    uint32_t *parent;
    uint4 *drec;        // [n][kRecSlots] delivery records {mask lo, mask hi, provider, level}
    uint32_t *drec_cnt; // [n] records written (may exceed kRecSlots)
    int R;
    ull all;
    MsCtrl *ctrl;
    bd_step *rec;
    int64_t rec_cap;
    int64_t alpha;
    uint32_t large_deg, chunk;
    int prefix;
    long long spin_limit;
    unsigned expected_ctas;
    int force_dir;  // -1 rule, kPush, kPull
    const PolicyBlob *policy;  // null: the rule decides
    const uint32_t *perm;      // caller id -> traversal id (BD_ORDER_HUB), or null
    // pull scans longer than long_arcs: what is left after so many arcs goes to
    // all warps in chunks of long_chunk arcs, listed in dq as {vertex, chunk}
    uint2 *dq;         // null: no list of the graph is that long
    int64_t long_arcs;
    uint32_t long_chunk;
};

struct MsLocal {
    ull vertices, degsum, lanes, done_degsum, lanes_or;
};

// Frontier word of v (zero outside the frontier).  Read directly: most arcs
// a pull scans lead to frontier hubs, whose words the hub layout keeps in
// L2, so checking the frontier bitmap first would only add a dependent load
// to every arc (same-box A/B: the direct read is 12 % faster at RMAT scale
// 24, 16 % at scale 20).  Plain loads: the buffers read in a step are not
// written in it, and every CTA passed the grid barrier's acquire before the
// step.
__device__ __forceinline__ ull frontier_word(const MsParams &p, int buf, uint32_t v)
{
    return p.F[buf][v];
}

__device__ __forceinline__ int64_t ms_degree(const MsParams &p, uint32_t v)
{
    return __ldg(&p.off[v + 1]) - __ldg(&p.off[v]);
}

// Warp-collective append of new frontier vertices, binned by degree
// (same scheme as the single-source kernel).
__device__ __forceinline__ void ms_append(const MsParams &p, MsAcc *acc, int qn, bool has,
                                          uint32_t v, int64_t deg, MsLocal &loc)
{
    if (has) {
        loc.vertices += 1;
        loc.degsum += (ull)deg;
    }
    const int lane = lane_id();
    const bool large = has && deg >= (int64_t)p.large_deg;
    const unsigned sm = __ballot_sync(kFullMask, has && !large);
    if (sm) {
        const int leader = __ffs(sm) - 1;
        ull base = 0;
        if (lane == leader) { base = atomicAdd(&acc->small_cnt, (ull)__popc(sm)); }
        base = __shfl_sync(kFullMask, base, leader);
        if (has && !large) { p.qs[qn][base + __popc(sm & lanemask_lt())] = v; }
    }
    const unsigned lm = __ballot_sync(kFullMask, large);
    if (lm) {
        const ull nch = large ? (ull)((deg + p.chunk - 1) / p.chunk) : 0ull;
        const ull incl = warp_incl_scan(nch);
        const ull total = __shfl_sync(kFullMask, incl, 31);
        const int leader = __ffs(lm) - 1;
        ull old = 0;
        if (lane == leader) {
            old = atomicAdd(&acc->large_packed, ((ull)__popc(lm) << kLargeShift) | total);
        }
        old = __shfl_sync(kFullMask, old, leader);
        if (large) {
            const ull pos = (old >> kLargeShift) + __popc(lm & lanemask_lt());
            p.ql[qn][pos] = v;
            p.qlb[qn][pos] = (old & kChunkMask) + incl - nch;
        }
    }
}

// Warp-collective append of up to K new frontier vertices per lane: one
// atomic for all the small-degree ones of the warp, one for the large ones.
template <int K>
__device__ __forceinline__ void ms_append_k(const MsParams &p, MsAcc *acc, int qn,
                                            const bool (&has)[K], const uint32_t (&v)[K],
                                            const int64_t (&deg)[K], MsLocal &loc)
{
    const int lane = lane_id();
    unsigned sm[K];
    bool large[K];
    unsigned total = 0, any_large = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (has[k]) {
            loc.vertices += 1;
            loc.degsum += (ull)deg[k];
        }
        large[k] = has[k] && deg[k] >= (int64_t)p.large_deg;
        sm[k] = __ballot_sync(kFullMask, has[k] && !large[k]);
        total += __popc(sm[k]);
        any_large |= __ballot_sync(kFullMask, large[k]);
    }
    if (total) {
        ull base = 0;
        if (lane == 0) { base = atomicAdd(&acc->small_cnt, (ull)total); }
        base = __shfl_sync(kFullMask, base, 0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (has[k] && !large[k]) { p.qs[qn][base + __popc(sm[k] & lanemask_lt())] = v[k]; }
            base += __popc(sm[k]);
        }
    }
    if (any_large) {
        unsigned count = 0;
        ull chunks = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (large[k]) {
                count += 1;
                chunks += (ull)((deg[k] + p.chunk - 1) / p.chunk);
            }
        }
        const unsigned ci = warp_incl_scan(count);
        const ull hi = warp_incl_scan(chunks);
        const unsigned ct = __shfl_sync(kFullMask, ci, 31);
        const ull ht = __shfl_sync(kFullMask, hi, 31);
        ull old = 0;
        if (lane == 0) { old = atomicAdd(&acc->large_packed, ((ull)ct << kLargeShift) | ht); }
        old = __shfl_sync(kFullMask, old, 0);
        ull pos = (old >> kLargeShift) + (ci - count);
        ull cbase = (old & kChunkMask) + (hi - chunks);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (large[k]) {
                p.ql[qn][pos] = v[k];
                p.qlb[qn][pos] = cbase;
                pos += 1;
                cbase += (ull)((deg[k] + p.chunk - 1) / p.chunk);
            }
        }
    }
}

// Lanes whose vertex has run out of delivery records: one depth and one
// parent entry per lane in the vertex-major rows.
__device__ __forceinline__ void write_rows(const MsParams &p, uint32_t v, ull lanes, int level,
                                           uint32_t parent)
{
    while (lanes) {
        const int r = __ffsll((long long)lanes) - 1;
        lanes &= lanes - 1;
        p.depth[(int64_t)v * p.R + r] = level;
        p.parent[(int64_t)v * p.R + r] = parent;
    }
}

// Delivery record `slot` of v: the lanes that `parent` delivered at `level`
// (one 16-byte store for all of them).  Past kRecSlots, per-lane rows.
__device__ __forceinline__ void put_record(const MsParams &p, uint32_t v, unsigned slot,
                                           ull lanes, int level, uint32_t parent)
{
    if (slot < kRecSlots) {
        p.drec[(int64_t)v * kRecSlots + slot] =
            make_uint4((uint32_t)lanes, (uint32_t)(lanes >> 32), parent, (uint32_t)level);
    } else {
        write_rows(p, v, lanes, level, parent);
    }
}

// A record from one of several concurrent deliverers (push, chunked pull).
__device__ __forceinline__ void record_shared(const MsParams &p, uint32_t v, ull lanes, int level,
                                              uint32_t parent)
{
    put_record(p, v, atomicAdd(&p.drec_cnt[v], 1u), lanes, level, parent);
}

struct MsView {
    int dir, level, step;
    long long f_small, f_large, f_chunks, p_small, p_large;
    int f_avg;
    ull active;
};

__device__ __forceinline__ MsView ms_view(const MsState &c)
{
    MsView v;
    v.dir = c.dir;
    v.level = c.level;
    v.step = c.step;
    v.f_small = c.f_small;
    v.f_large = c.f_large;
    v.f_chunks = c.f_chunks;
    v.p_small = c.p_small;
    v.p_large = c.p_large;
    v.f_avg = dev::average(c.f_degsum, c.f_count);
    v.active = c.active;
    return v;
}

// This warp among the grid's, consecutive ranks on different CTAs: work items are
// few on narrow levels, and their heavy ones stand together (the first words of a
// hub numbering), so ranks that fill one CTA after another put them on a few SMs,
// whose request rate then bounds the level (the first pull of 64 roots at scale 16:
// 30 us in CTA 0, under 5 in most others).
__device__ __forceinline__ long long ms_warp_rank()
{
    return (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}

// Zeroes the frontier words of the frontier read by the previous step.
__device__ void ms_clear_old(const MsParams &p, const MsView &sv)
{
    const int old = (sv.step + 2) % 3;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nt = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < sv.p_small; i += nt) { p.F[old][p.qs[old][i]] = 0ull; }
    for (long long i = t; i < sv.p_large; i += nt) { p.F[old][p.ql[old][i]] = 0ull; }
}

// push: lanes of frontier vertex u flow into neighbours [b, e), four arcs
// per lane per round with each stage's loads and atomics issued back to
// back.  One plain read of the neighbour's reach word filters the arcs
// that deliver nothing (a vertex every lane has reached holds all lanes in
// it, so no done-bit read is needed); the atomicOr on the
// reach word tells each deliverer which lanes it delivered first -- it
// writes one delivery record for them (a slot from an atomicAdd on the
// vertex's record count; every (vertex, lane) pair is delivered exactly
// once, so no two records hold the same pair; one 16-byte store instead of
// two 4-byte row stores per lane: 5 % off the scale-24 traversal) -- and an
// atomicOr on the next frontier word, issued together with the reach
// update rather than after it, tells which deliverer puts the neighbour on
// the next frontier's list.
constexpr int kPushU = 4;

// One round of up to kPushU arcs per lane: arc i of this lane goes from
// src[i] (whose frontier lanes are bits[i]) to v[i].
__device__ __forceinline__ void push_arcs(const MsParams &p, MsAcc *acc, int cur, int nxt,
                                          int new_level, const bool (&in)[kPushU],
                                          const uint32_t (&v)[kPushU],
                                          const uint32_t (&src)[kPushU],
                                          const ull (&bits)[kPushU], MsLocal &loc)
{
    ull g[kPushU];  // lanes to give, then the lanes this writer delivered first
#pragma unroll
    for (int i = 0; i < kPushU; ++i) {
        // a stale read only costs an atomic that changes nothing (a vertex
        // every lane has reached holds them all in its reach word)
        const ull have = in[i] ? __ldcg(&p.reach[v[i]]) : ~0ull;
        g[i] = bits[i] & ~have;
    }
    // Both atomics at once.  The frontier word takes the lanes v lacked
    // when the step began (the reach read above sees every earlier step's
    // lanes), so it ends up holding exactly the lanes delivered to v in this
    // step whichever deliverer's reach update lands first; the one writer
    // that finds it empty lists v, even if others delivered its lanes first.
    ull old_r[kPushU], old_f[kPushU];
#pragma unroll
    for (int i = 0; i < kPushU; ++i) {
        old_r[i] = g[i] ? atomicOr(&p.reach[v[i]], g[i]) : ~0ull;
        old_f[i] = g[i] ? atomicOr(&p.F[nxt][v[i]], g[i]) : ~0ull;
    }
    bool completed[kPushU], first[kPushU];
#pragma unroll
    for (int i = 0; i < kPushU; ++i) {
        first[i] = g[i] && old_f[i] == 0ull;
        g[i] &= ~old_r[i];
        completed[i] = g[i] && ((old_r[i] | g[i]) & p.all) == p.all;
    }
    int64_t deg[kPushU];
#pragma unroll
    for (int i = 0; i < kPushU; ++i) {
        deg[i] = 0;
        if (g[i]) {
            record_shared(p, v[i], g[i], new_level, src[i]);
            loc.lanes += __popcll(g[i]);
            loc.lanes_or |= g[i];
        }
        if (first[i] || completed[i]) { deg[i] = ms_degree(p, v[i]); }
        if (completed[i]) {
            loc.done_degsum += (ull)deg[i];
            atomicOr(&p.done[v[i] >> 5], 1u << (v[i] & 31));
        }
        if (!first[i]) { deg[i] = 0; }
    }
    ms_append_k<kPushU>(p, acc, nxt, first, v, deg, loc);
}

// Arcs [b, e) of frontier vertex u (lanes `bits`), all 32 lanes, coalesced.
__device__ __forceinline__ void push_edges(const MsParams &p, MsAcc *acc, int cur, int nxt,
                                           int new_level, uint32_t u, ull bits, int64_t b,
                                           int64_t e, MsLocal &loc)
{
    const int lane = lane_id();
    for (int64_t base = b; base < e; base += 32 * kPushU) {
        uint32_t v[kPushU], src[kPushU];
        ull bt[kPushU];
        bool in[kPushU];
#pragma unroll
        for (int i = 0; i < kPushU; ++i) {
            const int64_t k = base + 32 * i + lane;
            in[i] = k < e;
            v[i] = in[i] ? __ldg(&p.adj[k]) : 0u;
            src[i] = u;
            bt[i] = bits;
        }
        push_arcs(p, acc, cur, nxt, new_level, in, v, src, bt, loc);
    }
}

// Per-warp scratch of the small-vertex push: 32 frontier vertices, their
// lanes, list starts and the inclusive prefix of their degrees.
struct MsWarpScratch {
    int32_t incl[32];
    uint32_t u[32];
    int64_t beg[32];
    ull bits[32];
};

template <int BLOCK>
__device__ void ms_push_step(const MsParams &p, const MsView &sv, MsWarpScratch &ws, MsLocal &loc)
{
    const int lane = lane_id();
    const long long gw = ms_warp_rank();
    const long long nw = (long long)gridDim.x * (BLOCK / 32);
    const int cur = sv.step % 3, nxt = (sv.step + 1) % 3;
    MsAcc *acc = &p.ctrl->acc[sv.step % 3];
    const int new_level = sv.level + 1;
    // large frontier vertices: part of chunk c of vertex ql[i]
    const int cut = split_chunks(sv.f_chunks, p.chunk, nw);
    const int64_t part = split_part(p.chunk, cut);
    for (long long x = gw; x < sv.f_chunks << cut; x += nw) {
        const long long c = x >> cut;
        long long lo = 0, hi = sv.f_large - 1;
        while (lo < hi) {
            long long mid = (lo + hi + 1) >> 1;
            if ((long long)__ldcg(&p.qlb[cur][mid]) <= c) { lo = mid; } else { hi = mid - 1; }
        }
        const uint32_t u = __ldcg(&p.ql[cur][lo]);
        const long long j = c - (long long)__ldcg(&p.qlb[cur][lo]);
        const ull bits = __ldcg(&p.F[cur][u]);
        const int64_t ub = __ldg(&p.off[u]) + j * (int64_t)p.chunk;
        const int64_t ue = min(__ldg(&p.off[u + 1]), ub + (int64_t)p.chunk);
        const int64_t b = ub + (x & ((1ll << cut) - 1)) * part;
        push_edges(p, acc, cur, nxt, new_level, u, bits, b, min(ue, b + part), loc);
    }
    // small frontier vertices, up to 32 per warp: their lists are laid end to end
    // and dealt to the lanes kPushU x 32 arcs at a time
    const int group = split_group(sv.f_small, sv.f_avg, nw);
    for (long long g = gw; g << group < sv.f_small; g += nw) {
        const long long idx = (g << group) + lane;
        uint32_t u = 0;
        ull bits = 0;
        int64_t beg = 0;
        int32_t deg = 0;
        if (lane >> group == 0 && idx < sv.f_small) {
            u = __ldcg(&p.qs[cur][idx]);
            bits = __ldcg(&p.F[cur][u]);
            beg = __ldg(&p.off[u]);
            deg = (int32_t)(__ldg(&p.off[u + 1]) - beg);
        }
        const int32_t incl = warp_incl_scan(deg);
        const int32_t total = __shfl_sync(kFullMask, incl, 31);
        ws.incl[lane] = incl;
        ws.u[lane] = u;
        ws.beg[lane] = beg;
        ws.bits[lane] = bits;
        __syncwarp();
        for (int32_t base = 0; base < total; base += 32 * kPushU) {
            uint32_t v[kPushU], src[kPushU];
            ull bt[kPushU];
            bool in[kPushU];
#pragma unroll
            for (int i = 0; i < kPushU; ++i) {
                const int32_t e = base + i * 32 + lane;
                in[i] = e < total;
                v[i] = 0;
                src[i] = 0;
                bt[i] = 0;
                if (in[i]) {
                    int lo = 0, hi = 31;  // first owner with incl > e
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (ws.incl[mid] > e) { hi = mid; } else { lo = mid + 1; }
                    }
                    const int32_t excl = lo ? ws.incl[lo - 1] : 0;
                    src[i] = ws.u[lo];
                    bt[i] = ws.bits[lo];
                    v[i] = __ldg(&p.adj[ws.beg[lo] + (e - excl)]);
                }
            }
            push_arcs(p, acc, cur, nxt, new_level, in, v, src, bt, loc);
        }
        __syncwarp();
    }
}

// The part of a pull step that comes after ms_pull_step: the chunks of the long
// lists it left, one chunk per warp at a time.  A chunk ORs the lanes it finds
// into the vertex's next frontier word; the bits the atomic returns as new are
// the ones this chunk delivered first, so their parents come from this chunk.
template <int BLOCK>
__device__ void ms_pull_long(const MsParams &p, const MsView &sv, MsLocal &loc)
{
    const int lane = lane_id();
    const long long gw = ms_warp_rank();
    const long long nw = (long long)gridDim.x * (BLOCK / 32);
    const int cur = sv.step % 3, nxt = (sv.step + 1) % 3;
    MsAcc *acc = &p.ctrl->acc[sv.step % 3];
    const int new_level = sv.level + 1;
    const long long total = (long long)__ldcg(&acc->deferred);
    // chunks dealt round robin: the chunks of one vertex run on different
    // warps at once, and any of them may find the vertex's last missing lanes
    for (long long c = gw; c < total; c += nw) {
        const uint2 d = __ldcg(&p.dq[c]);
        const uint32_t v = d.x;
        // lanes v lacks that the frontier holds (other chunks of v may have
        // delivered some already this step)
        const ull need = p.all & ~__ldcg(&p.reach[v]) & sv.active;
        if (!need) { continue; }
        const int64_t vb = __ldg(&p.off[v]), ve = __ldg(&p.off[v + 1]);
        const int64_t b = vb + p.long_arcs + (int64_t)d.y * (int64_t)p.long_chunk;
        const int64_t e = min(ve, b + (int64_t)p.long_chunk);
        ull have = 0;  // lanes this chunk found or saw others deliver
        for (int64_t base = b; base < e && (have & need) != need; base += 128) {
            uint32_t u[4];
            ull fu[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t k = base + 32 * i + lane;
                u[i] = k < e ? __ldg(&p.adj[k]) : 0u;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t k = base + 32 * i + lane;
                fu[i] = k < e ? frontier_word(p, cur, u[i]) & need : 0ull;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ull f = fu[i] & ~have;
                if (!__any_sync(kFullMask, f != 0)) { continue; }
                const ull mine = f & ~warp_excl_or(f);
                const ull round = warp_or(f);
                ull old = 0, before = 0;
                if (lane == 0) {
                    // both atomics at once: the reach update takes the whole
                    // round (lanes another chunk delivered first are already
                    // in it), and the one update that completes v marks it
                    old = atomicOr(&p.F[nxt][v], round);
                    before = atomicOr(&p.reach[v], round) & p.all;
                }
                old = __shfl_sync(kFullMask, old, 0);
                const ull fresh = round & ~old;
                if (mine & fresh) { record_shared(p, v, mine & fresh, new_level, u[i]); }
                const bool first = lane == 0 && old == 0ull;
                if (lane == 0) {
                    loc.lanes += __popcll(fresh);
                    loc.lanes_or |= fresh;
                    if (before != p.all && ((before | round) & p.all) == p.all) {
                        loc.done_degsum += (ull)(ve - vb);
                        atomicOr(&p.done[v >> 5], 1u << (v & 31));
                    }
                }
                ms_append(p, acc, nxt, first, v, ve - vb, loc);
                have |= round | old;
            }
        }
    }
}

// The next chunk of a step's work for the calling warp: its own first
// (index gw, no atomic), then, when there are more chunks than warps, from
// the step's counter as chunk nw + k.
__device__ __forceinline__ ull ms_next_chunk(ull *counter, long long nw, long long chunks)
{
    if (chunks <= nw) { return (ull)chunks; }
    ull x = 0;
    if (lane_id() == 0) { x = atomicAdd(counter, 1ull); }
    return (ull)nw + __shfl_sync(kFullMask, x, 0);
}

// Warp-collective: lists the chunks of `rest` arcs of each lane with `has`.
__device__ __forceinline__ void ms_defer(const MsParams &p, MsAcc *acc, bool has, uint32_t v,
                                         int64_t rest)
{
    const unsigned k = has ? (unsigned)((rest + p.long_chunk - 1) / p.long_chunk) : 0u;
    const unsigned incl = warp_incl_scan(k);
    ull base = 0;
    if (lane_id() == 31) { base = atomicAdd(&acc->deferred, (ull)incl); }
    base = __shfl_sync(kFullMask, base, 31);
    unsigned owners = __ballot_sync(kFullMask, k != 0);
    while (owners) {
        const int o = __ffs(owners) - 1;
        owners &= owners - 1;
        const unsigned n = __shfl_sync(kFullMask, k, o);
        const ull at = base + __shfl_sync(kFullMask, incl, o) - n;
        const uint32_t vo = __shfl_sync(kFullMask, v, o);
        for (unsigned i = lane_id(); i < n; i += 32) { p.dq[at + i] = make_uint2(vo, i); }
    }
}

// pull: warp per 32 vertices; a lane scans the first `prefix` arcs of its own
// vertex, the warp goes on with the lists that still lack lanes, one after
// another, up to long_arcs arcs of each; what is left of longer lists is put on
// dq for all warps (ms_pull_long).  Leaving no long list to one warp is what
// bounds the step: a hub numbering puts 32 vertices of the highest degrees into
// one warp's word, and a lane of the batch whose frontier is still small keeps
// every scan from ending early.  With only lists above 4096 arcs dealt out, the
// first pull of 64 roots at scale 20 took 100 us or 1,170 us, by whether the
// batch had such a lane.
template <int BLOCK>
__device__ void ms_pull_step(const MsParams &p, const MsView &sv, MsLocal &loc)
{
    const int lane = lane_id();
    const int cur = sv.step % 3, nxt = (sv.step + 1) % 3;
    MsAcc *acc = &p.ctrl->acc[sv.step % 3];
    const int new_level = sv.level + 1;
    const long long words = (p.n + 31) / 32;
    // Which words a warp walks.  Large graphs (at least two 32-word chunks
    // per warp): chunks handed out dynamically -- the warp's own first, then
    // from a counter of the step -- because work per word varies widely and
    // dynamic hand-out keeps the warps of a CTA finishing together; chunk c
    // holds words c, c + C, c + 2C, ... (C chunks), so the heavy
    // low-numbered words of a hub layout are spread over all chunks.
    // Smaller graphs: warp gw owns words gw, gw + nw, gw + 2 nw, ... (a
    // chunk per warp would leave most warps idle).  Either way a warp loads
    // 32 skip masks at once (one per lane) and walks only the words with
    // work: done vertices have nothing to do.
    const long long gw = ms_warp_rank();
    const long long nw = (long long)gridDim.x * (BLOCK / 32);
    const long long chunks = (words + 31) / 32;
    const bool dynamic = chunks >= 2 * nw;
    const long long stride = dynamic ? chunks : nw;
    const long long limit = dynamic ? chunks : words;
    for (long long base = gw; base < limit;
         base = dynamic ? (long long)ms_next_chunk(&acc->work, nw, chunks) : base + 32 * nw) {
        const long long wl = base + lane * stride;
        const uint32_t sk = wl < words ? __ldcg(&p.done[wl]) : kFullMask;
        unsigned todo = __ballot_sync(kFullMask, sk != kFullMask);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const long long w = base + src * stride;
            const uint32_t skip = __shfl_sync(kFullMask, sk, src);
            const uint32_t v = (uint32_t)(w * 32 + lane);
            const bool live = !((skip >> lane) & 1u);
            ull need = 0, got = 0, s = 0;
            int64_t beg = 0, end = 0, next = 0;
            unsigned cnt = 0, cnt0 = 0;  // this vertex's delivery records
            if (live) {
                // lanes v lacks that some frontier vertex holds: only lanes
                // delivered by the previous step can arrive in this one
                s = __ldcg(&p.reach[v]);
                need = p.all & ~s & sv.active;
                if (need) {
                    beg = __ldg(&p.off[v]);
                    end = __ldg(&p.off[v + 1]);
                    cnt = cnt0 = __ldcg(&p.drec_cnt[v]);
                    const int64_t lim = min(end, beg + (int64_t)p.prefix);
                    int64_t k = beg;
                    // four arcs in flight per round
                    for (; k < lim && got != need; k += 4) {
                        uint32_t u[4];
                        ull fu[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) { u[i] = (k + i < lim) ? __ldg(&p.adj[k + i]) : 0u; }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            fu[i] = (k + i < lim) ? frontier_word(p, cur, u[i]) : 0ull;
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const ull f = fu[i] & need & ~got;
                            if (f) {
                                got |= f;
                                put_record(p, v, cnt++, f, new_level, u[i]);
                            }
                        }
                    }
                    next = (got == need) ? end : min(k, lim);
                }
            }
            const int64_t stop = p.dq ? min(end, beg + p.long_arcs) : end;
            unsigned pending = __ballot_sync(kFullMask, need != 0 && got != need && next < stop);
            while (pending) {
                const int owner = __ffs(pending) - 1;
                pending &= pending - 1;
                const int64_t b = __shfl_sync(kFullMask, next, owner);
                const int64_t e = __shfl_sync(kFullMask, stop, owner);
                const ull nd = __shfl_sync(kFullMask, need, owner);
                ull have = __shfl_sync(kFullMask, got, owner);
                const uint32_t vo = __shfl_sync(kFullMask, v, owner);
                unsigned c = __shfl_sync(kFullMask, cnt, owner);
                // 128 arcs per round: four independent gathers per lane
                for (int64_t base = b; base < e && have != nd; base += 128) {
                    uint32_t u[4];
                    ull fu[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int64_t k = base + 32 * i + lane;
                        u[i] = k < e ? __ldg(&p.adj[k]) : 0u;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int64_t k = base + 32 * i + lane;
                        fu[i] = k < e ? frontier_word(p, cur, u[i]) & nd : 0ull;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const ull f = fu[i] & ~have;
                        if (!__any_sync(kFullMask, f != 0)) { continue; }
                        // arcs earlier in the list win: each lane keeps the bits
                        // no lower lane of this batch already delivered
                        const ull mine = f & ~warp_excl_or(f);
                        const unsigned bm = __ballot_sync(kFullMask, mine != 0);
                        if (mine) {
                            put_record(p, vo, c + __popc(bm & lanemask_lt()), mine, new_level, u[i]);
                        }
                        c += __popc(bm);
                        have |= warp_or(f);
                    }
                }
                if (lane == owner) {
                    got = have;
                    cnt = c;
                }
            }
            if (cnt != cnt0) { p.drec_cnt[v] = cnt; }
            if (p.dq) {
                const bool more = need != 0 && got != need && stop < end;
                if (__any_sync(kFullMask, more)) { ms_defer(p, acc, more, v, end - stop); }
            }
            const bool gained = got != 0;
            const bool completed = gained && ((s | got) & p.all) == p.all;
            const unsigned cm = __ballot_sync(kFullMask, completed);
            if (lane == 0 && cm) { atomicOr(&p.done[w], cm); }
            if (gained) {
                // v is this lane's alone until the barrier before
                // ms_pull_long, so plain stores
                p.F[nxt][v] = got;
                p.reach[v] = s | got;
                loc.lanes += __popcll(got);
                loc.lanes_or |= got;
                if (completed) { loc.done_degsum += (ull)(end - beg); }
            }
            ms_append(p, acc, nxt, gained, v, end - beg, loc);
        }
    }
}

// Grid barrier: arrival (one release-add per CTA) and polling until
// every CTA has arrived.  Bounded by p.spin_limit polls.  Thread 0 of each CTA;
// b is the number of barriers passed before.
__device__ __forceinline__ bool ms_arrive_wait(const MsParams &p, long long b)
{
    MsCtrl *c = p.ctrl;
    red_release_add64(&c->bar, 1ull);
    const ull target = (ull)(b + 1) * p.expected_ctas;
    long long it = 0;
    while (ld_acquire64(&c->bar) < target) {
        if (++it > p.spin_limit) {
            atomicExch(&c->error, (int)BD_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(32);
    }
    return true;
}

template <int BLOCK>
struct MsShared {
    MsWarpScratch warp[BLOCK / 32];
    ull red[5][BLOCK / 32];
    MsState st;     // this CTA's copy of the state
    PolicyBlob pol; // the learned policy's weights, staged once
    int consult;    // the policy decides the next step
    bool listed;    // pull step: all chunks of long lists are on dq
};

// The rule: pull once the frontier's edges are a sizeable share of the edges
// still able to deliver a lane (Beamer's alpha test over the batch) ...
__device__ int ms_rule(const MsState &c, const MsParams &p)
{
    if (c.f_count == 0) { return kMsDone; }
    if (p.force_dir >= 0) { return p.force_dir; }
    // ... and only once the frontier holds at least n / 1024 vertices: a
    // pull step sweeps the done bitmap, which a handful of frontier
    // vertices pushing their arcs does not pay for
    return (c.f_degsum * p.alpha > c.arcs_left && c.f_count * 1024 >= p.n) ? kPull : kPush;
}

// Advances the state over the step that just ended.  One thread per CTA;
// every CTA computes the same result.
__device__ void ms_advance(MsState &c, const MsAcc &a, long long t_end)
{
    c.prev_dir = c.dir;
    c.prev_ns = t_end - c.t_last;
    c.t_last = t_end;
    c.lanes_total += (long long)a.lanes;
    c.active = a.lanes_or;
    c.arcs_left -= (long long)a.done_degsum;
    c.p_small = c.f_small;
    c.p_large = c.f_large;
    c.f_count = (long long)a.vertices;
    c.f_degsum = (long long)a.degsum;
    c.f_small = (long long)a.small_cnt;
    c.f_large = (long long)(a.large_packed >> kLargeShift);
    c.f_chunks = (long long)(a.large_packed & kChunkMask);
    if (c.dir == kPush) { c.push_steps += 1; } else { c.pull_steps += 1; }
    c.level += 1;
    c.step += 1;
}

// The end of a step: block reduction of the counters, arrival at the grid
// barrier (one release-add per CTA), acquire polling until all CTAs have
// arrived, then every CTA advances its copy of the state and decides the
// next direction.  Waits are bounded by p.spin_limit polls.
template <int BLOCK>
__device__ void ms_end_step(const MsParams &p, const MsView &sv, MsShared<BLOCK> &sh, MsLocal &loc)
{
    MsCtrl *c = p.ctrl;
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const ull a0 = warp_sum(loc.vertices), a1 = warp_sum(loc.degsum), a2 = warp_sum(loc.lanes),
              a3 = warp_sum(loc.done_degsum), a4 = warp_or(loc.lanes_or);
    if (lane == 0) {
        sh.red[0][warp] = a0;
        sh.red[1][warp] = a1;
        sh.red[2][warp] = a2;
        sh.red[3][warp] = a3;
        sh.red[4][warp] = a4;
    }
    loc = MsLocal{0, 0, 0, 0, 0};
    __syncthreads();
    if (threadIdx.x == 0) {
        ull t[4] = {0, 0, 0, 0}, lanes_or = 0;
        for (int i = 0; i < BLOCK / 32; ++i) {
            for (int j = 0; j < 4; ++j) { t[j] += sh.red[j][i]; }
            lanes_or |= sh.red[4][i];
        }
        const int s = sv.step;
        MsAcc *acc = &c->acc[s % 3];
        if (t[0]) { atomicAdd(&acc->vertices, t[0]); }
        if (t[1]) { atomicAdd(&acc->degsum, t[1]); }
        if (t[2]) { atomicAdd(&acc->lanes, t[2]); }
        if (t[3]) { atomicAdd(&acc->done_degsum, t[3]); }
        if (lanes_or) { atomicOr(&acc->lanes_or, lanes_or); }
        if (blockIdx.x == 0) {
            MsAcc *z = &c->acc[(s + 1) % 3];
            z->vertices = z->degsum = z->lanes = z->small_cnt = z->large_packed = 0;
            z->done_degsum = z->t_end = z->work = z->lanes_or = z->deferred = 0;
        }
        atomicMax(&acc->t_end, (ull)globaltimer());
        MsState &st = sh.st;
        const bool ok = ms_arrive_wait(p, st.bars);
        st.bars += 1;
        if (ok && __ldcg(&c->error) == 0) {
            // 16 bytes a request: all CTAs read this one line at once
            const ulonglong2 *from = reinterpret_cast<const ulonglong2 *>(acc);
            const ulonglong2 w0 = __ldcg(&from[0]), w1 = __ldcg(&from[1]), w2 = __ldcg(&from[2]),
                             w3 = __ldcg(&from[3]);
            MsAcc a;
            a.vertices = w0.x;
            a.degsum = w0.y;
            a.lanes = w1.x;
            a.small_cnt = w1.y;
            a.large_packed = w2.x;
            a.done_degsum = w2.y;
            a.lanes_or = w3.y;
            const long long t_end = (long long)w3.x;
            if (s == 0) { st.t_last = (long long)__ldcg(&c->t_start); }
            if (blockIdx.x == 0 && s < p.rec_cap) {
                bd_step r;
                r.dir = st.dir;
                r.level = st.level;
                r.frontier = st.f_count;
                r.frontier_edges = st.f_degsum;
                r.unexplored_edges = st.arcs_left;
                r.found = (long long)a.lanes;
                r.ns = t_end - st.t_last;
                p.rec[s] = r;
            }
            ms_advance(st, a, t_end);
        } else {
            st.f_count = 0;  // leave the loop
        }
        st.dir = ms_rule(st, p);
        // the network runs only where the frontier's degree sum over the
        // unexplored one lies in the band the policy was trained to decide in
        sh.consult = p.policy && p.force_dir < 0 && st.dir != kMsDone &&
                     policy_in_band(&sh.pol, st.f_degsum, st.arcs_left);
    }
    __syncthreads();
    if (sh.consult) {
        if (threadIdx.x < 32) {
            MsState &st = sh.st;
            const float gap = policy_gap_warp(&sh.pol, st.f_count, st.f_degsum, st.arcs_left,
                                              st.level, p.n, p.m, st.prev_dir, st.prev_ns);
            if (threadIdx.x == 0 && isfinite(gap) && fabsf(gap) >= sh.pol.margin) {
                const int pick = gap > 0.f ? kPull : kPush;
                if (pick != st.dir) { st.policy_overrides += 1; }
                st.dir = pick;
            }
        }
        __syncthreads();
    }
}

template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) msbfs_kernel(MsParams p)
{
    __shared__ MsShared<BLOCK> sh;
    MsCtrl *c = p.ctrl;
    if (threadIdx.x == 0) {
        sh.st = c->st;  // written by the init kernel before this launch
        atomicMin(&c->t_start, (ull)globaltimer());
    }
    if (p.policy) {
        const float *src = reinterpret_cast<const float *>(p.policy);
        float *dst = reinterpret_cast<float *>(&sh.pol);
        for (int i = threadIdx.x; i < (int)(sizeof(PolicyBlob) / sizeof(float)); i += BLOCK) {
            dst[i] = src[i];
        }
    }
    __syncthreads();
    MsLocal loc{0, 0, 0, 0, 0};
    while (sh.st.dir != kMsDone) {
        const MsView sv = ms_view(sh.st);
        ms_clear_old(p, sv);
        if (sv.dir == kPush) {
            ms_push_step<BLOCK>(p, sv, sh.warp[threadIdx.x >> 5], loc);
        } else {
            ms_pull_step<BLOCK>(p, sv, loc);
            if (p.dq) {
                // every CTA's part of the lists is scanned and its chunks are
                // listed (after a timeout they may not all be: none is read, and
                // the end of the step sees the error)
                __syncthreads();
                if (threadIdx.x == 0) {
                    sh.listed = ms_arrive_wait(p, sh.st.bars);
                    sh.st.bars += 1;
                }
                __syncthreads();
                if (sh.listed) { ms_pull_long<BLOCK>(p, sv, loc); }
            }
        }
        ms_end_step<BLOCK>(p, sv, sh, loc);
    }
    // Leave the frontier buffers zero for the next group or call: the only
    // words still set are those of the last frontier read (the queues of
    // step - 1); after an error the host clears them instead.
    if (__ldcg(&c->error) == 0) { ms_clear_old(p, ms_view(sh.st)); }
    if (blockIdx.x == 0 && threadIdx.x == 0) { c->st = sh.st; }
}

// Clears what a group starts from: its reach words and record counts, the
// done bitmap (isolated vertices are done), its counts and the control block
// (the error flag is the call's: only the first group clears it).  One launch instead of four
// memsets and a copy: each of those is a node of the captured graph, and on
// small graphs the gaps between nodes cost more than the bytes.
__global__ void ms_clear_kernel(MsParams p, const uint32_t *isolated, ull *counts, int keep_error)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    const int64_t words = (p.n + 31) / 32;
    for (int64_t v = t; v < p.n; v += nt) {
        p.reach[v] = 0ull;
        p.drec_cnt[v] = 0u;
    }
    for (int64_t w = t; w < words; w += nt) { p.done[w] = isolated[w]; }
    if (t < 128) { counts[t] = 0ull; }
    if (blockIdx.x == 0) {
        const int error = keep_error ? p.ctrl->error : 0;
        __syncthreads();
        uint32_t *c = reinterpret_cast<uint32_t *>(p.ctrl);
        for (unsigned i = threadIdx.x; i < sizeof(MsCtrl) / 4; i += blockDim.x) { c[i] = 0u; }
        __syncthreads();
        if (threadIdx.x == 0) { p.ctrl->error = error; }
    }
}

// Sources: lane r starts at sources[r].  One warp, two lanes of the batch per
// thread, so the dependent reads of all sources (renumbering, offsets) are in
// flight together: one thread walking 64 sources took 157 us at scale 20 (34 us
// for 16 sources at scale 12), a third of the group's traversal.  The lanes of
// equal sources share one record (a source is its own parent in every lane);
// the lowest of them lists the vertex.
__global__ void ms_init_kernel(MsParams p, const int64_t *sources, int count)
{
    __shared__ uint32_t src[64];
    MsCtrl *c = p.ctrl;
    const int lane = lane_id();
    int64_t deg[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int r = lane + 32 * k;
        src[r] = r < count ? (p.perm ? __ldg(&p.perm[sources[r]]) : (uint32_t)sources[r]) : 0u;
        deg[k] = r < count ? ms_degree(p, src[r]) : 0;
    }
    __syncwarp();
    bool first[2], large[2];
    ull mask[2];
    long long done = 0, degsum = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int r = lane + 32 * k;
        mask[k] = 0;
        first[k] = r < count;
        for (int q = 0; q < count; ++q) {
            const bool same = r < count && src[q] == src[r];
            mask[k] |= same ? 1ull << q : 0ull;
            first[k] = first[k] && !(same && q < r);
        }
        large[k] = first[k] && deg[k] >= (int64_t)p.large_deg;
        if (first[k]) {
            const uint32_t s = src[r];
            p.F[0][s] = mask[k];
            p.reach[s] = mask[k];
            p.drec_cnt[s] = 1u;
            put_record(p, s, 0u, mask[k], 0, s);
            degsum += deg[k];
            if (mask[k] == p.all) {
                done += deg[k];
                atomicOr(&p.done[s >> 5], 1u << (s & 31));
            }
        }
    }
    degsum = warp_sum(degsum);
    done = warp_sum(done);
    long long nf = 0, nsmall = 0, nlarge = 0, chunks = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const unsigned fm = __ballot_sync(kFullMask, first[k]);
        const unsigned lm = __ballot_sync(kFullMask, large[k]);
        const long long ch = large[k] ? (deg[k] + p.chunk - 1) / p.chunk : 0;
        const long long incl = warp_incl_scan(ch);
        if (large[k]) {
            const long long pos = nlarge + __popc(lm & lanemask_lt());
            p.ql[0][pos] = src[lane + 32 * k];
            p.qlb[0][pos] = (ull)(chunks + incl - ch);
        } else if (first[k]) {
            p.qs[0][nsmall + __popc(fm & ~lm & lanemask_lt())] = src[lane + 32 * k];
        }
        nf += __popc(fm);
        nlarge += __popc(lm);
        nsmall += __popc(fm & ~lm);
        chunks += __shfl_sync(kFullMask, incl, 31);
    }
    if (lane == 0) {
        c->t_start = ~0ull;
        MsState &st = c->st;  // zero but for these (ms_clear_kernel)
        st.f_count = nf;
        st.f_degsum = degsum;
        st.f_small = nsmall;
        st.f_large = nlarge;
        st.f_chunks = chunks;
        st.arcs_left = 2 * p.m - done;
        st.active = p.all;
        st.lanes_total = count;
        st.dir = ms_rule(st, p);
    }
}

// Per-lane reached count and degree sum (count_num_traversed_edges per root).
// Bound by the 16 bytes per vertex it reads.  A warp takes 32 vertices and goes
// over the DISTINCT reach words among them (in a graph with one giant component
// nearly always one or two): the vertices holding a word are counted and their
// degrees summed once, and thread t adds both to batch lanes t and t + 32 where
// the word has them.  Adding vertex by vertex to 64 shared counters instead, as
// soon as one root of the batch lies outside the giant component, put 63 shared
// atomics on every vertex: 1,609 us at scale 20 against 14 us.
__global__ void __launch_bounds__(256) ms_count_kernel(const ull *seen, const int64_t *off,
                                                       int64_t n, ull all, int R,
                                                       ull *out /* [2][64]: reached, degsum */)
{
    __shared__ ull s_cnt[64], s_deg[64];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) { s_cnt[i] = s_deg[i] = 0; }
    __syncthreads();
    const int lane = lane_id();
    ull cnt[2] = {0, 0}, dsum[2] = {0, 0};
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + lane;
        const ull s = v < n ? __ldg(&seen[v]) & all : 0ull;
        const ull d = s ? (ull)(__ldg(&off[v + 1]) - __ldg(&off[v])) : 0ull;
        unsigned left = __ballot_sync(kFullMask, s != 0);
        while (left) {
            const ull w = __shfl_sync(kFullMask, s, __ffs(left) - 1);
            const bool mine = s == w;
            const unsigned m = __ballot_sync(kFullMask, mine);
            left &= ~m;
            // 32 degrees summed in two halves (24 bits each leave room for the carries)
            const unsigned lo = __reduce_add_sync(kFullMask, mine ? (unsigned)(d & 0xFFFFFFu) : 0u);
            const unsigned hi = __reduce_add_sync(kFullMask, mine ? (unsigned)(d >> 24) : 0u);
            const ull sum = ((ull)hi << 24) + lo, c = (ull)__popc(m);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const bool has = (w >> (lane + 32 * k)) & 1ull;
                cnt[k] += has ? c : 0ull;
                dsum[k] += has ? sum : 0ull;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (cnt[k]) {
            atomicAdd(&s_cnt[lane + 32 * k], cnt[k]);
            atomicAdd(&s_deg[lane + 32 * k], dsum[k]);
        }
    }
    __syncthreads();
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        if (s_cnt[r]) { atomicAdd(&out[r], s_cnt[r]); }
        if (s_deg[r]) { atomicAdd(&out[64 + r], s_deg[r]); }
    }
}

// Lane r's depths and parents in the single-source output format.  Lane r
// reached v iff seen bit r is set; its depth and parent are in the record of
// v whose mask holds bit r, or, when v ran out of records, in the per-lane
// rows.  Nothing else is valid, so neither the rows nor the records need
// clearing between runs (only the record counts do).
__global__ void ms_extract_kernel(const int32_t *depth, const uint32_t *parent, const uint4 *rec,
                                  const uint32_t *rec_cnt, const ull *seen, const int64_t *off,
                                  int64_t n, int R, int r, const uint32_t *perm,
                                  const uint32_t *iperm, int32_t *depth_out, int64_t *parent_out)
{
    // v: the caller's vertex id (output index, off); t: its traversal id
    // (state index, parents named by traversal id) -- equal unless the
    // graph has a hub numbering
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = perm ? (int64_t)perm[v] : v;
        int32_t d = -1;
        uint32_t par = 0;
        if ((seen[t] >> r) & 1ull) {
            const unsigned cnt = min(rec_cnt[t], kRecSlots);
            bool found = false;
            for (unsigned i = 0; i < cnt && !found; ++i) {
                const uint4 x = rec[t * kRecSlots + i];
                const ull mask = ((ull)x.y << 32) | x.x;
                if ((mask >> r) & 1ull) {
                    d = (int32_t)x.w;
                    par = x.z;
                    found = true;
                }
            }
            if (!found) {
                d = depth[t * R + r];
                par = parent[t * R + r];
            }
        }
        if (depth_out) { depth_out[v] = d; }
        if (parent_out) {
            if (d >= 0) {
                parent_out[v] = (int64_t)(iperm && par < n ? iperm[par] : par);
            } else {
                const int64_t g = off[v + 1] - off[v];
                parent_out[v] = g != 0 ? -g : -1;
            }
        }
    }
}

// Every lane of one group in the single-source output format at once: root
// (root0 + r) gets depth_out[(root0 + r) * n + v] and parent_out[...] for
// every caller vertex v (caller ids, the reference's encoding: the source is
// its own parent, unreached vertices -deg or -1).  One pass over the group's
// state instead of one per lane: a thread takes V consecutive caller vertices
// (two where the rows allow 16-byte stores, n even, else one) and
//   fill   reads each vertex's seen word, record count and records once (a
//          record covers every lane one provider delivered at one level, so
//          the provider is renamed once per record) and the per-lane rows of
//          lanes past its records.  Every distinct (depth, parent) pair gets
//          a slot of a 16-entry table in shared memory (a record's slot is
//          its own; lanes one push delivered share a pair), and the slot of
//          every lane is kept as four 64-bit planes (bit r of plane b = bit b
//          of lane r's slot): a record sets its lanes in four ORs, whatever
//          their number, so the threads of a warp do not wait for the one
//          whose records hold the most lanes;
//   write  walks the roots eight at a time: a byte of each plane becomes eight
//          4-bit slots, a slot gives a lane's depth and parent with no branch,
//          and the CTA's threads store each root's row entries of consecutive
//          vertices, streaming past L2.
// No thread reads another's table, so there is no barrier and a warp's
// writes overlap another's loads.  A lane whose pair finds the table full
// reads its row in the write loop (more than 16 distinct deliverers).
//
// The bytes are 12 x 64 per vertex written and some 190 read in random sectors,
// but one vertex per thread with the planes shifted lane by lane cost 55
// instructions per (vertex, root) and was bound by issue and latency (scale 21:
// 490 us, DRAM at 47 %).
struct MsOutParams {
    const int32_t *depth;     // per-lane rows [n][R]
    const uint32_t *parent;
    const uint4 *rec;         // [n][kRecSlots]
    const uint32_t *rec_cnt;  // [n]
    const ull *seen;          // [n]
    const int64_t *off;       // the caller's CSR offsets (unreached encoding)
    const uint32_t *perm;     // caller id -> traversal id, or null
    const uint32_t *iperm;    // traversal id -> caller id, or null
    int64_t n;
    int R;                    // lane stride of the rows
    int lanes;                // roots in the group
    int32_t *depth_out;       // row of the group's first root
    int64_t *parent_out;
};

constexpr unsigned kMatSlots = 16;

// Adds `lanes` to the planes of slot k.
__device__ __forceinline__ void mat_set_slot(ull (&plane)[4], unsigned k, ull lanes)
{
#pragma unroll
    for (int b = 0; b < 4; ++b) { plane[b] |= ((k >> b) & 1u) ? lanes : 0ull; }
}

__device__ __forceinline__ uint32_t mat_rename(const MsOutParams &o, uint32_t provider)
{
    // (a provider id out of range would only come from a broken record; it is
    // passed through, not followed)
    return o.iperm && provider < o.n ? __ldg(&o.iperm[provider]) : provider;
}

// The table entries and planes of a vertex reached by lanes s: records x0, x1 and
// cnt are read already.  tab: the vertex's entry of slot 0, `stride` apart.
__device__ __forceinline__ void mat_fill(const MsOutParams &o, int64_t t, ull s, uint4 x0, uint4 x1,
                                         unsigned cnt, uint2 *tab, int stride, ull (&plane)[4],
                                         ull &row_lanes)
{
    const uint4 *rv = o.rec + t * kRecSlots;
    ull left = s;
    for (unsigned k0 = 0; k0 < cnt && left; k0 += 4) {
        uint4 x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x[j] = (k0 == 0 && j < 2) ? (j ? x1 : x0)
                                      : (k0 + j < cnt ? __ldcs(&rv[k0 + j]) : make_uint4(0, 0, 0, 0));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const ull mask = k0 + j < cnt ? (((ull)x[j].y << 32) | x[j].x) & left : 0ull;
            if (!mask) { continue; }
            left &= ~mask;
            const unsigned k = k0 + j;
            tab[k * stride] = make_uint2(x[j].w, mat_rename(o, x[j].z));
            mat_set_slot(plane, k, mask);
        }
    }
    // lanes past the records: their rows, four loads in flight; lanes
    // with the (depth, parent) pair of the previous one share its slot
    unsigned used = cnt;
    int32_t last_d = -2;
    uint32_t last_p = 0;
    unsigned last_k = kMatSlots;
    while (left) {
        int rr[4];
        int32_t dd[4];
        uint32_t pp[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            rr[j] = left ? __ffsll((long long)left) - 1 : -1;
            left &= left ? left - 1 : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            dd[j] = rr[j] >= 0 ? __ldcs(&o.depth[t * o.R + rr[j]]) : 0;
            pp[j] = rr[j] >= 0 ? __ldcs(&o.parent[t * o.R + rr[j]]) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (rr[j] < 0) { continue; }
            if (dd[j] != last_d || pp[j] != last_p) {
                last_d = dd[j];
                last_p = pp[j];
                last_k = kMatSlots;
                if (used < kMatSlots) {
                    last_k = used++;
                    tab[last_k * stride] = make_uint2((uint32_t)dd[j], mat_rename(o, pp[j]));
                }
            }
            const ull bit = 1ull << rr[j];
            if (last_k < kMatSlots) {
                mat_set_slot(plane, last_k, bit);
            } else {
                row_lanes |= bit;
            }
        }
    }
}

// Bits 0-7 of x to bits 0, 4, ... 28.
__device__ __forceinline__ uint32_t mat_spread(uint32_t x)
{
    x &= 0xFFu;
    x = (x | (x << 12)) & 0x000F000Fu;
    x = (x | (x << 6)) & 0x03030303u;
    return (x | (x << 3)) & 0x11111111u;
}

template <int V, int T>
__global__ void __launch_bounds__(T) ms_materialize_kernel(MsOutParams o)
{
    static_assert(V == 1 || V == 2, "rows are stored one or two entries at a time");
    extern __shared__ __align__(16) unsigned char mat_raw[];  // [kMatSlots][V][T] pairs
    constexpr int stride = V * T;
    uint2 *tab = reinterpret_cast<uint2 *>(mat_raw) + threadIdx.x;  // entry (k, i): [k * stride + i * T]
    const ull all = o.lanes >= 64 ? ~0ull : ((1ull << o.lanes) - 1);
    const long long tiles = (o.n + stride - 1) / stride;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t v = tile * stride + V * threadIdx.x;
        if (v >= o.n) { continue; }  // V == 2: n is even
        int64_t off[V + 1], t[V];
        ull s[V];
#pragma unroll
        for (int i = 0; i <= V; ++i) { off[i] = __ldg(&o.off[v + i]); }
#pragma unroll
        for (int i = 0; i < V; ++i) { t[i] = o.perm ? (int64_t)__ldg(&o.perm[v + i]) : v + i; }
#pragma unroll
        for (int i = 0; i < V; ++i) { s[i] = __ldcs(&o.seen[t[i]]) & all; }
        // the first two records are read together with the count (they lie
        // in the vertex's record block whatever the count says)
        uint4 x0[V], x1[V];
        unsigned cnt[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            cnt[i] = 0;
            x0[i] = x1[i] = make_uint4(0, 0, 0, 0);
            if (s[i]) {
                x0[i] = __ldcs(&o.rec[t[i] * kRecSlots]);
                x1[i] = __ldcs(&o.rec[t[i] * kRecSlots + 1]);
                cnt[i] = min(__ldcs(&o.rec_cnt[t[i]]), kRecSlots);
            }
        }
        ull plane[V][4], row_lanes[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            row_lanes[i] = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) { plane[i][b] = 0; }
            if (s[i]) {
                mat_fill(o, t[i], s[i], x0[i], x1[i], cnt[i], tab + i * T, stride, plane[i],
                         row_lanes[i]);
            }
        }
        int64_t unreached[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const int64_t deg = off[i + 1] - off[i];
            unreached[i] = deg != 0 ? -deg : -1;
        }
        int32_t *dp = o.depth_out + v;
        int64_t *pq = o.parent_out + v;
        for (int r0 = 0; r0 < o.lanes; r0 += 8) {
            uint32_t slots[V], got[V];
            uint32_t rows = 0;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                slots[i] = mat_spread((uint32_t)plane[i][0]) | (mat_spread((uint32_t)plane[i][1]) << 1) |
                           (mat_spread((uint32_t)plane[i][2]) << 2) |
                           (mat_spread((uint32_t)plane[i][3]) << 3);
                got[i] = (uint32_t)s[i] & 0xFFu;
                rows |= (uint32_t)row_lanes[i] & 0xFFu;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                int32_t d[V];
                int64_t par[V];
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const uint2 e = tab[((slots[i] >> (4 * j)) & 15u) * stride + i * T];
                    const bool has = (got[i] >> j) & 1u;
                    d[i] = has ? (int32_t)e.x : -1;
                    par[i] = has ? (int64_t)e.y : unreached[i];
                }
                if ((rows >> j) & 1u) {  // more pairs than slots: the lane's own row
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        if ((row_lanes[i] >> j) & 1ull) {
                            d[i] = __ldcs(&o.depth[t[i] * o.R + r0 + j]);
                            par[i] = (int64_t)mat_rename(o, __ldcs(&o.parent[t[i] * o.R + r0 + j]));
                        }
                    }
                }
                if (r0 + j < o.lanes) {
                    if constexpr (V == 2) {
                        __stcs(reinterpret_cast<int2 *>(dp), make_int2(d[0], d[1]));
                        __stcs(reinterpret_cast<longlong2 *>(pq), make_longlong2(par[0], par[1]));
                    } else {
                        __stcs(dp, d[0]);
                        __stcs(pq, par[0]);
                    }
                }
                dp += o.n;
                pq += o.n;
            }
#pragma unroll
            for (int i = 0; i < V; ++i) {
                s[i] >>= 8;
                row_lanes[i] >>= 8;
#pragma unroll
                for (int b = 0; b < 4; ++b) { plane[i][b] >>= 8; }
            }
        }
    }
}

__global__ void ms_long_chunks_kernel(const int64_t *off, int64_t n, int64_t long_arcs,
                                      uint32_t long_chunk, ull *chunks)
{
    ull c = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t rest = off[v + 1] - off[v] - long_arcs;
        if (rest > 0) { c += (ull)((rest + long_chunk - 1) / long_chunk); }
    }
    c = warp_sum(c);
    if (lane_id() == 0 && c) { atomicAdd(chunks, c); }
}

using MsRowsKernel = void (*)(MsOutParams);
struct MsRows {
    MsRowsKernel fn;
    int threads;
    size_t smem;
};

// Which variant writes the rows of a graph of n vertices.  Two vertices a thread
// where the rows' 16-byte stores are aligned and that still fills the device
// (scale 24 rows 3.68 -> 3.04 ms); on small graphs smaller blocks, so that more of
// them share the work.
MsRows ms_rows(int64_t n)
{
    const size_t entry = kMatSlots * sizeof(uint2);
    if (n < 148 * 256) { return {ms_materialize_kernel<1, 64>, 64, 64 * entry}; }
    if (n % 2 == 0 && n >= 148 * 3 * 512) { return {ms_materialize_kernel<2, 256>, 256, 512 * entry}; }
    return {ms_materialize_kernel<1, 256>, 256, 256 * entry};
}

using MsKernel = void (*)(MsParams);

int ms_grid_for(int64_t items)
{
    int64_t b = (items + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 32));
}

}  // namespace
}  // namespace bd

using namespace bd;

struct bd_msbfs {
    bd_graph *g = nullptr;
    int device = 0;
    int R = 64;          // lanes per group (= lane stride of the output rows)
    int groups = 1;      // result slices
    int max_roots = 64;
    bd_msbfs_opts opts{};
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    ull *seen = nullptr;         // [groups][n]: a group's final words mark its valid lanes
    ull *F[3] = {nullptr, nullptr, nullptr};
    uint32_t *qs[3] = {nullptr, nullptr, nullptr};
    uint32_t *ql[3] = {nullptr, nullptr, nullptr};
    ull *qlb[3] = {nullptr, nullptr, nullptr};
    int32_t *depth = nullptr;    // [groups][n][R]
    uint32_t *parent = nullptr;  // [groups][n][R]
    uint4 *drec = nullptr;       // [groups][n][kRecSlots]
    uint32_t *drec_cnt = nullptr;  // [groups][n]
    uint32_t *done = nullptr;      // [n/32], rewritten for each group
    MsCtrl *ctrl = nullptr;
    bd_step *rec = nullptr;
    int64_t *d_sources = nullptr;         // [max_roots]
    unsigned long long *d_counts = nullptr;  // [groups][128]
    int64_t cap_large = 0;
    int grid = 0;
    int block = 512;
    int count = 0;  // roots in the last run
    std::vector<int64_t> sources;  // roots of the last run
    bool ran = false;
    PolicyBlob *policy = nullptr;  // device copy, or null
    MinParentScratch min_scratch;  // opts.min_parent
    CheckScratch check;
    uint2 *dq = nullptr;  // chunks of long pull scans, or null: no list is that long
    cudaGraphExec_t graph = nullptr;
    int graph_count = -1;
    bool graph_ok = true;
    bool frontier_clean = false;  // F is all zero (kernels leave it so)
    MsCtrlHead last{};
    MsHostIo *io = nullptr;  // pinned, with its arrays behind it
    std::vector<unsigned long long> counts;
    // opts.materialize: every root's results, written by each run
    int32_t *out_depth = nullptr;   // [max_roots][n]
    int64_t *out_parent = nullptr;  // [max_roots][n]
    int mat_grid = 0;
    // otherwise: one root's results, extracted when they are read
    void *xbuf = nullptr;           // 8 n bytes
};

namespace bd {
namespace {

MsKernel ms_pick(int block)
{
    switch (block) {
        case 256: return msbfs_kernel<256, 4>;
        case 1024: return msbfs_kernel<1024, 1>;
        default: return msbfs_kernel<512, 2>;
    }
}

MsParams ms_params(bd_msbfs *b, int group, int count)
{
    MsParams p{};
    p.off = traversal_off(b->g);
    p.adj = traversal_adj(b->g);
    p.perm = b->g->d_perm;
    p.done = b->done;
    p.n = b->g->n;
    p.m = b->g->m;
    p.reach = b->seen + group * b->g->n;
    for (int i = 0; i < 3; ++i) {
        p.F[i] = b->F[i];
        p.qs[i] = b->qs[i];
        p.ql[i] = b->ql[i];
        p.qlb[i] = b->qlb[i];
    }
    const int64_t slice = b->g->n * (int64_t)b->R;
    p.depth = b->depth + group * slice;
    p.drec = b->drec + group * b->g->n * (int64_t)kRecSlots;
    p.drec_cnt = b->drec_cnt + group * b->g->n;
    p.parent = b->parent + group * slice;
    p.R = b->R;
    p.all = count >= 64 ? ~0ull : ((1ull << count) - 1);
    p.ctrl = b->ctrl;
    p.rec = b->rec;
    p.rec_cap = kMsRecCap;
    p.alpha = b->opts.alpha;
    p.large_deg = (uint32_t)b->opts.large_degree;
    p.chunk = (uint32_t)b->opts.chunk_edges;
    p.prefix = b->opts.pull_prefix;
    p.spin_limit = b->opts.spin_limit;
    p.expected_ctas = (unsigned)b->grid;
    p.force_dir = b->opts.force_dir;
    p.policy = b->policy;
    p.dq = b->dq;
    p.long_arcs = b->opts.heavy_degree;
    p.long_chunk = (uint32_t)b->opts.heavy_chunk;
    return p;
}

// Every lane of a finished group into its roots' output rows, and with
// opts.min_parent each root's smallest-parent tree on the caller's CSR.
bd_status ms_enqueue_materialize(bd_msbfs *b, int group, int count)
{
    const int64_t n = b->g->n;
    MsOutParams o{};
    const int64_t slice = n * (int64_t)b->R;
    o.depth = b->depth + group * slice;
    o.parent = b->parent + group * slice;
    o.rec = b->drec + group * n * (int64_t)kRecSlots;
    o.rec_cnt = b->drec_cnt + group * n;
    o.seen = b->seen + group * n;
    o.off = b->g->d_off;
    o.perm = b->g->d_perm;
    o.iperm = b->g->d_iperm;
    o.n = n;
    o.R = b->R;
    o.lanes = count;
    o.depth_out = b->out_depth + (int64_t)group * 64 * n;
    o.parent_out = b->out_parent + (int64_t)group * 64 * n;
    const MsRows rows = ms_rows(n);
    rows.fn<<<b->mat_grid, rows.threads, rows.smem, b->stream>>>(o);
    BD_CUDA(cudaGetLastError());
    if (b->opts.min_parent) {
        for (int r = 0; r < count; ++r) {
            const int64_t row = ((int64_t)group * 64 + r) * n;
            BD_CUDA(launch_min_parent(b->g, b->min_scratch, b->out_depth + row,
                                      b->out_parent + row, b->stream));
        }
    }
    return BD_OK;
}

// One group: clear, init, the
// persistent kernel, the per-lane counts (and with opts.materialize the
// roots' output rows).
bd_status ms_enqueue_group(bd_msbfs *b, int group, int count)
{
    const int64_t n = b->g->n;
    MsParams p = ms_params(b, group, count);
    unsigned long long *dst = b->d_counts + 128 * group;
    ms_clear_kernel<<<ms_grid_for(n), 256, 0, b->stream>>>(p, traversal_isolated(b->g), dst,
                                                              group > 0);
    BD_CUDA(cudaGetLastError());
    ms_init_kernel<<<1, 32, 0, b->stream>>>(p, b->d_sources + group * 64, count);
    BD_CUDA(cudaGetLastError());
    void *args[] = {&p};
    BD_CUDA(cudaLaunchCooperativeKernel((const void *)ms_pick(b->block), dim3(b->grid),
                                        dim3(b->block), args, 0, b->stream));
    ms_count_kernel<<<std::min(ms_grid_for(n), 148 * 8), 256, 0, b->stream>>>(
        p.reach, p.off, n, p.all, count, dst);
    BD_CUDA(cudaGetLastError());
    if (b->opts.materialize) { BD_TRY(ms_enqueue_materialize(b, group, count)); }
    return BD_OK;
}

bd_status ms_enqueue_all(bd_msbfs *b, int count)
{
    for (int gi = 0; gi * 64 < count; ++gi) {
        BD_TRY(ms_enqueue_group(b, gi, std::min(64, count - gi * 64)));
    }
    return BD_OK;
}

// Captures the groups of a `count`-root call into one CUDA graph (once per
// count); falls back to plain stream launches if capture is refused.
bd_status ms_launch(bd_msbfs *b, int count)
{
    // The kernels leave F zero; after a first use or an error, zero
    // them here (outside any captured graph).
    if (!b->frontier_clean) {
        const int64_t n = b->g->n;
        for (int i = 0; i < 3; ++i) {
            BD_CUDA(cudaMemsetAsync(b->F[i], 0, sizeof(ull) * n, b->stream));
        }
    }
    b->frontier_clean = false;  // until this call is known to have finished cleanly
    if (b->opts.use_graph && b->graph_ok) {
        if (b->graph_count != count) {
            if (b->graph) {
                cudaGraphExecDestroy(b->graph);
                b->graph = nullptr;
            }
            cudaGraph_t gr = nullptr;
            if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                bd_status st = ms_enqueue_all(b, count);
                cudaError_t e = cudaStreamEndCapture(b->stream, &gr);
                if (st == BD_OK && e == cudaSuccess &&
                    cudaGraphInstantiate(&b->graph, gr, 0) == cudaSuccess) {
                    b->graph_count = count;
                } else {
                    b->graph = nullptr;
                    b->graph_ok = false;
                }
                if (gr) { cudaGraphDestroy(gr); }
            } else {
                b->graph_ok = false;
            }
            cudaGetLastError();  // a refused capture leaves no sticky error
        }
        if (b->graph) {
            BD_CUDA(cudaGraphLaunch(b->graph, b->stream));
            return BD_OK;
        }
    }
    return ms_enqueue_all(b, count);
}

void ms_free(bd_msbfs *b)
{
    if (!b) { return; }
    cudaSetDevice(b->device);
    if (b->stream) { cudaStreamSynchronize(b->stream); }
    if (b->graph) { cudaGraphExecDestroy(b->graph); }
    cudaFree(b->seen);
    cudaFree(b->done);
    for (int i = 0; i < 3; ++i) {
        cudaFree(b->F[i]);
        cudaFree(b->qs[i]);
        cudaFree(b->ql[i]);
        cudaFree(b->qlb[i]);
    }
    cudaFree(b->depth);
    cudaFree(b->parent);
    cudaFree(b->drec);
    cudaFree(b->drec_cnt);
    cudaFree(b->ctrl);
    cudaFree(b->rec);
    cudaFree(b->d_sources);
    cudaFree(b->d_counts);
    if (b->io) { cudaFreeHost(b->io); }
    cudaFree(b->policy);
    cudaFree(b->dq);
    min_parent_free(&b->min_scratch);
    check_free(&b->check);
    cudaFree(b->out_depth);
    cudaFree(b->out_parent);
    cudaFree(b->xbuf);
    if (b->ev0) { cudaEventDestroy(b->ev0); }
    if (b->ev1) { cudaEventDestroy(b->ev1); }
    if (b->stream) { cudaStreamDestroy(b->stream); }
    delete b;
}

// Chunks of the arcs past opts.heavy_degree over all lists of the traversal CSR
// (counted in the handle's d_counts, which no run uses yet).
bd_status ms_long_chunks(bd_msbfs *b, unsigned long long *chunks)
{
    BD_CUDA(cudaMemsetAsync(b->d_counts, 0, sizeof(unsigned long long), b->stream));
    ms_long_chunks_kernel<<<ms_grid_for(b->g->n), 256, 0, b->stream>>>(
        traversal_off(b->g), b->g->n, b->opts.heavy_degree, (uint32_t)b->opts.heavy_chunk,
        b->d_counts);
    BD_CUDA(cudaGetLastError());
    BD_CUDA(cudaMemcpyAsync(chunks, b->d_counts, sizeof(*chunks), cudaMemcpyDeviceToHost,
                            b->stream));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    return BD_OK;
}

bd_status ms_check_root(bd_msbfs *b, int32_t root_index)
{
    if (!b->ran) { return BD_ERR_STATE; }
    if (root_index < 0 || root_index >= b->count) { return BD_ERR_RANGE; }
    return BD_OK;
}

// One root's depths or parents (caller ids, reference encoding) into a
// device buffer of n entries, queued on the handle's stream.
cudaError_t ms_extract_async(bd_msbfs *b, int32_t root_index, int32_t *d_depth, int64_t *d_parent)
{
    const int64_t n = b->g->n;
    const int group = root_index / 64, lane = root_index % 64;
    const int64_t slice = n * (int64_t)b->R;
    ms_extract_kernel<<<ms_grid_for(n), 256, 0, b->stream>>>(
        b->depth + group * slice, b->parent + group * slice, b->drec + group * n * (int64_t)kRecSlots,
        b->drec_cnt + group * n, b->seen + group * n, b->g->d_off, n, b->R, lane, b->g->d_perm,
        b->g->d_iperm, d_depth, d_parent);
    return cudaGetLastError();
}

// One root's depths or parents (caller ids, reference encoding) in device
// memory: its materialized row, or extracted into the handle's buffer.
bd_status ms_root_device(bd_msbfs *b, int32_t root_index, bool want_depth, const void **out)
{
    BD_TRY(ms_check_root(b, root_index));
    BD_CUDA(cudaSetDevice(b->device));
    const int64_t n = b->g->n;
    if (b->opts.materialize) {
        *out = want_depth ? (const void *)(b->out_depth + (int64_t)root_index * n)
                          : (const void *)(b->out_parent + (int64_t)root_index * n);
        return BD_OK;
    }
    BD_CUDA(ms_extract_async(b, root_index, want_depth ? static_cast<int32_t *>(b->xbuf) : nullptr,
                             want_depth ? nullptr : static_cast<int64_t *>(b->xbuf)));
    *out = b->xbuf;
    return BD_OK;
}

bd_status ms_extract(bd_msbfs *b, int32_t root_index, int32_t *depth, int64_t *parent)
{
    const void *src = nullptr;
    BD_TRY(ms_root_device(b, root_index, depth != nullptr, &src));
    const size_t bytes = depth ? sizeof(int32_t) * b->g->n : sizeof(int64_t) * b->g->n;
    BD_CUDA(cudaMemcpyAsync(depth ? (void *)depth : (void *)parent, src, bytes,
                            cudaMemcpyDeviceToHost, b->stream));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    return BD_OK;
}

}  // namespace
}  // namespace bd

extern "C" {

void bd_msbfs_default_opts(bd_msbfs_opts *o)
{
    if (!o) { return; }
    memset(o, 0, sizeof(*o));
    o->alpha = 4;
    o->force_dir = -1;
    o->use_graph = 1;
}

bd_status bd_msbfs_create(bd_graph *g, int32_t max_roots, const bd_msbfs_opts *opts,
                          bd_msbfs **out)
{
    if (!g || !out || max_roots < 1 || max_roots > 65536) { return BD_ERR_INVALID; }
    bd_msbfs_opts o;
    bd_msbfs_default_opts(&o);
    if (opts) { o = *opts; }
    if (o.alpha <= 0 || o.force_dir < -1 || o.force_dir > 1) { return BD_ERR_INVALID; }
    if (o.block_size == 0) { o.block_size = 512; }
    if (o.block_size != 256 && o.block_size != 512 && o.block_size != 1024) { return BD_ERR_INVALID; }
    if (o.large_degree <= 0) { o.large_degree = 32; }
    if (o.large_degree > (1 << 20)) { return BD_ERR_INVALID; }
    if (o.chunk_edges <= 0) { o.chunk_edges = 256; }
    if (o.pull_prefix <= 0) { o.pull_prefix = 16; }
    if (o.spin_limit <= 0) { o.spin_limit = kMsDefaultSpin; }
    if (o.materialize < 0 || o.materialize > 1 || o.min_parent < 0 || o.min_parent > 1) {
        return BD_ERR_INVALID;
    }
    if (o.min_parent) { o.materialize = 1; }
    if (g->n > (int64_t)UINT32_MAX) { return BD_ERR_LIMIT; }
    BD_TRY(ensure_device());
    auto *b = new bd_msbfs();
    b->g = g;
    b->device = current_device();
    b->max_roots = max_roots;
    b->R = std::min(64, (int)max_roots);
    b->groups = (max_roots + 63) / 64;
    b->opts = o;
    b->block = o.block_size;
    const int64_t n = g->n;
    b->cap_large = std::min<int64_t>(n, g->arcs / o.large_degree + 1);
    auto fail = [&](bd_status st) { ms_free(b); return st; };
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess) {
        return fail(BD_ERR_CUDA);
    }
    const size_t slots = (size_t)n * b->R * b->groups;
    bool ok = cudaMalloc(&b->seen, sizeof(ull) * n * b->groups) == cudaSuccess &&
              cudaMalloc(&b->done, sizeof(uint32_t) * ((n + 31) / 32)) == cudaSuccess &&
              cudaMalloc(&b->depth, sizeof(int32_t) * slots) == cudaSuccess &&
              cudaMalloc(&b->parent, sizeof(uint32_t) * slots) == cudaSuccess &&
              cudaMalloc(&b->drec, sizeof(uint4) * (size_t)n * kRecSlots * b->groups) == cudaSuccess &&
              cudaMalloc(&b->drec_cnt, sizeof(uint32_t) * (size_t)n * b->groups) == cudaSuccess &&
              cudaMalloc(&b->ctrl, sizeof(MsCtrl)) == cudaSuccess &&
              cudaMalloc(&b->rec, sizeof(bd_step) * kMsRecCap) == cudaSuccess &&
              cudaMalloc(&b->d_sources, sizeof(int64_t) * 64 * b->groups) == cudaSuccess &&
              cudaMalloc(&b->d_counts, sizeof(unsigned long long) * 128 * b->groups) == cudaSuccess;
    ok = ok &&
         (!o.min_parent || min_parent_alloc(g, &b->min_scratch, b->stream) == cudaSuccess);
    for (int i = 0; i < 3 && ok; ++i) {
        ok = cudaMalloc(&b->F[i], sizeof(ull) * n) == cudaSuccess &&
             cudaMalloc(&b->qs[i], sizeof(uint32_t) * n) == cudaSuccess &&
             cudaMalloc(&b->ql[i], sizeof(uint32_t) * b->cap_large) == cudaSuccess &&
             cudaMalloc(&b->qlb[i], sizeof(ull) * b->cap_large) == cudaSuccess;
    }
    if (ok && o.materialize) {
        const size_t rows = (size_t)n * (size_t)max_roots;
        ok = cudaMalloc(&b->out_depth, sizeof(int32_t) * rows) == cudaSuccess &&
             cudaMalloc(&b->out_parent, sizeof(int64_t) * rows) == cudaSuccess;
    } else if (ok) {
        ok = cudaMalloc(&b->xbuf, sizeof(int64_t) * n) == cudaSuccess;
    }
    if (ok) {
        void *io = nullptr;
        ok = cudaHostAlloc(&io, sizeof(MsHostIo) + (size_t)b->groups * (64 * sizeof(int64_t) + 128 * sizeof(ull)),
                           cudaHostAllocDefault) == cudaSuccess;
        if (ok) {
            b->io = static_cast<MsHostIo *>(io);
            b->io->sources = reinterpret_cast<int64_t *>(b->io + 1);
            b->io->counts = reinterpret_cast<ull *>(b->io->sources + 64 * b->groups);
        }
    }
    if (!ok) { return fail(BD_ERR_OOM); }
    if (o.materialize) {
        int per_sm = 0, sms = 0;
        const MsRows rows = ms_rows(n);
        if (cudaFuncSetAttribute((const void *)rows.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)rows.smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)rows.fn, rows.threads,
                                                          rows.smem) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device) != cudaSuccess ||
            per_sm < 1) {
            return fail(BD_ERR_CUDA);
        }
        b->mat_grid = per_sm * sms;
    }
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)ms_pick(b->block),
                                                      b->block, 0) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device) != cudaSuccess ||
        per_sm < 1) {
        return fail(BD_ERR_CUDA);
    }
    b->grid = per_sm * sms;
    // Where a pull scan leaves a list to all warps (0 = this rule).  A warp takes
    // a word of 32 vertices, so up to 32 x heavy_degree arcs one after another,
    // to be held against the arcs an average warp scans in a full pull (arcs /
    // warps): a word may take a good third of that where the scans are bound by
    // latency, the whole of it on graphs far beyond L2, where leaving a list
    // early costs re-reads.  Traversal ms by heavy_degree, hub layout, 64 roots
    // (scale 16) and sums over four batches:
    //   scale 16 (rule 32)    32: 0.14   64: 0.15   256: 0.28   4096: 0.73
    //   scale 20 (rule 83)    64: 1.74  256: 1.83   512: 1.92   1024: 2.19
    //   scale 21 (rule 167)  128: 2.77  256: 2.65   512: 2.79   1024: 2.96
    //   scale 22 (rule 337)  128: 5.48  256: 5.46   512: 5.47   1024: 5.67
    //   scale 23 (rule 681)  256: 9.12  512: 9.07  1024: 9.17   4096: 9.42
    //   scale 24 (rule 3430) 512: 13.60 1024: 13.44 2048: 13.52 4096: 13.57
    // (from scale 22 on the minimum is flat, so the step of the rule between 23 and
    // 24, at 65536 arcs a warp, costs and gains 1 %).
    // Lists up to 1024 arcs in a numbering that does not put the hubs together are
    // not left at all: a word then holds one or two of them, which take less time
    // than the barrier.  Four batches, none left and the rule above it: degree
    // order, longest list 801 0.383 and 0.408 ms, 943 0.363 and 0.353, 1002 0.361 and
    // 0.383; longer lists 1168 0.426 and 0.378, 1326 0.466 and 0.404; file order 1002
    // 0.420 and 0.400, 1326 0.557 and 0.441.
    const int64_t per_warp = g->arcs / ((int64_t)b->grid * (b->block / 32));
    if (b->opts.heavy_degree <= 0) {
        b->opts.heavy_degree = (int32_t)std::min<int64_t>(
            4096, std::max<int64_t>(32, per_warp < 65536 ? per_warp / 80 : per_warp / 32));
        if (!g->d_perm && g->max_degree <= 1024) { b->opts.heavy_degree = 1024; }
    }
    if (b->opts.heavy_chunk <= 0) { b->opts.heavy_chunk = dev::long_chunk(b->opts.heavy_degree); }
    b->opts.pull_prefix = std::min(b->opts.pull_prefix, b->opts.heavy_degree);
    // room for every chunk a pull step can leave to ms_pull_long
    {
        ull chunks = 0;
        const bd_status st = ms_long_chunks(b, &chunks);
        if (st != BD_OK) { return fail(st); }
        if (chunks && cudaMalloc(&b->dq, sizeof(uint2) * chunks) != cudaSuccess) {
            return fail(BD_ERR_OOM);
        }
    }
    *out = b;
    return BD_OK;
}

bd_status bd_msbfs_run(bd_msbfs *b, const int64_t *sources, int32_t count, bd_run_stats *stats)
{
    if (!b || !sources || count < 1 || count > b->max_roots) { return BD_ERR_INVALID; }
    for (int i = 0; i < count; ++i) {
        if (sources[i] < 0 || sources[i] >= b->g->n) { return BD_ERR_RANGE; }
    }
    BD_CUDA(cudaSetDevice(b->device));
    // group g's sources start at d_sources + 64 g
    std::copy(sources, sources + count, b->io->sources);
    BD_CUDA(cudaMemcpyAsync(b->d_sources, b->io->sources, sizeof(int64_t) * count,
                            cudaMemcpyHostToDevice, b->stream));
    BD_CUDA(cudaEventRecord(b->ev0, b->stream));
    BD_TRY(ms_launch(b, count));
    BD_CUDA(cudaEventRecord(b->ev1, b->stream));
    const int used = (count + 63) / 64;
    BD_CUDA(cudaMemcpyAsync(b->io->counts, b->d_counts, sizeof(ull) * 128 * used,
                            cudaMemcpyDeviceToHost, b->stream));
    BD_CUDA(cudaMemcpyAsync(&b->io->head, b->ctrl, sizeof(MsCtrlHead), cudaMemcpyDeviceToHost,
                            b->stream));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    b->counts.assign(b->io->counts, b->io->counts + 128 * used);
    b->last = b->io->head;
    b->count = count;
    b->sources.assign(sources, sources + count);
    b->ran = true;
    b->frontier_clean = b->last.error == 0;
    if (b->last.error) { return (bd_status)b->last.error; }
    if (stats) {
        float ms = 0.f;
        BD_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
        stats->ms = ms;
        stats->num_steps = b->last.st.step;
        int64_t edges = 0, reached = 0;
        for (int i = 0; i < count; ++i) {
            const size_t base = (size_t)(i / 64) * 128;
            edges += (int64_t)(b->counts[base + 64 + i % 64] / 2);
            reached += (int64_t)b->counts[base + i % 64];
        }
        stats->traversed_edges = edges;
        stats->reached = reached;
        stats->top_down_steps = b->last.st.push_steps;
        stats->bottom_up_steps = b->last.st.pull_steps;
    }
    return BD_OK;
}

bd_status bd_msbfs_get_depths(bd_msbfs *b, int32_t root_index, int32_t *depth)
{
    if (!b || !depth) { return BD_ERR_INVALID; }
    return ms_extract(b, root_index, depth, nullptr);
}

bd_status bd_msbfs_get_parents(bd_msbfs *b, int32_t root_index, int64_t *parent)
{
    if (!b || !parent) { return BD_ERR_INVALID; }
    return ms_extract(b, root_index, nullptr, parent);
}

// hybrid_bfs::check of one root's parents, extracted and checked in HBM
// (bd_check.cu).
bd_status bd_msbfs_check(bd_msbfs *b, int32_t root_index, int32_t *ok)
{
    if (!b || !ok) { return BD_ERR_INVALID; }
    const void *parent = nullptr;
    BD_TRY(ms_root_device(b, root_index, false, &parent));
    BD_CUDA(cudaStreamSynchronize(b->stream));
    return check_parents_device(b->g, b->sources[root_index], static_cast<const int64_t *>(parent),
                                ok, nullptr, &b->check);
}

// Borrowed device pointers to one root's materialized results.
bd_status bd_msbfs_device_results(bd_msbfs *b, int32_t root_index, const int32_t **depth,
                                  const int64_t **parent)
{
    if (!b) { return BD_ERR_INVALID; }
    if (!b->opts.materialize) { return BD_ERR_STATE; }
    const void *d = nullptr, *p = nullptr;
    BD_TRY(ms_root_device(b, root_index, true, &d));
    BD_TRY(ms_root_device(b, root_index, false, &p));
    if (depth) { *depth = static_cast<const int32_t *>(d); }
    if (parent) { *parent = static_cast<const int64_t *>(p); }
    return BD_OK;
}

bd_status bd_msbfs_count_traversed_edges(bd_msbfs *b, int32_t root_index, int64_t *edges,
                                         int64_t *reached)
{
    if (!b) { return BD_ERR_INVALID; }
    BD_TRY(ms_check_root(b, root_index));
    const size_t base = (size_t)(root_index / 64) * 128;
    if (edges) { *edges = (int64_t)(b->counts[base + 64 + root_index % 64] / 2); }
    if (reached) { *reached = (int64_t)b->counts[base + root_index % 64]; }
    return BD_OK;
}

bd_status bd_msbfs_counts(bd_msbfs *b, int64_t *edges, int64_t *reached)
{
    if (!b) { return BD_ERR_INVALID; }
    if (!b->ran) { return BD_ERR_STATE; }
    for (int32_t i = 0; i < b->count; ++i) {
        BD_TRY(bd_msbfs_count_traversed_edges(b, i, edges ? edges + i : nullptr,
                                              reached ? reached + i : nullptr));
    }
    return BD_OK;
}

bd_status bd_msbfs_get_steps(bd_msbfs *b, bd_step *steps, int64_t capacity, int64_t *count)
{
    if (!b || !count || capacity < 0 || (!steps && capacity)) { return BD_ERR_INVALID; }
    if (!b->ran) { return BD_ERR_STATE; }
    const int64_t have = std::min<int64_t>(b->last.st.step, kMsRecCap);
    const int64_t take = std::min(have, capacity);
    if (take) {
        BD_CUDA(cudaSetDevice(b->device));
        BD_CUDA(cudaMemcpy(steps, b->rec, sizeof(bd_step) * take, cudaMemcpyDeviceToHost));
    }
    *count = have;
    return BD_OK;
}

bd_status bd_msbfs_set_policy(bd_msbfs *b, const float *params, const float *mean,
                              const float *inv_std, const float *lo, const float *hi, float margin)
{
    if (!b) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(b->device));
    if (!params || isinf(margin)) {  // +inf margin: the rule decides, nothing is evaluated
        cudaFree(b->policy);
        b->policy = nullptr;
        b->graph_count = -1;  // captured launches hold the old pointer
        return BD_OK;
    }
    PolicyBlob blob;
    BD_TRY(policy_blob(params, mean, inv_std, lo, hi, margin, &blob));
    if (!b->policy) {
        BD_CUDA(cudaMalloc(&b->policy, sizeof(PolicyBlob)));
        b->graph_count = -1;
    }
    BD_CUDA(cudaMemcpy(b->policy, &blob, sizeof(PolicyBlob), cudaMemcpyHostToDevice));
    return BD_OK;
}

bd_status bd_msbfs_destroy(bd_msbfs *b)
{
    if (!b) { return BD_ERR_INVALID; }
    ms_free(b);
    return BD_OK;
}

}  // extern "C"
