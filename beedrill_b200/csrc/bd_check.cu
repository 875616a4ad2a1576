// bd_check.cu -- hybrid_bfs::check (hybrid_bfs.cc:281-379) on the device.
//
// The reference validates a parent array against the depths of its own
// serial queue BFS: a vertex that both reached must have its parent among
// its neighbours exactly one level up (the source is its own parent at
// depth 0), and the two must agree on which vertices were reached.  The
// verdict depends only on the BFS depths, which do not depend on the order
// of the search, so a parallel search gives the same verdict:
//
//   check_search         level-synchronous search in one cooperative launch: a
//                        queue of vertices whose arcs are claimed by atomicCAS,
//                        or, on graphs known to be symmetric, a sweep in which
//                        each unreached vertex looks for a neighbour of the last
//                        level, whichever has fewer arcs to read.  It shares no
//                        code with the traversal kernels, so it is an independent
//                        witness of the depths they claim.
//   check_verify         the reference's per-vertex test, all vertices at once, in
//                        the same launch.  A failing vertex raises a shared
//                        maximum of complements, so the lowest failing vertex --
//                        the one the reference's ascending loop stops at and
//                        logs -- is reported.
//
// At scale 20 the search took 2.9 ms as one launch per level, one warp per queued
// vertex (a hub's list is 10^5 arcs) and one queue atomic per vertex, the test
// 0.34 ms, and the call 11 to 29 ms with its device allocations; a handle that
// checks its own results keeps them instead (CheckScratch).
//
// Device memory: 12 bytes per vertex (depths and two queues) and 24 bytes per
// 1024 arcs.
//
// components::check (components.cc:155-200) runs a serial BFS from one
// vertex of each distinct label, requires every neighbour it meets to carry
// that label, and requires every vertex to be visited.  That verdict is:
// every arc joins two vertices of the same label, and each component holds
// the representative of its label (so no label spans two components).
// Here the representatives come from a radix sort of (label, vertex); a
// multi-source run of check_search from all of them marks what they
// reach; check_components_kernel tests both conditions for every vertex.
// Device memory: 36 bytes per vertex plus the sort's scratch.
#include <cub/cub.cuh>

#include <algorithm>

#include "bd_device_util.cuh"
#include "bd_internal.h"

namespace bd {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

int grid_for_warps(int64_t warps)
{
    int64_t b = (warps + kWarps - 1) / kWarps;
    if (b < 1) { b = 1; }
    if (b > 148 * 64) { b = 148 * 64; }  // warp-stride beyond this
    return (int)b;
}

constexpr int kSearch = 512;            // threads per CTA of the search
constexpr int kSearchWarps = kSearch / 32;
constexpr int64_t kLong = 1024;         // arcs above which a queued list is cut into chunks
constexpr int64_t kBlockList = 2048;    // arcs above which a whole CTA looks through a list
constexpr int kShift = 38;              // long-queue counter: vertices << 38 | chunks
constexpr unsigned long long kLowMask = (1ull << kShift) - 1;
using ull = unsigned long long;
using namespace dev;

// A frontier's counters: level k uses slot k % 3; slot (k + 2) % 3 is cleared
// while level k runs.
struct CheckLevel {
    ull small;   // vertices of at most kLong arcs
    ull packed;  // the others and their chunks
    ull degsum;
};

}  // namespace

struct CheckCtl {
    ull bar;        // barrier arrivals
    ull bad;        // complement of the lowest failing vertex, or 0
    int error, pad;
    CheckLevel level[3];
};

namespace {

struct CheckParams {
    const int64_t *off;
    const uint32_t *adj;
    int64_t n, arcs;
    bool symmetric;
    long long polls;  // bound of a barrier's wait
    int32_t *depth;
    uint32_t *qs[2], *ql[2];
    ull *cb[2];  // first chunk of each entry of ql
    CheckCtl *ctl;
};

// Grid barrier b; false after a timeout.  All threads.
__device__ bool check_barrier(const CheckParams &p, long long b, int &flag)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        red_release_add64(&p.ctl->bar, 1ull);
        const ull target = (ull)(b + 1) * gridDim.x;
        long long it = 0;
        while (ld_acquire64(&p.ctl->bar) < target && ++it <= p.polls) { __nanosleep(32); }
        if (it > p.polls) { atomicExch(&p.ctl->error, (int)BD_ERR_TIMEOUT); }
        flag = __ldcg(&p.ctl->error);
    }
    __syncthreads();
    return flag == 0;
}

// Warp-collective: vertex v of degree deg of each lane with `has` joins frontier
// `slot` in queues `q`; one atomic per warp and kind.
__device__ __forceinline__ void check_append(const CheckParams &p, int slot, int q, bool has,
                                             uint32_t v, int64_t deg, ull &degsum)
{
    CheckLevel &lv = p.ctl->level[slot];
    const bool big = has && deg > kLong;
    const unsigned sm = __ballot_sync(kFullMask, has && !big), lm = __ballot_sync(kFullMask, big);
    if (has) { degsum += (ull)deg; }
    if (sm) {
        ull at = 0;
        if (lane_id() == 0) { at = atomicAdd(&lv.small, (ull)__popc(sm)); }
        at = __shfl_sync(kFullMask, at, 0);
        if (has && !big) { p.qs[q][at + __popc(sm & lanemask_lt())] = v; }
    }
    if (lm) {
        const ull ch = big ? (ull)((deg + kLong - 1) / kLong) : 0ull;
        const ull incl = warp_incl_scan(ch);
        ull old = 0;
        if (lane_id() == 31) { old = atomicAdd(&lv.packed, ((ull)__popc(lm) << kShift) | incl); }
        old = __shfl_sync(kFullMask, old, 31);
        if (big) {
            const ull at = (old >> kShift) + __popc(lm & lanemask_lt());
            p.ql[q][at] = v;
            p.cb[q][at] = (old & kLowMask) + incl - ch;
        }
    }
}

// Arc k of a lane (valid if `in`): claims its head for the next level.
__device__ __forceinline__ void check_claim(const CheckParams &p, int slot, int q, int32_t next,
                                            bool in, int64_t k, ull &degsum)
{
    const uint32_t v = in ? __ldg(&p.adj[k]) : 0u;
    const bool won = in && __ldcg(&p.depth[v]) == -1 && atomicCAS(&p.depth[v], -1, next) == -1;
    if (__any_sync(kFullMask, won)) {
        check_append(p, slot, q, won, v, won ? __ldg(&p.off[v + 1]) - __ldg(&p.off[v]) : 0, degsum);
    }
}

struct CheckScratchWarp {
    int32_t incl[32];
    int64_t beg[32];
};

// Levels of the search from the frontier in slot 0 / queues 0.  All CTAs.
__device__ void check_search(const CheckParams &p, CheckScratchWarp &ws, long long &barrier,
                             int &flag)
{
    const int lane = lane_id();
    // consecutive ranks on different CTAs, as the traversals deal a narrow level
    const int64_t gw = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const int64_t nw = (int64_t)gridDim.x * kSearchWarps;
    int64_t left = p.arcs;  // arcs of vertices not reached yet
    for (int32_t level = 0;; ++level) {
        const CheckLevel &lv = p.ctl->level[level % 3];
        const int64_t small = (int64_t)__ldcg(&lv.small), degsum = (int64_t)__ldcg(&lv.degsum);
        const ull packed = __ldcg(&lv.packed);
        const int64_t large = (int64_t)(packed >> kShift), chunks = (int64_t)(packed & kLowMask);
        if (small + large == 0) { return; }
        left -= degsum;
        const int cur = level & 1, q = cur ^ 1, slot = (level + 1) % 3;
        ull found = 0;
        if (p.symmetric && degsum * 4 > left) {
            // every unreached vertex looks for a neighbour of this level: its
            // first 8 arcs by its lane, the rest by the warp
            for (int64_t w = gw; w * 32 < p.n; w += nw) {
                const int64_t v = w * 32 + lane;
                int64_t b = 0, e = 0;
                if (v < p.n && __ldcg(&p.depth[v]) == -1) {
                    b = __ldg(&p.off[v]);
                    e = __ldg(&p.off[v + 1]);
                }
                bool hit = false;
                for (int64_t k = b; k < min(e, b + 8) && !hit; k += 4) {
                    uint32_t u[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) { u[j] = k + j < e ? __ldg(&p.adj[k + j]) : 0u; }
#pragma unroll
                    for (int j = 0; j < 4; ++j) { hit |= k + j < e && __ldcg(&p.depth[u[j]]) == level; }
                }
                unsigned todo = __ballot_sync(kFullMask, !hit && e - b > 8);
                while (todo) {
                    const int o = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int64_t ob = __shfl_sync(kFullMask, b, o) + 8, oe = __shfl_sync(kFullMask, e, o);
                    bool any = false;
                    for (int64_t base = ob; base < oe && !any; base += 128) {
                        bool mine = false;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int64_t k = base + 32 * j + lane;
                            mine |= k < oe && __ldcg(&p.depth[__ldg(&p.adj[min(k, oe - 1)])]) == level;
                        }
                        any = __any_sync(kFullMask, mine);
                    }
                    if (lane == o) { hit = any; }
                }
                if (hit) { p.depth[v] = level + 1; }
                check_append(p, slot, q, hit, (uint32_t)v, e - b, found);
            }
        } else {
            for (int64_t c = gw; c < chunks; c += nw) {
                int64_t lo = 0, hi = large - 1;  // last entry that starts at or before chunk c
                while (lo < hi) {
                    const int64_t mid = (lo + hi + 1) >> 1;
                    if ((int64_t)__ldcg(&p.cb[cur][mid]) <= c) { lo = mid; } else { hi = mid - 1; }
                }
                const uint32_t u = __ldcg(&p.ql[cur][lo]);
                const int64_t b = __ldg(&p.off[u]) + (c - (int64_t)__ldcg(&p.cb[cur][lo])) * kLong;
                const int64_t e = min(__ldg(&p.off[u + 1]), b + kLong);
                for (int64_t base = b; base < e; base += 32) {
                    check_claim(p, slot, q, level + 1, base + lane < e, base + lane, found);
                }
            }
            // short lists, up to 32 vertices a warp, their arcs laid end to end.  A
            // frontier of few vertices is spread thinner: with 32 vertices a warp it
            // was one warp's work, a chain of a thousand claims (check at scale 14
            // 0.66 ms, now 0.15; 16: 0.56 -> 0.17; 20: 0.52 -> 0.27)
            const int group = split_group(small, average(degsum, small + large), nw);
            for (int64_t g = gw; g << group < small; g += nw) {
                const int64_t i = (g << group) + lane;
                int64_t beg = 0;
                int32_t len = 0;
                if (lane >> group == 0 && i < small) {
                    const uint32_t u = __ldcg(&p.qs[cur][i]);
                    beg = __ldg(&p.off[u]);
                    len = (int32_t)(__ldg(&p.off[u + 1]) - beg);
                }
                const int32_t incl = warp_incl_scan(len);
                const int32_t total = __shfl_sync(kFullMask, incl, 31);
                ws.incl[lane] = incl;
                ws.beg[lane] = beg;
                __syncwarp();
                for (int32_t e = lane; e - lane < total; e += 32) {
                    int at = 0;  // lists that end at or before arc e
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) {
                        if (ws.incl[at + d - 1] <= e) { at += d; }
                    }
                    const int64_t k = ws.beg[at] + (e - (at ? ws.incl[at - 1] : 0));
                    check_claim(p, slot, q, level + 1, e < total, k, found);
                }
                __syncwarp();
            }
        }
        found = warp_sum(found);
        if (lane == 0 && found) { atomicAdd(&p.ctl->level[slot].degsum, found); }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            p.ctl->level[(level + 2) % 3] = CheckLevel{0, 0, 0};
        }
        if (!check_barrier(p, barrier++, flag)) { return; }
    }
}

// hybrid_bfs::check's test of every vertex (hybrid_bfs.cc:331-371).  A parent one
// level up must be among the vertex's neighbours: 16 arcs are looked through by the
// vertex's lane, lists of up to kBlockList arcs by its warp, longer ones by the
// CTA.  On a symmetric graph the shorter of the two lists (the vertex's and its
// parent's) will do.
__device__ void check_verify(const CheckParams &p, int64_t source, const int64_t *parent,
                             int *listed, uint32_t *list_vertex, uint32_t *list_parent)
{
    const int lane = lane_id();
    for (int64_t base = blockIdx.x * (int64_t)kSearch; base < p.n; base += (int64_t)gridDim.x * kSearch) {
        const int64_t u = base + threadIdx.x;
        bool bad = false, look = false;
        int64_t b = 0, e = 0;
        uint32_t target = 0, par = 0;
        if (u < p.n) {
            const int32_t d = __ldcg(&p.depth[u]);
            const int64_t q = __ldg(&parent[u]);
            if (d < 0 || q < 0) {
                bad = (d < 0) != (q < 0);
            } else if (u == source) {
                bad = !(q == u && d == 0);
            } else if (q >= p.n || __ldcg(&p.depth[q]) != d - 1) {
                bad = true;  // no neighbour, or a neighbour of another level
            } else {
                look = true;
                par = target = (uint32_t)q;
                b = __ldg(&p.off[u]);
                e = __ldg(&p.off[u + 1]);
                if (p.symmetric && e - b > 16) {
                    const int64_t pb = __ldg(&p.off[q]), pe = __ldg(&p.off[q + 1]);
                    if (pe - pb < e - b) {
                        b = pb;
                        e = pe;
                        target = (uint32_t)u;
                    }
                }
            }
        }
        const int64_t end = min(e, b + 16);
        for (int64_t k = b; k < end && look; k += 4) {
            uint32_t x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { x[j] = __ldg(&p.adj[min(k + j, e - 1)]); }
            look = x[0] != target && x[1] != target && x[2] != target && x[3] != target;
        }
        bad |= look && end == e;
        const bool more = look && end < e;
        if (more && e - b > kBlockList) {
            const int at = atomicAdd(listed, 1);
            list_vertex[at] = (uint32_t)u;
            list_parent[at] = par;
        }
        unsigned todo = __ballot_sync(kFullMask, more && e - b <= kBlockList);
        while (todo) {
            const int o = __ffs(todo) - 1;
            todo &= todo - 1;
            const int64_t ob = __shfl_sync(kFullMask, end, o), oe = __shfl_sync(kFullMask, e, o);
            const uint32_t t = __shfl_sync(kFullMask, target, o);
            bool any = false;
            for (int64_t kb = ob; kb < oe && !any; kb += 128) {
                bool mine = false;
#pragma unroll
                for (int j = 0; j < 4; ++j) { mine |= __ldg(&p.adj[min(kb + 32 * j + lane, oe - 1)]) == t; }
                any = __any_sync(kFullMask, mine);
            }
            if (lane == o) { bad = !any; }
        }
        if (bad) { atomicMax(&p.ctl->bad, ~(ull)u); }
        __syncthreads();
        const int count = *listed;
        for (int i = 0; i < count; ++i) {
            const uint32_t v = list_vertex[i], q = list_parent[i];
            int64_t lb = __ldg(&p.off[v]), le = __ldg(&p.off[v + 1]);
            uint32_t t = q;
            const int64_t pb = __ldg(&p.off[q]), pe = __ldg(&p.off[q + 1]);
            if (p.symmetric && pe - pb < le - lb) {
                lb = pb;
                le = pe;
                t = v;
            }
            bool any = false;
            for (int64_t kb = lb; kb < le && !any; kb += 4 * kSearch) {
                bool mine = false;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    mine |= __ldg(&p.adj[min(kb + kSearch * j + (int64_t)threadIdx.x, le - 1)]) == t;
                }
                any = __syncthreads_or(mine);
            }
            if (threadIdx.x == 0 && !any) { atomicMax(&p.ctl->bad, ~(ull)v); }
        }
        __syncthreads();
        if (threadIdx.x == 0) { *listed = 0; }
        __syncthreads();
    }
}

// The search alone (source < 0: the frontier in slot 0 is given), or from one
// source with the test of a parent array behind it.
__global__ void __launch_bounds__(kSearch, 2) check_search_kernel(const CheckParams p, int64_t source,
                                                                  const int64_t *parent)
{
    __shared__ CheckScratchWarp scratch[kSearchWarps];
    __shared__ uint32_t list_vertex[kSearch], list_parent[kSearch];
    __shared__ int listed, flag;
    if (threadIdx.x == 0) { listed = 0; }
    long long barrier = 0;
    if (source >= 0) {
        const int64_t t = blockIdx.x * (int64_t)kSearch + threadIdx.x;
        for (int64_t v = t; v < p.n; v += (int64_t)gridDim.x * kSearch) {
            p.depth[v] = v == source ? 0 : -1;
        }
        if (blockIdx.x == 0 && threadIdx.x < 32) {
            const bool one = threadIdx.x == 0;
            ull degsum = 0;
            check_append(p, 0, 0, one, (uint32_t)source, p.off[source + 1] - p.off[source], degsum);
            if (one) { p.ctl->level[0].degsum = degsum; }
        }
        if (!check_barrier(p, barrier++, flag)) { return; }
    }
    check_search(p, scratch[threadIdx.x >> 5], barrier, flag);
    __syncthreads();
    if (parent && __ldcg(&p.ctl->error) == 0) {
        check_verify(p, source, parent, &listed, list_vertex, list_parent);
    }
}

__global__ void iota_kernel(uint32_t *v, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        v[i] = (uint32_t)i;
    }
}

// The first vertex of each run of equal labels in sorted order becomes a
// source: depth 0, queued in slot 0.
__global__ void label_sources_kernel(const CheckParams p, const int64_t *sorted_label,
                                     const uint32_t *sorted_vertex)
{
    ull degsum = 0;
    for (int64_t i0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane_id(); i0 < p.n;
         i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + lane_id();
        const bool has = i < p.n && (i == 0 || sorted_label[i] != sorted_label[i - 1]);
        const uint32_t v = has ? sorted_vertex[i] : 0u;
        if (has) { p.depth[v] = 0; }
        check_append(p, 0, 0, has, v, has ? p.off[v + 1] - p.off[v] : 0, degsum);
    }
    degsum = warp_sum(degsum);
    if (lane_id() == 0 && degsum) { atomicAdd(&p.ctl->level[0].degsum, degsum); }
}

__global__ void __launch_bounds__(kThreads) check_components_kernel(
    const int64_t *off, const uint32_t *adj, int64_t n, const int32_t *depth,
    const int64_t *label, unsigned long long *bad_complement)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * kWarps;
    for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; u < n; u += warps) {
        bool bad = depth[u] < 0;
        const int64_t mine = label[u], e = off[u + 1];
        for (int64_t k0 = off[u]; k0 < e && !bad; k0 += 32) {
            const int64_t k = k0 + lane;
            bad = __any_sync(0xffffffffu, k < e && label[adj[k]] != mine);
        }
        if (bad && lane == 0) { atomicMax(bad_complement, ~(unsigned long long)u); }
    }
}

int grid_for(int64_t items)
{
    int64_t b = (items + kThreads - 1) / kThreads;
    if (b < 1) { b = 1; }
    if (b > 148 * 64) { b = 148 * 64; }
    return (int)b;
}

// The search's launch: as many CTAs as can be resident at once.
cudaError_t launch_search(const CheckParams &p, int device, int64_t source, const int64_t *parent)
{
    int per_sm = 0, sms = 0;
    cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, check_search_kernel, kSearch, 0);
    if (e == cudaSuccess) { e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); }
    if (e != cudaSuccess) { return e; }
    CheckParams q = p;
    void *args[] = {&q, &source, &parent};
    return cudaLaunchCooperativeKernel((const void *)check_search_kernel, dim3(per_sm * sms),
                                       dim3(kSearch), args, 0, 0);
}

CheckParams check_params(const bd_graph *g, const CheckScratch &s)
{
    CheckParams p{};
    p.off = g->d_off;
    p.adj = g->d_adj;
    p.n = g->n;
    p.arcs = g->arcs;
    p.symmetric = g->symmetric;
    p.polls = check_polls(g->max_degree);
    p.depth = s.depth;
    for (int i = 0; i < 2; ++i) {
        p.qs[i] = s.qs[i];
        p.ql[i] = s.ql[i];
        p.cb[i] = s.cb[i];
    }
    p.ctl = s.ctl;
    return p;
}

// The verdict in ctl.
bd_status read_verdict(const CheckCtl *ctl, int32_t *ok, int64_t *bad_vertex)
{
    CheckCtl h{};
    BD_CUDA(cudaMemcpy(&h, ctl, sizeof h, cudaMemcpyDeviceToHost));
    if (h.error) { return (bd_status)h.error; }
    *ok = h.bad == 0 ? 1 : 0;
    if (bad_vertex) { *bad_vertex = h.bad == 0 ? -1 : (int64_t)~h.bad; }
    return BD_OK;
}

}  // namespace

void check_free(CheckScratch *s)
{
    cudaFree(s->depth);
    for (int i = 0; i < 2; ++i) {
        cudaFree(s->qs[i]);
        cudaFree(s->ql[i]);
        cudaFree(s->cb[i]);
    }
    cudaFree(s->ctl);
    *s = CheckScratch{};
}

bd_status check_alloc(const bd_graph *g, CheckScratch *s)
{
    if (s->ctl) { return BD_OK; }
    const int64_t longs = g->arcs / kLong + 1;
    bool ok = cudaMalloc(&s->depth, sizeof(int32_t) * g->n) == cudaSuccess;
    for (int i = 0; i < 2 && ok; ++i) {
        ok = cudaMalloc(&s->qs[i], sizeof(uint32_t) * g->n) == cudaSuccess &&
             cudaMalloc(&s->ql[i], sizeof(uint32_t) * longs) == cudaSuccess &&
             cudaMalloc(&s->cb[i], sizeof(ull) * longs) == cudaSuccess;
    }
    if (ok && cudaMalloc(&s->ctl, sizeof(CheckCtl)) == cudaSuccess) { return BD_OK; }
    cudaGetLastError();
    check_free(s);
    return BD_ERR_OOM;
}

bd_status check_parents_device(const bd_graph *g, int64_t source, const int64_t *d_parent,
                               int32_t *ok, int64_t *bad_vertex, CheckScratch *scratch)
{
    if (source < 0 || source >= g->n) { return BD_ERR_RANGE; }
    BD_CUDA(cudaSetDevice(g->device));
    CheckScratch own;
    CheckScratch *s = scratch ? scratch : &own;
    BD_TRY(check_alloc(g, s));
    cudaError_t e = cudaMemsetAsync(s->ctl, 0, sizeof(CheckCtl), 0);
    if (e == cudaSuccess) { e = launch_search(check_params(g, *s), g->device, source, d_parent); }
    const bd_status st = e == cudaSuccess ? read_verdict(s->ctl, ok, bad_vertex)
                                          : cuda_fail(e, "device check", __FILE__, __LINE__);
    check_free(&own);
    return st;
}

bd_status check_components_device(const bd_graph *g, const int64_t *d_label, int32_t *ok,
                                  int64_t *bad_vertex)
{
    const int64_t n = g->n;
    if (n <= 0) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(g->device));
    int64_t *sorted_label = nullptr;
    uint32_t *vertex = nullptr, *sorted_vertex = nullptr;
    CheckScratch own;
    void *scratch = nullptr;
    size_t scratch_bytes = 0;
    auto release = [&]() {
        cudaFree(sorted_label);
        cudaFree(vertex);
        cudaFree(sorted_vertex);
        cudaFree(scratch);
        check_free(&own);
    };
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, scratch_bytes, d_label, sorted_label,
                                                    vertex, sorted_vertex, n);
    if (e != cudaSuccess) { return cuda_fail(e, "components check", __FILE__, __LINE__); }
    if (cudaMalloc(&sorted_label, sizeof(int64_t) * n) != cudaSuccess ||
        cudaMalloc(&vertex, sizeof(uint32_t) * n) != cudaSuccess ||
        cudaMalloc(&sorted_vertex, sizeof(uint32_t) * n) != cudaSuccess ||
        cudaMalloc(&scratch, scratch_bytes ? scratch_bytes : 1) != cudaSuccess ||
        check_alloc(g, &own) != BD_OK) {
        release();
        return BD_ERR_OOM;
    }
    auto step = [&](cudaError_t r) {
        if (e == cudaSuccess) { e = r; }
        return e == cudaSuccess;
    };
    const CheckParams p = check_params(g, own);
    iota_kernel<<<grid_for(n), kThreads>>>(vertex, n);
    step(cudaGetLastError());
    step(cub::DeviceRadixSort::SortPairs(scratch, scratch_bytes, d_label, sorted_label, vertex,
                                         sorted_vertex, n));
    step(cudaMemsetAsync(p.depth, 0xff, sizeof(int32_t) * n, 0));
    step(cudaMemsetAsync(p.ctl, 0, sizeof(CheckCtl), 0));
    if (e == cudaSuccess) {
        label_sources_kernel<<<grid_for(n), kThreads>>>(p, sorted_label, sorted_vertex);
        step(cudaGetLastError());
    }
    if (e == cudaSuccess) { step(launch_search(p, g->device, -1, nullptr)); }
    if (e == cudaSuccess) {
        check_components_kernel<<<grid_for_warps(n), kThreads>>>(g->d_off, g->d_adj, n, p.depth,
                                                                 d_label, &p.ctl->bad);
        step(cudaGetLastError());
    }
    const bd_status st = e == cudaSuccess ? read_verdict(p.ctl, ok, bad_vertex)
                                          : cuda_fail(e, "components check", __FILE__, __LINE__);
    release();
    return st;
}

}  // namespace bd

extern "C" {

bd_status bd_graph_check_parents(const bd_graph *g, int64_t source, const int64_t *parent,
                                 int32_t *ok, int64_t *bad_vertex)
{
    if (!g || !parent || !ok) { return BD_ERR_INVALID; }
    if (source < 0 || source >= g->n) { return BD_ERR_RANGE; }
    BD_TRY(bd::ensure_device());
    BD_CUDA(cudaSetDevice(g->device));
    int64_t *d_parent = nullptr;
    if (cudaMalloc(&d_parent, sizeof(int64_t) * g->n) != cudaSuccess) { return BD_ERR_OOM; }
    const cudaError_t e =
        cudaMemcpy(d_parent, parent, sizeof(int64_t) * g->n, cudaMemcpyHostToDevice);
    const bd_status st = e == cudaSuccess
                             ? bd::check_parents_device(g, source, d_parent, ok, bad_vertex, nullptr)
                             : bd::cuda_fail(e, "copy parents", __FILE__, __LINE__);
    cudaFree(d_parent);
    return st;
}


bd_status bd_graph_check_components(const bd_graph *g, const int64_t *component, int32_t *ok,
                                    int64_t *bad_vertex)
{
    if (!g || !component || !ok) { return BD_ERR_INVALID; }
    if (g->n <= 0) { return BD_ERR_INVALID; }
    BD_TRY(bd::ensure_device());
    BD_CUDA(cudaSetDevice(g->device));
    int64_t *d_label = nullptr;
    if (cudaMalloc(&d_label, sizeof(int64_t) * g->n) != cudaSuccess) { return BD_ERR_OOM; }
    const cudaError_t e =
        cudaMemcpy(d_label, component, sizeof(int64_t) * g->n, cudaMemcpyHostToDevice);
    const bd_status st = e == cudaSuccess
                             ? bd::check_components_device(g, d_label, ok, bad_vertex)
                             : bd::cuda_fail(e, "copy labels", __FILE__, __LINE__);
    cudaFree(d_label);
    return st;
}

}  // extern "C"
