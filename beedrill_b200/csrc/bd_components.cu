// bd_components.cu -- connected components (components.cc:38-118) on the
// device.
//
// The reference labels every vertex with the smallest vertex id of its
// component by label propagation: passes over all arcs lower a vertex's
// label to a neighbour's smaller one, pointer jumping shortens label
// chains, and passes repeat until nothing changes (num_iters of them).
// The labelling it converges to is unique -- each vertex gets the minimum
// id of its component -- so any algorithm that finds the components and
// names each by its minimum id gives the reference's labels exactly.
//
// Here a union-find forest in HBM (one uint32 parent per vertex; at scale
// 24 the 64 MB array stays in L2) is built by joins of arcs; joining links
// the larger root under the smaller one with one atomicCAS on the larger
// root's parent word, so every parent id is smaller than its child's and
// every root is the minimum id of its tree: the final roots are exactly the
// reference's labels.  Finds shorten paths as they walk (path splitting:
// each visited vertex is pointed at its grandparent, an ancestor, so the
// forest stays valid under concurrent finds and links).  Every loop ends: a
// find walks strictly decreasing ids, and a join retries only after another
// thread's link took its root, which happens at most n - 1 times in all.
//
// Which arcs are joined (symmetric CSR, every edge stored both ways), after
// Sutton, Ben-Nun and Barak, "Optimizing Parallel Graph Connectivity
// Computation via Subgraph Sampling" (IPDPS 2018, "Afforest"):
//   cc_hook_kernel        every vertex points at the smallest of itself and its
//                         first kHookArcs neighbours (a plain store: smaller ids
//                         cannot form a cycle), then at its root
//                         (cc_flatten_kernel);
//   cc_merge_kernel       for one more arc of every vertex, the larger of the two
//                         roots is lowered to the smaller by an atomicMin that
//                         nobody waits for.  Where several arcs lower one root the
//                         smallest wins and the others are dropped: nothing here
//                         has to join every sampled arc, because the walk below
//                         joins all arcs of what is left outside;
//   cc_probe_kernel       the largest tree, by a vote of kProbe vertices' roots;
//   cc_walk_kernel        every vertex OUTSIDE that tree (its parent word
//                         is not the tree's root) joins all of its
//                         arcs.  An edge between the largest tree and
//                         another vertex is stored at that other vertex
//                         too, and is joined from there, so skipping the
//                         largest tree's own arcs loses no edge.  A warp
//                         loads 32 vertices' parent words at once and walks
//                         only the lists of those with work; lists of more
//                         than kHeavy arcs go to cc_heavy_kernel, which
//                         deals every listed vertex's arcs over the grid in
//                         one flat range (a binary search per chunk, the
//                         chunk prefix from cc_heavy_chunks_kernel).
// (Joining the sampled arcs properly, by finds and atomicCAS, is what the first
// version did: whenever two large trees met, every vertex between them tried the
// same root word.  On file-order RMAT graphs that was 330 to 390 us for scale 18,
// where hooking, two rounds of merging and three flattenings take 33; 170 to 510 us
// at scale 22, where they take 180.)
//   cc_compress_kernel    labels (each vertex's root), sizes per label
//                         (one atomic per distinct label of a warp) and the
//                         count of roots.
// A CSR that does not hold every edge both ways takes every arc of every
// vertex instead (the same cc_walk_kernel / cc_heavy_kernel pair).

#include <algorithm>

#include "bd_device_util.cuh"
#include "bd_internal.h"

namespace bd {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int64_t kHeavy = 4096;    // arcs above which a vertex is split over the grid
constexpr int kHookArcs = 4;        // arcs a vertex looks at for its first parent
constexpr int kMergeRounds = 2;     // and a third where the probe asks for it
constexpr int kProbeOutside = 4;    // probed vertices outside the largest tree that do
constexpr int kProbeInside = 2;     // ... unless it holds no two of them
constexpr int kProbe = 256;         // vertices whose roots vote for the largest tree (one block)
constexpr int64_t kHeavyChunk = 1024;  // arcs per unit of the heavy pass

int grid_for_warps(int64_t warps)
{
    int64_t b = (warps + kWarps - 1) / kWarps;
    if (b < 1) { b = 1; }
    if (b > 148 * 64) { b = 148 * 64; }
    return (int)b;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x)
{
    for (int d = 16; d > 0; d >>= 1) { x += __shfl_xor_sync(0xffffffffu, x, d); }
    return x;
}

// Root of x's tree, pointing each vertex on the way at its grandparent.
//
// The loads go through L1 (ld.ca), which is not coherent between SMs, so a
// load may return an older value of a parent word.  That is safe: every
// value a parent word holds while joins run is an ancestor of its vertex with a
// smaller id (links and path splitting only write ancestors, and a tree
// only grows), so a stale walk still descends strictly and ends at a
// vertex that is, or was, a root of x's tree.  A join acts on such a root
// only through atomicCAS, which sees the current word.  (cc_merge_kernel may
// move a root from one tree to another, but in launches of its own, and L1
// starts empty in each launch.)  What L1 buys: nearly every vertex points at the
// largest tree's root by then, and checking that root's own word from every
// thread put millions of loads on one L2 slice (three times the time of a pass
// over the same bytes); from L1 each SM loads it once.
__device__ __forceinline__ uint32_t cc_find(uint32_t *parent, uint32_t x)
{
    uint32_t p = __ldca(&parent[x]);
    while (p != x) {
        const uint32_t gp = __ldca(&parent[p]);
        if (gp != p) { __stcg(&parent[x], gp); }
        x = p;
        p = gp;
    }
    return x;
}

// Root of x's tree without writes, for passes in which no join runs (the
// roots stay fixed, so the walk ends at x's current root).
__device__ __forceinline__ uint32_t cc_root(const uint32_t *parent, uint32_t x)
{
    uint32_t p = __ldca(&parent[x]);
    while (p != x) {
        x = p;
        p = __ldca(&parent[x]);
    }
    return x;
}

// Joins the trees of a and b: the larger root goes under the smaller.
__device__ __forceinline__ void cc_join(uint32_t *parent, uint32_t a, uint32_t b)
{
    // one parent word each: vertices pointing at the same vertex share a
    // tree (after a flatten, the common case)
    if (__ldca(&parent[a]) == __ldca(&parent[b])) { return; }
    uint32_t ra = cc_find(parent, a), rb = cc_find(parent, b);
    while (ra != rb) {
        if (ra < rb) {
            const uint32_t t = ra;
            ra = rb;
            rb = t;
        }
        const uint32_t old = atomicCAS(&parent[ra], ra, rb);
        if (old == ra) { return; }
        // ra was linked under `old` meanwhile; both roots may have moved.
        ra = cc_find(parent, old);
        rb = cc_find(parent, rb);
    }
}

__global__ void cc_init_kernel(uint32_t *parent, int64_t n, int64_t *size)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        parent[v] = (uint32_t)v;
        size[v] = 0;
    }
}

// Every vertex's first parent, the arc cc_merge_kernel takes, and sizes: the
// smallest of the vertex and its first kHookArcs neighbours (they share a sector
// or two); of the others the first, or the vertex itself if there is none.
// Isolated vertices are components of one already.
__global__ void cc_hook_kernel(const int64_t *off, const uint32_t *adj, int64_t n,
                               uint32_t *parent, uint32_t *second, int64_t *size)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = off[v], e = off[v + 1];
        const uint32_t u = (uint32_t)v;
        uint32_t a[kHookArcs], lo = u, other = u;
#pragma unroll
        for (int j = 0; j < kHookArcs; ++j) { a[j] = b + j < e ? __ldg(&adj[b + j]) : u; }
#pragma unroll
        for (int j = 0; j < kHookArcs; ++j) { lo = min(lo, a[j]); }
#pragma unroll
        for (int j = kHookArcs - 1; j >= 0; --j) { other = a[j] != lo && a[j] != u ? a[j] : other; }
        parent[v] = lo;
        __stcs(&second[v], other);
        __stcs(&size[v], (int64_t)(b == e));
    }
}

// Every vertex points at its root.  A warp lowers each distinct larger root once,
// and a block only to less than it has sent before (kSent roots, the first ones it
// meets): the arcs between two large trees all lower the same word, and one L2
// slice takes about one such request a nanosecond.  At scale 22 a request from
// every warp took 155 us, of which 16 are the reads; hence also few, large blocks.
constexpr int kMergeThreads = 1024;
constexpr int kSent = 2048;
__global__ void __launch_bounds__(kMergeThreads) cc_merge_kernel(const uint32_t *second, int64_t n,
                                                                 uint32_t *parent,
                                                                 const uint32_t *wanted)
{
    if (wanted && *wanted == 0) { return; }
    __shared__ uint32_t key[kSent], sent[kSent];
    for (int i = threadIdx.x; i < kSent; i += kMergeThreads) { key[i] = sent[i] = 0xffffffffu; }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t u = base + lane;
        uint32_t hi = 0, lo = 0;
        if (u < n) {
            const uint32_t v = __ldcs(&second[u]);
            // roots hooked meanwhile point elsewhere: that only changes which
            // of the two trees' vertices is compared
            const uint32_t ru = __ldca(&parent[u]), rv = v != (uint32_t)u ? __ldca(&parent[v]) : ru;
            hi = max(ru, rv);
            lo = min(ru, rv);
        }
        const bool want = hi != lo;
        const unsigned live = __ballot_sync(0xffffffffu, want);
        if (want) {
            const unsigned same = __match_any_sync(live, hi);
            const uint32_t least = __reduce_min_sync(same, lo);
            if (lane == __ffs(same) - 1) {
                const unsigned h = (hi * 2654435761u) >> 21;  // 11 bits: kSent
                const uint32_t k = atomicCAS(&key[h], 0xffffffffu, hi);
                if ((k != 0xffffffffu && k != hi) || least < atomicMin(&sent[h], least)) {
                    atomicMin(&parent[hi], least);
                }
            }
        }
    }
}

// Every vertex pointed at its root (a vertex already there is not
// written).  No join runs meanwhile, so the roots are fixed, and a thread
// writes its own vertex's word only, so none moves a word that has already
// been pointed at its root.  A walk longer than kNear moves that word along as
// it goes, and reads past L1: walks that come through the vertex then jump as
// far as its own has come, and a chain is crossed in some log2 of its length.
// (Hooking makes chains wherever ids follow a path, as in the rows of a grid.)
// Blocks start in the order of the ids, each with the next F * kThreads, and
// chains lead to smaller ids, so that they end where a block has been: a
// 4000 x 4003 grid took 1750 us in blocks that stride over the ids, without
// moving words, and takes 210.
constexpr int kNear = 8;
template <int F>
__global__ void __launch_bounds__(kThreads) cc_flatten_kernel(uint32_t *parent, int64_t n,
                                                              const uint32_t *wanted)
{
    if (wanted && *wanted == 0) { return; }
    const int64_t first = blockIdx.x * (int64_t)(F * kThreads) + threadIdx.x;
    uint32_t p[F], up[F];
#pragma unroll
    for (int k = 0; k < F; ++k) {
        const int64_t v = first + k * kThreads;
        p[k] = v < n ? __ldcg(&parent[v]) : 0u;
    }
#pragma unroll
    for (int k = 0; k < F; ++k) { up[k] = __ldca(&parent[p[k]]); }
#pragma unroll
    for (int k = 0; k < F; ++k) {
        const int64_t v = first + k * kThreads;
        if (v >= n || up[k] == p[k]) { continue; }
        uint32_t r = up[k], q = __ldca(&parent[r]);
        for (int i = 1; i < kNear && q != r; ++i) {
            r = q;
            q = __ldca(&parent[r]);
        }
        while (q != r) {
            __stcg(&parent[v], q);
            r = q;
            q = __ldcg(&parent[r]);
        }
        __stcg(&parent[v], r);
    }
}

// Two vertices a thread where five device-fuls of threads and more have a vertex
// each (148 SMs x 2048 threads): fewer blocks, and the reads of two walks at once.  A run
// in us with one and with two: grid 1021 x 1031 110, 134; 1400 x 1402 151, 140; scale
// 22 225, 203; 24 735, 649.
void launch_flatten(uint32_t *parent, int64_t n, const uint32_t *wanted, cudaStream_t s)
{
    const int64_t blocks = std::max<int64_t>(1, (n + kThreads - 1) / kThreads);
    if (n < 5ll * 148 * 2048) {
        cc_flatten_kernel<1><<<(unsigned)blocks, kThreads, 0, s>>>(parent, n, wanted);
    } else {
        cc_flatten_kernel<2><<<(unsigned)((blocks + 1) / 2), kThreads, 0, s>>>(parent, n, wanted);
    }
}

// giant[0]: the most frequent root of kProbe vertices spread evenly over the ids
// (the smallest of equally frequent ones).  giant[1]: whether another merging round
// pays, because kProbeOutside of them have neighbours but lie outside that tree (a
// second large tree is left now and then; the walk would then read all its arcs:
// scale 22 in file order 373 us without the third round, 278 with it, where other
// graphs lose 20 to 75 us by a round they do not need) -- unless no two share a
// root, as in a forest of small trees, where no large one is in the making (a
// shuffled path of 3 M vertices 330 -> 280 us).  One block, so that the host need
// not look.
__global__ void __launch_bounds__(kProbe) cc_probe_kernel(const uint32_t *parent, int64_t n,
                                                          const uint32_t *isolated, uint32_t *giant,
                                                          const uint32_t *wanted)
{
    if (wanted && *wanted == 0) { return; }
    __shared__ __align__(16) uint32_t root[kProbe];
    __shared__ unsigned long long best[kProbe / 32];
    const uint32_t v = (uint32_t)(((uint64_t)threadIdx.x * (uint64_t)n) / kProbe);
    const uint32_t mine = cc_root(parent, v);
    const bool lone = (isolated[v >> 5] >> (v & 31)) & 1u;
    root[threadIdx.x] = mine;
    __syncthreads();
    unsigned votes = 0;
    const uint4 *r4 = reinterpret_cast<const uint4 *>(root);
#pragma unroll 8
    for (int i = 0; i < kProbe / 4; ++i) {
        const uint4 r = r4[i];
        votes += (r.x == mine) + (r.y == mine) + (r.z == mine) + (r.w == mine);
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, votes);
    const uint32_t who = __reduce_min_sync(0xffffffffu, votes == top ? mine : 0xffffffffu);
    if ((threadIdx.x & 31) == 0) { best[threadIdx.x >> 5] = ((unsigned long long)top << 32) | ~who; }
    __syncthreads();
    unsigned long long m = 0;
    for (int i = 0; i < kProbe / 32; ++i) { m = best[i] > m ? best[i] : m; }
    const uint32_t g = ~(uint32_t)m;
    const int outside = __syncthreads_count(mine != g && !lone);
    if (threadIdx.x == 0) {
        giant[0] = g;
        giant[1] = outside >= kProbeOutside && (unsigned)(m >> 32) >= kProbeInside;
    }
}

struct CcWalk {
    int32_t incl[32];
    int64_t beg[32];
};

// The arcs of the vertices of a warp's 32-vertex group that have
// work; lists longer than kHeavy are appended to `heavy` instead.
// giant: vertices whose root is this id have no work (the largest tree), and the
// lists of the others are laid end to end and dealt to the lanes, 32 arcs a round
// (list by list, a graph without a large tree kept two lanes busy at degree 2: a
// shuffled path of 3 M vertices 295 us, now 75).  null: every vertex has work, and
// the whole warp takes one list at a time.  Nothing is joined yet then, and arcs of
// 32 vertices at once contend for the roots of the large trees more than arcs of
// one (RMAT scale 18 given as a CSR, us a run: end to end 250, list by list 205; 8
// arcs a vertex 245, 178; a 1000 x 1000 grid 176, 339).
__global__ void __launch_bounds__(kThreads) cc_walk_kernel(
    const int64_t *off, const uint32_t *adj, int64_t n, uint32_t *parent, const uint32_t *giant,
    uint32_t *heavy, unsigned long long *heavy_count)
{
    __shared__ CcWalk scratch[kWarps];
    CcWalk &ws = scratch[threadIdx.x >> 5];
    const uint32_t skip_root = giant ? *giant : 0u;
    const int lane = threadIdx.x & 31;
    const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = gw * 32; base < n; base += nw * 32) {
        const int64_t u = base + lane;
        int64_t b = 0, e = 0;
        bool work = false;
        if (u < n) {
            work = !giant || __ldcg(&parent[u]) != skip_root;
            if (work) {
                b = off[u];
                e = off[u + 1];
                work = b < e;
            }
            if (work && e - b > kHeavy) {
                heavy[atomicAdd(heavy_count, 1ull)] = (uint32_t)u;
                work = false;
            }
        }
        if (!giant) {
            unsigned todo = __ballot_sync(0xffffffffu, work);
            while (todo) {
                const int owner = __ffs(todo) - 1;
                todo &= todo - 1;
                const int64_t bb = __shfl_sync(0xffffffffu, b, owner);
                const int64_t ee = __shfl_sync(0xffffffffu, e, owner);
                for (int64_t k = bb + lane; k < ee; k += 32) {
                    cc_join(parent, (uint32_t)(base + owner), __ldg(&adj[k]));
                }
            }
            continue;
        }
        const int32_t incl = dev::warp_incl_scan(work ? (int32_t)(e - b) : 0);
        const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (total == 0) { continue; }
        ws.incl[lane] = incl;
        ws.beg[lane] = b;
        __syncwarp();
        for (int32_t k = lane; k < total; k += 32) {
            int at = 0;  // lists that end at or before arc k
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                if (ws.incl[at + d - 1] <= k) { at += d; }
            }
            const int64_t arc = ws.beg[at] + (k - (at ? ws.incl[at - 1] : 0));
            cc_join(parent, (uint32_t)(base + at), __ldg(&adj[arc]));
        }
        __syncwarp();
    }
}

// Chunk prefix of the heavy list: cbase[i] = chunks of heavy vertices < i.
// One block of 1024 threads scans 1024 entries per round.
__global__ void __launch_bounds__(1024) cc_heavy_chunks_kernel(
    const int64_t *off, const uint32_t *heavy, const unsigned long long *heavy_count,
    unsigned long long *cbase)
{
    __shared__ unsigned long long warp_tot[32];
    __shared__ unsigned long long carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t count = (int64_t)*heavy_count;
    if (threadIdx.x == 0) { carry = 0; }
    __syncthreads();
    for (int64_t base = 0; base < count; base += 1024) {
        const int64_t i = base + threadIdx.x;
        unsigned long long c = 0;
        if (i < count) {
            const uint32_t u = heavy[i];
            const int64_t len = off[u + 1] - off[u];
            c = (unsigned long long)((len + kHeavyChunk - 1) / kHeavyChunk);
        }
        unsigned long long incl = c;
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) { incl += y; }
        }
        if (lane == 31) { warp_tot[warp] = incl; }
        __syncthreads();
        if (warp == 0) {
            unsigned long long t = warp_tot[lane];
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, t, d);
                if (lane >= d) { t += y; }
            }
            warp_tot[lane] = t;  // inclusive prefix over warps
        }
        __syncthreads();
        const unsigned long long before = carry + (warp ? warp_tot[warp - 1] : 0ull);
        if (i < count) { cbase[i] = before + incl - c; }
        __syncthreads();
        if (threadIdx.x == 1023) { carry = before + incl; }
        __syncthreads();
    }
    if (threadIdx.x == 0) { cbase[count] = carry; }
}

// The heavy vertices' arcs as one flat range of kHeavyChunk-arc chunks dealt
// to the warps of the grid (a warp per chunk, a binary search for its
// vertex), so no thread walks one vertex's chunks after another.
__global__ void __launch_bounds__(kThreads) cc_heavy_kernel(
    const int64_t *off, const uint32_t *adj, uint32_t *parent, const uint32_t *heavy,
    const unsigned long long *heavy_count, const unsigned long long *cbase)
{
    const int lane = threadIdx.x & 31;
    const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t count = (int64_t)*heavy_count;
    if (count == 0) { return; }
    const int64_t total = (int64_t)cbase[count];
    for (int64_t c = gw; c < total; c += nw) {
        int64_t lo = 0, hi = count - 1;  // last i with cbase[i] <= c
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if ((int64_t)cbase[mid] <= c) { lo = mid; } else { hi = mid - 1; }
        }
        const uint32_t u = heavy[lo];
        const int64_t b = off[u] + (c - (int64_t)cbase[lo]) * kHeavyChunk;
        const int64_t e = min(off[u + 1], b + kHeavyChunk);
        for (int64_t k = b + lane; k < e; k += 32) {
            cc_join(parent, u, __ldg(&adj[k]));
        }
    }
}

// Labels, sizes and roots.  `hint` is a vertex of the largest tree (or null):
// the lanes whose label is that tree's root count it in a block-wide
// total added once per block, as do the roots; the lanes of a warp that
// share any other label add it once (__match_any_sync).  Isolated vertices, with
// `isolated` given, have their size already.  (One atomic per
// warp on the largest component's size and on the root count put a few
// hundred thousand atomics on two addresses, which serialise at their L2
// slices.)
__global__ void cc_compress_kernel(uint32_t *parent, int64_t n, const uint32_t *hint,
                                   const uint32_t *isolated, int64_t *label, int64_t *size,
                                   unsigned long long *roots)
{
    __shared__ uint32_t giant;
    __shared__ unsigned long long blk_giant, blk_roots;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        giant = hint ? cc_root(parent, *hint) : 0xFFFFFFFFu;
        blk_giant = blk_roots = 0;
    }
    __syncthreads();
    const uint32_t g = giant;
    unsigned long long my_giant = 0, my_roots = 0;
    for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; base < n;
         base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + lane;
        const bool valid = v < n;
        uint32_t r = 0xFFFFFFFFu;
        if (valid) {
            // a vertex pointing at the largest tree's root needs no walk
            const uint32_t p = __ldcs(&parent[v]);
            r = p == g ? g : cc_root(parent, p);
            __stcs(&label[v], (int64_t)r);
        }
        const bool alone = valid && isolated && (__ldg(&isolated[v >> 5]) >> lane) & 1u;
        const bool other = valid && r != g && !alone;
        const unsigned same = __match_any_sync(0xffffffffu, other ? r : 0xFFFFFFFFu);
        if (other && lane == __ffs(same) - 1) {
            atomicAdd(reinterpret_cast<unsigned long long *>(&size[r]),
                      (unsigned long long)__popc(same));
        }
        my_giant += (valid && r == g && !alone) ? 1ull : 0ull;
        my_roots += (valid && r == (uint32_t)v) ? 1ull : 0ull;
    }
    my_giant = warp_sum_u64(my_giant);
    my_roots = warp_sum_u64(my_roots);
    if (lane == 0) {
        if (my_giant) { atomicAdd(&blk_giant, my_giant); }
        if (my_roots) { atomicAdd(&blk_roots, my_roots); }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (blk_giant) {
            atomicAdd(reinterpret_cast<unsigned long long *>(&size[g]), blk_giant);
        }
        if (blk_roots) { atomicAdd(roots, blk_roots); }
    }
}

int grid_for(int64_t items)
{
    int64_t b = (items + kThreads - 1) / kThreads;
    if (b < 1) { b = 1; }
    if (b > 148 * 64) { b = 148 * 64; }
    return (int)b;
}

}  // namespace
}  // namespace bd

// Handle: the graph it borrows, its stream and the device arrays.
struct bd_components {
    int device = 0;
    bd_graph *g = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    uint32_t *parent = nullptr;            // [n] union-find forest
    uint32_t *heavy = nullptr;             // [arcs / kHeavy + 1] vertices split over the grid
    unsigned long long *cbase = nullptr;   // [arcs / kHeavy + 2] their chunk prefix
    uint32_t *giant = nullptr;             // [0] root of the largest tree, [1] merge again
    unsigned long long *counters = nullptr;  // [0] heavy vertices, [1] roots
    int64_t *label = nullptr;              // [n] component_ (components.h:13)
    int64_t *size = nullptr;               // [n] component_size_ (components.h:15)
    bool ran = false;
    bd_components_stats last{};
};

namespace {

void components_free(bd_components *c)
{
    if (!c) { return; }
    cudaSetDevice(c->device);
    if (c->stream) { cudaStreamSynchronize(c->stream); }
    cudaFree(c->parent);
    cudaFree(c->heavy);
    cudaFree(c->cbase);
    cudaFree(c->giant);
    cudaFree(c->counters);
    cudaFree(c->label);
    cudaFree(c->size);
    if (c->ev0) { cudaEventDestroy(c->ev0); }
    if (c->ev1) { cudaEventDestroy(c->ev1); }
    if (c->stream) { cudaStreamDestroy(c->stream); }
    delete c;
}

}  // namespace

extern "C" {

bd_status bd_components_create(bd_graph *g, bd_components **out)
{
    if (!g || !out) { return BD_ERR_INVALID; }
    BD_TRY(bd::ensure_device());
    BD_CUDA(cudaSetDevice(g->device));
    auto *c = new bd_components();
    c->device = g->device;
    c->g = g;
    const int64_t n = g->n;
    const int64_t heavy_cap = g->arcs / bd::kHeavy + 1;
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
        cudaMalloc(&c->parent, sizeof(uint32_t) * (n ? n : 1)) != cudaSuccess ||
        cudaMalloc(&c->heavy, sizeof(uint32_t) * heavy_cap) != cudaSuccess ||
        cudaMalloc(&c->cbase, sizeof(unsigned long long) * (heavy_cap + 1)) != cudaSuccess ||
        cudaMalloc(&c->giant, sizeof(uint32_t) * 2) != cudaSuccess ||
        cudaMalloc(&c->counters, sizeof(unsigned long long) * 2) != cudaSuccess ||
        cudaMalloc(&c->label, sizeof(int64_t) * (n ? n : 1)) != cudaSuccess ||
        cudaMalloc(&c->size, sizeof(int64_t) * (n ? n : 1)) != cudaSuccess) {
        components_free(c);
        return BD_ERR_OOM;
    }
    *out = c;
    return BD_OK;
}

// components::clear (components.cc:33-36) does nothing; run() starts over.
bd_status bd_components_clear(bd_components *c)
{
    if (!c) { return BD_ERR_INVALID; }
    return BD_OK;
}

bd_status bd_components_run(bd_components *c, bd_components_stats *stats)
{
    if (!c) { return BD_ERR_INVALID; }
    BD_CUDA(cudaSetDevice(c->device));
    const bd_graph *g = c->g;
    const int64_t n = g->n;
    cudaStream_t s = c->stream;
    BD_CUDA(cudaEventRecord(c->ev0, s));
    BD_CUDA(cudaMemsetAsync(c->counters, 0, sizeof(unsigned long long) * 2, s));
    const uint32_t *giant = nullptr, *isolated = nullptr;
    if (g->symmetric) {
        // (the label array, written only by the final pass, holds the
        // arcs to merge meanwhile)
        uint32_t *second = reinterpret_cast<uint32_t *>(c->label);
        bd::cc_hook_kernel<<<bd::grid_for(n), bd::kThreads, 0, s>>>(g->d_off, g->d_adj, n, c->parent,
                                                                    second, c->size);
        bd::launch_flatten(c->parent, n, nullptr, s);
        const int merge_grid = std::min(bd::grid_for(n) / 4 + 1, 148 * 2);
        const uint32_t *wanted = nullptr;  // the last round's kernels ask the probe
        for (int round = 0; round <= bd::kMergeRounds; ++round) {
            bd::cc_merge_kernel<<<merge_grid, bd::kMergeThreads, 0, s>>>(second, n, c->parent, wanted);
            bd::launch_flatten(c->parent, n, wanted, s);
            if (round + 1 >= bd::kMergeRounds) {
                bd::cc_probe_kernel<<<1, bd::kProbe, 0, s>>>(c->parent, n, g->d_isolated, c->giant,
                                                             wanted);
                wanted = c->giant + 1;
            }
        }
        giant = c->giant;
        isolated = g->d_isolated;
    } else {
        bd::cc_init_kernel<<<bd::grid_for(n), bd::kThreads, 0, s>>>(c->parent, n, c->size);
    }
    // symmetric: the arcs of vertices outside the largest tree;
    // otherwise every arc of every vertex
    bd::cc_walk_kernel<<<bd::grid_for_warps(n), bd::kThreads, 0, s>>>(
        g->d_off, g->d_adj, n, c->parent, giant, c->heavy, c->counters);
    bd::cc_heavy_chunks_kernel<<<1, 1024, 0, s>>>(g->d_off, c->heavy, c->counters, c->cbase);
    bd::cc_heavy_kernel<<<148 * 8, bd::kThreads, 0, s>>>(g->d_off, g->d_adj, c->parent, c->heavy,
                                                        c->counters, c->cbase);
    bd::cc_compress_kernel<<<bd::grid_for(n), bd::kThreads, 0, s>>>(
        c->parent, n, giant, isolated, c->label, c->size, c->counters + 1);
    BD_CUDA(cudaGetLastError());
    BD_CUDA(cudaEventRecord(c->ev1, s));
    unsigned long long roots = 0;
    BD_CUDA(cudaMemcpyAsync(&roots, c->counters + 1, sizeof(roots), cudaMemcpyDeviceToHost, s));
    BD_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    BD_CUDA(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
    c->last.num_components = (int64_t)roots;
    c->last.num_iters = 1;
    c->last.ms = ms;
    c->ran = true;
    if (stats) { *stats = c->last; }
    return BD_OK;
}

bd_status bd_components_get_labels(bd_components *c, int64_t *component)
{
    if (!c || !component) { return BD_ERR_INVALID; }
    if (!c->ran) { return BD_ERR_STATE; }
    BD_CUDA(cudaSetDevice(c->device));
    BD_CUDA(cudaMemcpy(component, c->label, sizeof(int64_t) * c->g->n, cudaMemcpyDeviceToHost));
    return BD_OK;
}

bd_status bd_components_get_sizes(bd_components *c, int64_t *component_size)
{
    if (!c || !component_size) { return BD_ERR_INVALID; }
    if (!c->ran) { return BD_ERR_STATE; }
    BD_CUDA(cudaSetDevice(c->device));
    BD_CUDA(cudaMemcpy(component_size, c->size, sizeof(int64_t) * c->g->n, cudaMemcpyDeviceToHost));
    return BD_OK;
}

bd_status bd_components_device_labels(bd_components *c, const int64_t **component)
{
    if (!c || !component) { return BD_ERR_INVALID; }
    if (!c->ran) { return BD_ERR_STATE; }
    *component = c->label;
    return BD_OK;
}

bd_status bd_components_check(bd_components *c, int32_t *ok)
{
    if (!c || !ok) { return BD_ERR_INVALID; }
    if (!c->ran) { return BD_ERR_STATE; }
    return bd::check_components_device(c->g, c->label, ok, nullptr);
}

bd_status bd_components_destroy(bd_components *c)
{
    if (!c) { return BD_ERR_INVALID; }
    components_free(c);
    return BD_OK;
}

}  // extern "C"
