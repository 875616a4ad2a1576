// bd_split.h -- how finely a frontier too small to occupy the device is dealt to
// its warps.  Plain arithmetic, for host and device code.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define BD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define BD_HOST_DEVICE inline
#endif

namespace bd {
namespace dev {

// How finely a frontier is dealt to nw warps when it is too small to give each a
// full round of arcs.  A warp's round costs time in proportion to its arcs (each
// takes some eight scattered requests through the warp's SM: 128 arcs of a batched
// push 8,000 to 12,000 cycles), so few arcs are spread thinner, down to 32
// a warp: the first push of 64 roots 25 -> 13 us at scales 12 to 22, pushes on a
// 509 x 523 grid 13.0 -> 9.7 ms (a quarter as many work items: 11.2).
//
// log2 of the parts a chunk of `chunk` arcs is cut into, of 32 arcs or more each.
BD_HOST_DEVICE int split_chunks(long long chunks, uint32_t chunk, long long nw)
{
    int k = 0;
    while ((chunks << (k + 1)) <= nw && (chunk >> (k + 1)) >= 32) { ++k; }
    return k;
}

// Arcs of one of a chunk's 1 << cut parts: a whole number of warp reads, rounded up
// at both steps so that the parts cover the chunk whatever its length (the last ones
// may be short or empty).
BD_HOST_DEVICE int64_t split_part(uint32_t chunk, int cut)
{
    return ((((int64_t)chunk - 1) >> cut) + 32) / 32 * 32;
}

// Arcs per chunk of what a batched pull leaves of a list after `arcs` of its arcs:
// about two such lengths (scale 22, 512 arcs: 4.59 ms with 512 a chunk, 4.63 with 2048).
BD_HOST_DEVICE int32_t long_chunk(int32_t arcs)
{
    return arcs < 64 ? 128 : arcs < 1024 ? 2 * arcs : 2048;
}

// Polls a barrier of the device check waits at most: some 2 s, and more where a list
// is long, since one warp may look through it between two barriers, 128 arcs in the
// time of two or three polls (the bound allows 32 such lists, a warp's share).
BD_HOST_DEVICE long long check_polls(long long max_degree) { return 4000000 + max_degree; }

// log2 of the vertices a warp takes at once: 32, or fewer of about 32 arcs
// together (avg: the frontier's average degree).
BD_HOST_DEVICE int split_group(long long vertices, int avg, long long nw)
{
    int k = 5;
    while (k > 0 && (avg << k) > 32 && (vertices >> (k - 1)) < nw) { --k; }
    return k;
}

}  // namespace dev
}  // namespace bd
