// Supersteps run by one CTA: sizes and the scan shared by BFS and SSSP.
//
// A frontier is small when one CTA expands it in about the time a superstep
// of the kernel chain takes on an empty one (15-17 us): at most kSmallCap
// vertices (two per thread) with at most kSmallEdges out-edges (four rounds
// of kSmallItems edges per thread).
#pragma once
#include "olive_b200/olv_advance.cuh"

namespace olv {

constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallCap = 2 * kSmallThreads;
constexpr uint32_t kSmallEdges = 16384;
constexpr int kSmallItems = 4;

// The edges of the vertices being expanded, numbered 0 .. total - 1 in entry
// order: where each entry's edges begin, and the owner of every 16th edge, so
// that a thread finds the owner of its edge between two neighbours of that
// list (a few steps, where a search over all entries takes eleven).
struct SmallIndex {
    uint32_t beg[kSmallCap];                   // entry -> first edge (CSR position)
    uint16_t off[kSmallCap];                   // entry -> first edge number
    uint16_t own[kSmallEdges / 16 + 2];        // edge number / 16 -> owner
    uint32_t warp[2][32];                      // warp totals, by turns

    // Whole CTA: number the edges of n <= kSmallCap entries; entry i has
    // deg(i) edges from CSR position first(i).  Returns the total; above
    // kSmallEdges nothing is numbered.  One barrier; the caller's next one
    // makes the numbering visible.
    template <class Deg, class First>
    __device__ __forceinline__ uint32_t number(uint32_t n, uint32_t turn, Deg deg, First first) {
        const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
        const bool two = n > kSmallThreads;
        const uint32_t i = two ? 2 * threadIdx.x : threadIdx.x;
        const uint32_t d0 = i < n ? deg(i) : 0, d1 = two && i + 1 < n ? deg(i + 1) : 0;
        uint32_t incl = d0 + d1;
        if (wid * (two ? 64 : 32) < n) {   // warps without entries have no sum
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += t;
            }
        }
        if (lane == 31) warp[turn & 1][wid] = incl;
        __syncthreads();
        const uint32_t w = warp[turn & 1][lane];
        const uint32_t total = __reduce_add_sync(0xffffffffu, w);
        if (total > kSmallEdges) return total;
        if (wid * (two ? 64 : 32) < n) {
            const uint32_t o0 = __reduce_add_sync(0xffffffffu, lane < wid ? w : 0) + incl - d0 - d1;
            if (i < n) put(i, o0, d0, first(i));
            if (two && i + 1 < n) put(i + 1, o0 + d0, d1, first(i + 1));
        }
        if (threadIdx.x == 0) own[(total + 15) / 16] = (uint16_t)(n - 1);
        return total;
    }
    __device__ __forceinline__ void put(uint32_t i, uint32_t o, uint32_t d, uint32_t b) {
        beg[i] = b;
        off[i] = (uint16_t)o;
        for (uint32_t c = (o + 15) / 16; 16 * c < o + d; c++) own[c] = (uint16_t)i;
    }
    // Owner of edge k: the last entry whose first edge is <= k.
    __device__ __forceinline__ uint32_t owner(uint32_t k) const {
        uint32_t lo = own[k / 16], hi = own[k / 16 + 1];
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) / 2;
            if (off[mid] <= k)
                lo = mid;
            else
                hi = mid - 1;
        }
        return lo;
    }
};

// Whole warp: places for the flagged items of its lanes (N per lane) in a list
// counted in shared memory: pos[j] of lane's item j, one atomic for the warp.
template <int N>
__device__ __forceinline__ void small_place(const bool (&p)[N], uint32_t *n, uint32_t (&pos)[N]) {
    unsigned m[N];
    uint32_t tot = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
        m[j] = __ballot_sync(0xffffffffu, p[j]);
        tot += __popc(m[j]);
    }
    if (!tot) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(n, tot);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int j = 0; j < N; j++) {
        pos[j] = base + __popc(m[j] & ((1u << lane_id()) - 1u));
        base += __popc(m[j]);
    }
}

}  // namespace olv
