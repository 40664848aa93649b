// Row sums over a relabelled, degree-sorted CSR-shaped structure: the pull
// core of PageRank.
//
// The rows (vertices) are renumbered by length, longest first, and the
// neighbour ids inside the rows are renumbered the same way, so that
//   * a warp's rows have nearly equal lengths, and a fixed group of G lanes
//     per row (G = 1..32, chosen from the row length) keeps every lane busy
//     with about kTileU entries per round and no segmented scan;
//   * the high-degree vertices, whose values most rows gather, sit together
//     at the front of every per-vertex array, so their lines stay in L1/L2;
//   * the per-row inputs and outputs are read and written as contiguous runs.
// Rows longer than kTileLong are cut into kTileSeg-entry segments summed by
// k_row_segments and folded in segment order.
//
// Every sum has a fixed evaluation order: lane j of a row's group adds the
// row's entries j, j+G, j+2G, ... in order with compensated (two-sum) FP32
// arithmetic, then a fixed shuffle tree combines the group's lanes.  Warps
// take tiles by a fixed stride over a fixed grid, so the FP64 partials the
// row updates produce are also summed in a fixed order.
//
// An Op supplies (row ids are the new ids):
//   void begin()                                per-launch setup (ping-pong choice)
//   float term(uint32_t e, uint32_t j)          value of entry e with neighbour j
//   struct Row; Row row(uint32_t v)             per-row inputs of the update
//   void finish(uint32_t v, float s, float c, const Row &r, double &res, double &aux)
//                                               consume the row sum s + c; res and aux
//                                               are FP64 partials
//   const uint32_t *done                        the kernels return when *done
#pragma once
#include "olv_rowsolve.cuh"

namespace olv {

constexpr uint32_t kTileLong = 2048;   // rows longer than this are segmented
#ifndef OLV_TILE_SEG
#define OLV_TILE_SEG 512
#endif
constexpr uint32_t kTileSeg = OLV_TILE_SEG;   // entries per segment of a long row
#ifndef OLV_TILE_U
#define OLV_TILE_U 8
#endif
#ifndef OLV_TILE_MINB
#define OLV_TILE_MINB 6
#endif
constexpr int kTileU = OLV_TILE_U;     // entries per lane per round (loads in flight)
constexpr int kTileMinBlocks = OLV_TILE_MINB;   // resident CTAs per SM of the tile pass
constexpr int kStrips = 8;             // 32-entry strips per warp with loads in flight (segments)
constexpr uint32_t kNoSeg = 0xffffffu;
constexpr uint32_t kTileCTAs = 148 * kTileMinBlocks;  // fixed grid of the tile pass
                                                      // (fixed partial order), one wave

// Relabelled structure and its tiles.  tiles[t] = (first row, lg | first
// segment << 8): the tile covers rows first .. first + (32 >> lg) - 1 with
// G = 1 << lg lanes per row; a long row has a tile of its own (lg = 5) whose
// first segment index is below kNoSeg.
struct TilePlan {
    DevBuf perm;      // new id -> old id
    DevBuf newid;     // old id -> new id
    DevBuf ptr;       // [n + 1] row offsets in the new order
    DevBuf idx;       // neighbour ids, relabelled, rows in the new order
    DevBuf tiles, seg_range, segs, partials;
    uint32_t n = 0, ntiles = 0, nsegs = 0;
    void release() {
        perm.release(); newid.release(); ptr.release(); idx.release();
        tiles.release(); seg_range.release(); segs.release(); partials.release();
    }
};

// Build the plan from a device row-offset array (n rows) and its neighbour
// array (rowplan.cu).  lanes_u: entries per lane per round the grouping aims at
// (rows get the fewest lanes G = 1..32 with G * lanes_u >= row length); the
// autotuner's "pr_tile_u".
int build_tile_plan(const uint32_t *ptr_dev, const uint32_t *idx_dev, uint32_t n, cudaStream_t s,
                    TilePlan &p, uint32_t lanes_u = kTileU);

// One warp per segment of a long row: each lane sums its entries (stride 32,
// kStrips loads in flight) in order, then a fixed shuffle tree combines the
// lanes.
template <class Op>
__global__ void __launch_bounds__(kBlock)
k_row_segments(const uint32_t *__restrict__ idx, const uint2 *__restrict__ seg_range,
               uint32_t nsegs, Op op, float2 *__restrict__ segs) {
    if (*op.done) return;
    op.begin();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w = (blockIdx.x * kBlock + threadIdx.x) >> 5;
    if (w >= nsegs) return;   // whole warps only
    const uint2 r = seg_range[w];
    float s = 0.0f, c = 0.0f;
    for (uint32_t base = r.x; base < r.y; base += 32 * kStrips) {
        uint32_t j[kStrips];
#pragma unroll
        for (int q = 0; q < kStrips; q++) {
            const uint32_t i = base + q * 32 + lane;
            j[q] = i < r.y ? __ldg(&idx[i]) : 0u;
        }
        float x[kStrips];
#pragma unroll
        for (int q = 0; q < kStrips; q++) {
            const uint32_t i = base + q * 32 + lane;
            x[q] = i < r.y ? op.term(i, j[q]) : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < kStrips; q++) two_sum_acc(s, c, x[q]);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float s2 = __shfl_down_sync(0xffffffffu, s, o);
        const float c2 = __shfl_down_sync(0xffffffffu, c, o);
        pair_add(s, c, s2, c2);
    }
    if (lane == 0) segs[w] = make_float2(s, c);
}

template <class Op>
__global__ void __launch_bounds__(kBlock, kTileMinBlocks)
k_row_tiles(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ idx,
            const uint2 *__restrict__ tiles, uint32_t ntiles, uint32_t nrows,
            const float2 *__restrict__ segs, Op op, double *__restrict__ partials) {
    if (*op.done) return;
    op.begin();
    constexpr unsigned kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * kBlock + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * kBlock) >> 5;
    double res = 0.0, aux = 0.0;
    uint2 tdn = gw < ntiles ? tiles[gw] : make_uint2(0, 0);
    for (uint32_t t = gw; t < ntiles; t += nw) {
        const uint2 td = tdn;   // the next tile's descriptor is fetched one tile ahead
        if (t + nw < ntiles) tdn = tiles[t + nw];
        const uint32_t lg = td.y & 7u, G = 1u << lg;
        const uint32_t r = td.x + (lane >> lg);
        const uint32_t sub = lane & (G - 1);
        const bool valid = r < nrows;
        uint32_t b = 0, e = 0;
        if (valid) {
            b = __ldg(&ptr[r]);
            e = __ldg(&ptr[r + 1]);
        }
        typename Op::Row rd{};
        if (valid && sub == 0) rd = op.row(r);
        float s = 0.0f, c = 0.0f;
        const uint32_t fs = td.y >> 8;
        if (fs != kNoSeg) {   // one long row: fold its segment sums in order
            if (lane == 0) {
                const uint32_t nseg = (e - b + kTileSeg - 1) / kTileSeg;
                for (uint32_t q = 0; q < nseg; q++) {
                    const float2 pq = segs[fs + q];
                    pair_add(s, c, pq.x, pq.y);
                }
            }
        } else {
            for (uint32_t i = b + sub; i < e; i += G * kTileU) {
                uint32_t j[kTileU];
                float x[kTileU];
#pragma unroll
                for (int u = 0; u < kTileU; u++) {
                    const uint32_t ii = i + u * G;
                    j[u] = ii < e ? __ldg(&idx[ii]) : 0u;
                }
#pragma unroll
                for (int u = 0; u < kTileU; u++) {
                    const uint32_t ii = i + u * G;
                    x[u] = ii < e ? op.term(ii, j[u]) : 0.0f;
                }
#pragma unroll
                for (int u = 0; u < kTileU; u++) two_sum_acc(s, c, x[u]);
            }
            // fixed tree over the row's G lanes (width G keeps groups apart)
            for (uint32_t o = G >> 1; o; o >>= 1) {
                const float s2 = __shfl_down_sync(kFull, s, o, G);
                const float c2 = __shfl_down_sync(kFull, c, o, G);
                pair_add(s, c, s2, c2);
            }
        }
        if (valid && sub == 0) op.finish(r, s, c, rd, res, aux);
    }
    // fixed-order reduction of the FP64 partials: warp tree, then warps in order
    __shared__ double s_dred[2][kBlock / 32];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        res += __shfl_down_sync(kFull, res, o);
        aux += __shfl_down_sync(kFull, aux, o);
    }
    if (lane == 0) {
        s_dred[0][threadIdx.x >> 5] = res;
        s_dred[1][threadIdx.x >> 5] = aux;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        for (int i = 0; i < kBlock / 32; i++) {
            a += s_dred[0][i];
            b += s_dred[1][i];
        }
        partials[2 * blockIdx.x] = a;
        partials[2 * blockIdx.x + 1] = b;
    }
}

// Add the kernels of one tiled row pass (segments, then tiles) to a launch sink.
template <class Op, class Sink>
int tile_pass(const TilePlan &p, Op &op, Sink &&sink) {
    const uint32_t *ptr = p.ptr.as<uint32_t>();
    const uint32_t *idx = p.idx.as<uint32_t>();
    const uint2 *tiles = p.tiles.as<uint2>();
    const uint2 *seg_range = p.seg_range.as<uint2>();
    float2 *segs = p.segs.as<float2>();
    const float2 *csegs = segs;
    double *partials = p.partials.as<double>();
    if (p.nsegs) {
        uint32_t nsegs = p.nsegs;
        void *a_seg[] = {&idx, &seg_range, &nsegs, &op, &segs};
        OLV_TRY(sink((const void *)k_row_segments<Op>,
                     dim3((nsegs + kBlock / 32 - 1) / (kBlock / 32)), dim3(kBlock), a_seg));
    }
    uint32_t ntiles = p.ntiles, n = p.n;
    void *a_t[] = {&ptr, &idx, &tiles, &ntiles, &n, &csegs, &op, &partials};
    OLV_TRY(sink((const void *)k_row_tiles<Op>, dim3(kTileCTAs), dim3(kBlock), a_t));
    return OLV_OK;
}

}  // namespace olv
