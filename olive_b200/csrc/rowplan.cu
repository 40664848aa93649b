// Row orders and solve plans, built on the device (olv_rowsolve.cuh): sorting
// rows by length and laying the entries out in the order the lanes read them.
#include <algorithm>
#include <vector>

#include <cub/cub.cuh>

#include "olv_driver.h"
#include "olv_rowsolve.cuh"
#include "olv_rowtiles.cuh"

namespace olv {

namespace {

constexpr int kPlanBlocks = 148 * 8;

__global__ void k_row_lengths(const uint32_t *__restrict__ ptr, uint32_t n,
                              uint32_t *__restrict__ len, uint32_t *__restrict__ id) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x) {
        len[v] = ptr[v + 1] - ptr[v];
        if (id) id[v] = (uint32_t)v;
    }
}

__global__ void k_lengths_of(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ row,
                             uint32_t n, uint32_t *__restrict__ len) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = row[i];
        len[i] = ptr[r + 1] - ptr[r];
    }
}

struct Bounds {
    uint32_t x[8];
};

// counts[i]: the first row of at most b.x[i] entries (rows sorted, longest first).
__global__ void k_rows_longer(const uint32_t *__restrict__ ptr, uint32_t n, Bounds b, int nb,
                              uint32_t *__restrict__ counts) {
    const int i = threadIdx.x;
    if (i >= nb) return;
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (ptr[mid + 1] - ptr[mid] > b.x[i])
            lo = mid + 1;
        else
            hi = mid;
    }
    counts[i] = lo;
}

__global__ void k_inverse(const uint32_t *__restrict__ perm, uint32_t n,
                          uint32_t *__restrict__ newid) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        newid[perm[i]] = (uint32_t)i;
}

// Class of a row by its length (RowClassTable): 0 segmented, 1..6 for 32..1
// lanes, 7 empty.
__host__ __device__ __forceinline__ uint32_t row_class(uint32_t len, uint32_t lanes_u) {
    if (len == 0) return kRowClasses - 1;
    if (len > kRowLong) return 0;
    uint32_t lg = 0;
    while (lg < 5 && (1u << lg) * lanes_u < len) lg++;
    return 6 - lg;
}

// Rows are sorted by length, longest first, so classes are ranges: a row whose
// class differs from its predecessor's begins one (and the classes skipped).
__global__ void k_class_starts(const uint32_t *__restrict__ ptr, uint32_t n, uint32_t lanes_u,
                               uint32_t *__restrict__ row0) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n;
         r += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t k = row_class(ptr[r + 1] - ptr[r], lanes_u);
        const uint32_t before = r ? row_class(ptr[r] - ptr[r - 1], lanes_u) : 0u;
        for (uint32_t j = before + 1; j <= k; j++) row0[j] = (uint32_t)r;
        if (r + 1 == n)
            for (uint32_t j = k + 1; j <= kRowClasses; j++) row0[j] = n;
    }
}

struct PlanView {
    RowClassTable c;
    const uint32_t *ptr;                  // old structure
    const uint32_t *idx, *eid;
    const uint32_t *perm, *newid;
    const uint32_t *seg_row, *seg_first;
};

// Entries [b, e) of the old structure that row i (of its 32 / G) of tile t holds.
__device__ __forceinline__ void tile_row(const PlanView &p, uint32_t t, uint32_t k, uint32_t i,
                                         uint32_t &b, uint32_t &e) {
    b = e = 0;
    if (k == 0) {
        const uint32_t r = p.seg_row[t], v = p.perm[r];
        b = p.ptr[v] + (t - p.seg_first[r]) * kRowSeg;
        e = p.ptr[v + 1] - b > kRowSeg ? b + kRowSeg : p.ptr[v + 1];
    } else {
        const uint32_t lg = 6 - k;
        const uint32_t r = p.c.row0[k] + (((t - p.c.tile0[k]) << 5) >> lg) + i;
        if (r < p.c.row0[k + 1]) {
            const uint32_t v = p.perm[r];
            b = p.ptr[v];
            e = p.ptr[v + 1];
        }
    }
}

// Units of every tile with entries: its first row is its longest.
__global__ void k_tile_units(PlanView p, uint32_t *__restrict__ units) {
    const uint32_t nfull = p.c.tile0[kRowClasses - 1];
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t <= nfull;
         t += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t u = 0;
        if (t < nfull) {
            uint32_t k = 0, b, e;
            while (t >= p.c.tile0[k + 1]) k++;
            tile_row(p, (uint32_t)t, k, 0, b, e);
            const uint32_t per = 4u << (k == 0 ? 5 : 6 - k);
            u = (e - b + per - 1) / per;
        }
        units[t] = u;
    }
}

// The entries of every tile, one warp per tile: place 4u + q of lane l is entry
// (4u + q) G + l % G of the lane's row; places past the row's end hold id none.
__global__ void k_fill_tiles(PlanView p, const uint32_t *__restrict__ units, uint32_t none,
                             uint4 *__restrict__ idx, uint4 *__restrict__ pos) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nfull = p.c.tile0[kRowClasses - 1];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = warp; t < nfull; t += nwarps) {
        uint32_t k = 0, b, e;
        while (t >= p.c.tile0[k + 1]) k++;
        const uint32_t lg = k == 0 ? 5 : 6 - k, sub = lane & ((1u << lg) - 1u);
        tile_row(p, t, k, lane >> lg, b, e);
        const uint32_t u0 = units[t], u1 = units[t + 1];
        for (uint32_t u = u0; u < u1; u++) {
            uint32_t id[4], ps[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint64_t x = (uint64_t)b + (((uint64_t)(4 * (u - u0) + q)) << lg) + sub;
                id[q] = none;
                ps[q] = 0xffffffffu;
                if (x < e) {
                    id[q] = p.newid[p.idx[x]];
                    ps[q] = p.eid ? p.eid[x] : (uint32_t)x;
                }
            }
            idx[(size_t)u * 32 + lane] = make_uint4(id[0], id[1], id[2], id[3]);
            if (pos) pos[(size_t)u * 32 + lane] = make_uint4(ps[0], ps[1], ps[2], ps[3]);
        }
    }
}

// idx[ptr[i] + k] = newid[old_idx[old_ptr[perm[i]] + k]], one warp per row.
__global__ void k_relabel_rows(const uint32_t *__restrict__ old_ptr,
                               const uint32_t *__restrict__ old_idx,
                               const uint32_t *__restrict__ perm,
                               const uint32_t *__restrict__ newid,
                               const uint32_t *__restrict__ ptr, uint32_t n,
                               uint32_t *__restrict__ idx) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = w; i < n; i += nw) {
        const uint32_t v = perm[i];
        const uint32_t b = old_ptr[v], e = old_ptr[v + 1], o = ptr[i];
        for (uint32_t k = lane; k < e - b; k += 32) idx[o + k] = newid[old_idx[b + k]];
    }
}

// Tiles [tile0, tile0 + n) of one class: rows from row0 on, 32 >> lg each.
__global__ void k_class_tiles(uint2 *__restrict__ tiles, uint32_t tile0, uint32_t n, uint32_t row0,
                              uint32_t lg) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
        tiles[tile0 + t] = make_uint2(row0 + t * (32u >> lg), lg | (kNoSeg << 8));
}

int sort_desc(const uint32_t *key, uint32_t *key_out, const uint32_t *val, uint32_t *val_out,
              uint32_t n, cudaStream_t s) {
    size_t tb = 0;
    OLV_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, key, key_out, val, val_out,
                                                       (int64_t)n, 0, 32, s));
    DevBuf temp;
    OLV_TRY(temp.ensure(tb));
    OLV_CUDA(cub::DeviceRadixSort::SortPairsDescending(temp.p, tb, key, key_out, val, val_out,
                                                       (int64_t)n, 0, 32, s));
    OLV_CUDA(cudaStreamSynchronize(s));   // the scratch dies here
    return OLV_OK;
}

int exclusive_scan(const uint32_t *in, uint32_t *out, uint64_t n, cudaStream_t s) {
    size_t tb = 0;
    OLV_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, (int64_t)n, s));
    DevBuf temp;
    OLV_TRY(temp.ensure(tb));
    OLV_CUDA(cub::DeviceScan::ExclusiveSum(temp.p, tb, in, out, (int64_t)n, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    return OLV_OK;
}

}  // namespace

int sort_rows(const uint32_t *ptr, uint32_t n, cudaStream_t s, uint32_t *perm, uint32_t *newid,
              uint32_t *new_ptr) {
    DevBuf len, id, sorted;
    OLV_TRY(len.ensure((size_t)n * 4 + 16));
    OLV_TRY(id.ensure((size_t)n * 4 + 16));
    OLV_TRY(sorted.ensure(((size_t)n + 1) * 4 + 16));
    k_row_lengths<<<kPlanBlocks, kBlock, 0, s>>>(ptr, n, len.as<uint32_t>(), id.as<uint32_t>());
    // stable: equal lengths keep the order of their ids
    OLV_TRY(sort_desc(len.as<uint32_t>(), sorted.as<uint32_t>(), id.as<uint32_t>(), perm, n, s));
    k_inverse<<<kPlanBlocks, kBlock, 0, s>>>(perm, n, newid);
    OLV_CUDA(cudaMemsetAsync(sorted.as<uint32_t>() + n, 0, 4, s));
    OLV_TRY(exclusive_scan(sorted.as<uint32_t>(), new_ptr, (uint64_t)n + 1, s));
    OLV_CUDA(cudaGetLastError());
    return OLV_OK;
}

int permuted_offsets(const uint32_t *ptr, const uint32_t *perm, uint32_t n, cudaStream_t s,
                     uint32_t *new_ptr) {
    DevBuf len;
    OLV_TRY(len.ensure(((size_t)n + 1) * 4));
    OLV_CUDA(cudaMemsetAsync(len.as<uint32_t>() + n, 0, 4, s));
    k_lengths_of<<<kPlanBlocks, kBlock, 0, s>>>(ptr, perm, n, len.as<uint32_t>());
    OLV_TRY(exclusive_scan(len.as<uint32_t>(), new_ptr, (uint64_t)n + 1, s));
    OLV_CUDA(cudaGetLastError());
    return OLV_OK;
}

int rows_longer(const uint32_t *sorted_ptr, uint32_t n, const uint32_t *bounds, int nb,
                cudaStream_t s, uint32_t *counts) {
    DevBuf d;
    OLV_TRY(d.ensure(32));
    Bounds b = {};
    std::copy(bounds, bounds + nb, b.x);
    k_rows_longer<<<1, 32, 0, s>>>(sorted_ptr, n, b, nb, d.as<uint32_t>());
    OLV_CUDA(cudaMemcpyAsync(counts, d.p, (size_t)nb * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    return OLV_OK;
}

bool stream_has_whole_gpu(cudaStream_t s) {
    static const auto green = driver_entry<PFN_cuStreamGetGreenCtx_v12040>("cuStreamGetGreenCtx", 12040);
    CUgreenCtx c = nullptr;
    return !green || green(s, &c) != CUDA_SUCCESS || !c;
}

// First row of every class (RowClassTable::row0) of the sorted rows sptr.
static int class_rows(const uint32_t *sptr, uint32_t n, uint32_t lanes_u, cudaStream_t s,
                      uint32_t (&rows)[kRowClasses + 1]) {
    DevBuf row0;
    OLV_TRY(row0.ensure((kRowClasses + 1) * 4));
    OLV_CUDA(cudaMemsetAsync(row0.p, 0, (kRowClasses + 1) * 4, s));
    k_class_starts<<<kPlanBlocks, kBlock, 0, s>>>(sptr, n, lanes_u, row0.as<uint32_t>());
    OLV_CUDA(cudaMemcpyAsync(rows, row0.p, (kRowClasses + 1) * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    return OLV_OK;
}

static_assert(kTileLong == kRowLong, "the row classes serve both layouts");

int build_tile_plan(const uint32_t *ptr_dev, const uint32_t *idx_dev, uint32_t n, cudaStream_t s,
                    TilePlan &p, uint32_t lanes_u) {
    p.n = n;
    OLV_TRY(p.perm.ensure((size_t)n * 4 + 16));
    OLV_TRY(p.newid.ensure((size_t)n * 4 + 16));
    OLV_TRY(p.ptr.ensure(((size_t)n + 1) * 4 + 16));
    OLV_TRY(sort_rows(ptr_dev, n, s, p.perm.as<uint32_t>(), p.newid.as<uint32_t>(),
                      p.ptr.as<uint32_t>()));
    uint32_t row0[kRowClasses + 1];
    OLV_TRY(class_rows(p.ptr.as<uint32_t>(), n, lanes_u, s, row0));
    const uint32_t nlong = row0[1];
    std::vector<uint32_t> lp((size_t)nlong + 1);
    uint32_t E = 0;
    OLV_CUDA(cudaMemcpyAsync(lp.data(), p.ptr.p, lp.size() * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaMemcpyAsync(&E, p.ptr.as<uint32_t>() + n, 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    std::vector<uint2> ltiles, ranges;
    for (uint32_t r = 0; r < nlong; r++) {
        ltiles.push_back(make_uint2(r, 5u | ((uint32_t)ranges.size() << 8)));
        for (uint32_t x = lp[r]; x < lp[r + 1];) {
            const uint32_t e = lp[r + 1] - x > kTileSeg ? x + kTileSeg : lp[r + 1];
            ranges.push_back(make_uint2(x, e));
            x = e;
        }
    }
    if (ranges.size() >= kNoSeg) {
        set_error("row plan: %zu segments exceed the tile format", ranges.size());
        return OLV_ERR_LIMIT;
    }
    // a tile's lanes per row are those of its first row's class: the last tile of
    // a class may go on into the next one, whose tiles begin behind it
    uint32_t first[kRowClasses], count[kRowClasses], tiles = nlong, at = nlong;
    for (int k = 1; k < kRowClasses; k++) {
        const uint32_t per = k == kRowClasses - 1 ? 32u : 32u >> (6 - k);
        first[k] = at;
        count[k] = at < row0[k + 1] ? (row0[k + 1] - at + per - 1) / per : 0;
        at += count[k] * per;
        tiles += count[k];
    }
    p.ntiles = tiles;
    p.nsegs = (uint32_t)ranges.size();
    OLV_TRY(p.idx.ensure((size_t)E * 4 + 16));
    OLV_TRY(p.tiles.ensure((size_t)tiles * 8 + 16));
    OLV_TRY(p.seg_range.ensure(ranges.size() * 8 + 16));
    OLV_TRY(p.segs.ensure(ranges.size() * 8 + 16));
    OLV_TRY(p.partials.ensure((size_t)kTileCTAs * 16 + 16));
    if (nlong) {
        OLV_CUDA(cudaMemcpyAsync(p.tiles.p, ltiles.data(), (size_t)nlong * 8,
                                 cudaMemcpyHostToDevice, s));
        OLV_CUDA(cudaMemcpyAsync(p.seg_range.p, ranges.data(), ranges.size() * 8,
                                 cudaMemcpyHostToDevice, s));
    }
    uint32_t t0 = nlong;
    for (int k = 1; k < kRowClasses; k++) {
        if (!count[k]) continue;
        k_class_tiles<<<kPlanBlocks, kBlock, 0, s>>>(p.tiles.as<uint2>(), t0, count[k], first[k],
                                                     k == kRowClasses - 1 ? 0u : 6u - k);
        t0 += count[k];
    }
    k_relabel_rows<<<kPlanBlocks, kBlock, 0, s>>>(ptr_dev, idx_dev, p.perm.as<uint32_t>(),
                                                 p.newid.as<uint32_t>(), p.ptr.as<uint32_t>(), n,
                                                 p.idx.as<uint32_t>());
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaStreamSynchronize(s));   // the host vectors die here
    return OLV_OK;
}

int build_solve_plan(const uint32_t *ptr, const uint32_t *idx, const uint32_t *eid, uint32_t n,
                     uint64_t nnz, uint32_t lanes_u, bool with_pos, int num_sms, cudaStream_t s,
                     SolvePlan &p) {
    p.n = n;
    p.cluster = n <= kClusterRows && nnz <= kClusterEntries;
    // entries per lane: one cluster's warps are best off with a tile each (a tile
    // costs about 250 instructions beside its entries'); the whole GPU's with four
    // entries per lane where eight would leave most without a tile
    if (p.cluster) {
        lanes_u = 4;
        while (lanes_u < 16 && (uint64_t)lanes_u * kClusterCTAs * kClusterThreads < nnz) lanes_u *= 2;
    } else if (lanes_u > 4 && !solve_lanes_free(nnz, n, num_sms)) {
        lanes_u = 4;
    }
    DevBuf sptr;
    OLV_TRY(p.perm.ensure((size_t)n * 4 + 16));
    OLV_TRY(p.newid.ensure((size_t)n * 4 + 16));
    OLV_TRY(sptr.ensure(((size_t)n + 1) * 4 + 16));
    OLV_TRY(sort_rows(ptr, n, s, p.perm.as<uint32_t>(), p.newid.as<uint32_t>(),
                      sptr.as<uint32_t>()));
    RowClassTable &c = p.cls;
    OLV_TRY(class_rows(sptr.as<uint32_t>(), n, lanes_u, s, c.row0));
    // segments of the long rows
    p.nlong = c.row0[1];
    std::vector<uint32_t> lp((size_t)p.nlong + 1), first((size_t)p.nlong + 1, 0), seg_row;
    OLV_CUDA(cudaMemcpyAsync(lp.data(), sptr.p, lp.size() * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    for (uint32_t r = 0; r < p.nlong; r++) {
        first[r] = (uint32_t)seg_row.size();
        const uint32_t ns = (lp[r + 1] - lp[r] + kRowSeg - 1) / kRowSeg;
        seg_row.insert(seg_row.end(), ns, r);
    }
    first[p.nlong] = p.nsegs = (uint32_t)seg_row.size();
    OLV_TRY(p.seg_row.ensure(seg_row.size() * 4 + 16));
    OLV_TRY(p.seg_first.ensure(first.size() * 4 + 16));
    OLV_TRY(p.seg_sum.ensure(seg_row.size() * 8 + 16));
    OLV_TRY(p.seg_done.ensure((size_t)p.nlong * 4 + 16));
    if (p.nsegs)
        OLV_CUDA(cudaMemcpyAsync(p.seg_row.p, seg_row.data(), seg_row.size() * 4,
                                 cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaMemcpyAsync(p.seg_first.p, first.data(), first.size() * 4, cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaMemsetAsync(p.seg_done.p, 0, (size_t)p.nlong * 4 + 16, s));
    // tiles
    c.tile0[0] = 0;
    c.tile0[1] = p.nsegs;
    for (int k = 1; k < kRowClasses; k++) {
        const uint32_t rows = c.row0[k + 1] - c.row0[k];
        const uint32_t per = k == kRowClasses - 1 ? 32 : 32u >> (6 - k);
        c.tile0[k + 1] = c.tile0[k] + (rows + per - 1) / per;
    }
    const uint32_t nfull = c.tile0[kRowClasses - 1], ntiles = c.tile0[kRowClasses];
    p.grid = std::max(1u, std::min((uint32_t)(num_sms * kSolveMinBlocks),
                                   (ntiles + kBlock / 32 - 1) / (kBlock / 32)));
    const PlanView v = {c, ptr, idx, eid, p.perm.as<uint32_t>(), p.newid.as<uint32_t>(),
                        p.seg_row.as<uint32_t>(), p.seg_first.as<uint32_t>()};
    DevBuf nu;
    OLV_TRY(nu.ensure(((size_t)nfull + 1) * 4));
    OLV_TRY(p.units.ensure(((size_t)nfull + 1) * 4 + 16));
    k_tile_units<<<kPlanBlocks, kBlock, 0, s>>>(v, nu.as<uint32_t>());
    OLV_TRY(exclusive_scan(nu.as<uint32_t>(), p.units.as<uint32_t>(), (uint64_t)nfull + 1, s));
    uint32_t units = 0;
    OLV_CUDA(cudaMemcpyAsync(&units, p.units.as<uint32_t>() + nfull, 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    p.entries = (uint64_t)units * 128;
    OLV_TRY(p.idx.ensure(p.entries * 4 + 16));
    if (with_pos) OLV_TRY(p.pos.ensure(p.entries * 4 + 16));
    k_fill_tiles<<<kPlanBlocks * 2, kBlock, 0, s>>>(v, p.units.as<uint32_t>(), n, p.idx.as<uint4>(),
                                                   with_pos ? p.pos.as<uint4>() : nullptr);
    OLV_TRY(p.partials.ensure(4 * ((size_t)std::max(p.grid, (uint32_t)kClusterCTAs) + p.nlong) * 8 + 16));
    OLV_TRY(p.ctl.ensure(sizeof(SolveCtl)));
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaStreamSynchronize(s));   // the host vectors and scratch die here
    return OLV_OK;
}

}  // namespace olv
