// Iterated row sums over a degree-sorted structure, a whole solve in one
// launch: the core of PageRank, weighted PageRank and its adjoint.
//
// The rows (vertices) are renumbered by length, longest first, the neighbour
// ids inside them too (the values most rows gather then sit together at the
// front and stay in L1), and the entries are stored in the order the lanes read
// them.  A tile is 32 / G consecutive rows with G = 1..32 lanes per row (G from
// the row length); its entries are dealt to the lanes step by step and stored
// lane by lane, four steps of a lane together (a unit: 128 places), so that
// every index load of a warp is 512 contiguous bytes whatever the row lengths.
// Rows longer than kRowLong are cut into kRowSeg-entry segments, a tile each;
// the warp that finishes a row's last segment folds them in order.
//
// All iterations run in one launch.  Small structures (at most kClusterRows
// rows and kClusterEntries entries) take one thread-block cluster of 16 CTAs:
// every CTA copies all gathered values to shared memory at the start of an
// iteration (at most 32 KB, contiguous), where 32 gathers take
// 3-4 cycles of bank conflicts instead of 32 lookups in L1, and the barrier
// between two iterations is the cluster's.  Larger ones take the whole GPU (join_team
// below): at the grid barrier the last CTA to arrive adds up the
// FP64 partials in a fixed order and takes the decision for all.  What bounds
// those is the gathers: a 4-byte gather that misses L1 is a request of its own
// to L2 and an SM sends one per cycle, so as many warps as possible keep eight
// gathers per lane in flight, the index loads cost 4 requests per 128 entries,
// and no fence (which would empty L1) stands inside an iteration.
// Measured: PageRank on a uniform digraph of 20,011 vertices, 50 iterations, 600
// -> 374 us; weighted PageRank on RMAT-20, 100 sweeps and their adjoint, 20.2 ->
// 12.7 ms.  A copy of only the most gathered
// values (16 to 217 KB of shared memory) in the whole-GPU form was slower at
// every size: a gather in flight holds a line of L1, which the copy takes away.
//
// Every sum has a fixed evaluation order: lane j of a row's group adds entries
// j, j + G, ... of the row, even and odd steps apart (two packed FP32 adds per
// instruction), with compensated (two-sum) arithmetic, then combines the two and
// a fixed shuffle tree the group's lanes; tiles go to warps by a fixed stride.
//
// An Op supplies:
//   static constexpr bool kGather     entries gather a value of their neighbour
//   static constexpr bool kWeighted   entries carry a weight
//   static constexpr bool kStore      a row yields the value to gather next time; without,
//                                     the solve is one pass (max_it 1) and has no sums
//   double first_aux()                the aux sum before the first iteration
//   void begin(uint32_t it, double aux)   iteration it (from 0) starts; aux: the
//                                     last iteration's aux sum
//   const float *in() / float *out()  gathered values by new id (kGather, kStore)
//   struct Row; Row row(uint32_t r)   per-row inputs of the update
//   float finish(uint32_t r, float s, float c, const Row &q, double &res, double &aux)
//                                     consume the row sum s + c; the value to
//                                     gather next (kStore)
#pragma once
#include <cooperative_groups.h>

#include "olv_internal.cuh"

namespace olv {

// (s, c) <- s + x with the rounding error of the addition accumulated in c.
__device__ __forceinline__ void two_sum_acc(float &s, float &c, float x) {
    const float t = s + x;
    const float bp = t - s;
    c += (s - (t - bp)) + (x - bp);
    s = t;
}

__device__ __forceinline__ void pair_add(float &s, float &c, float s2, float c2) {
    two_sum_acc(s, c, s2);
    c += c2;
}

// Two FP32 values in one 64-bit register and their lane-wise sums: sm_100a's
// packed adds, each half rounded as a scalar add.
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float low2(unsigned long long a) {
    return __uint_as_float((uint32_t)a);
}
__device__ __forceinline__ float high2(unsigned long long a) {
    return __uint_as_float((uint32_t)(a >> 32));
}

// Two compensated sums side by side.
struct Sum2 {
    unsigned long long s, c;
    __device__ __forceinline__ void add(float x, float y) {
        const unsigned long long v = pack2(x, y), t = add2(s, v), bp = sub2(t, s);
        c = add2(c, add2(sub2(s, sub2(t, bp)), sub2(v, bp)));
        s = t;
    }
};

constexpr int kClusterCTAs = 16, kClusterThreads = 1024;
// Structures of at most so many rows and entries take one cluster.  Above, the copy of
// the values and 16 SMs' share of the entries cost more than the grid barrier.
// PageRank / weighted PageRank (forward and adjoint), 20 iterations, us, one cluster
// against the whole GPU: RMAT of 4096 vertices, 53 K edges 157 / 450 against 192 / 490,
// 171 K edges 191 / 528 against 233 / 597; uniform digraphs of 8000 vertices, 32 K edges
// 147 / 384 against 159 / 416, 200 K 174 / 484 against 184 / 461, 391 K 203 / 556 against
// 209 / 524, 1 M 424 / 1090 against 268 / 680; of 30,000 vertices, 210 K edges 210 / 543
// against 179 / 473; of 54,000, 108 K edges 261 / 684 against 175 / 462.
constexpr uint32_t kClusterRows = 8192;       // 32 KB of shared memory
constexpr uint32_t kClusterEntries = 3u << 16;
constexpr uint32_t kRowLong = 2048;    // rows with more entries are segmented
constexpr uint32_t kRowSeg = 512;      // entries per segment
constexpr int kRowClasses = 8;         // segments, 32..1 lanes per row, empty rows
// CTAs per SM: 5 at 48 registers; 6 spill (weighted PageRank, RMAT-20: 13.4 ms
// against 12.7), 4 hide less latency (13.7)
constexpr int kSolveMinBlocks = 5;

// Tiles [tile0[k], tile0[k + 1]) are of class k: 0 segments of the rows
// [0, row0[1]); 1..6 rows from row0[k] on with 32 >> (k - 1) lanes each; 7
// empty rows, 32 per tile.
struct RowClassTable {
    uint32_t tile0[kRowClasses + 1], row0[kRowClasses + 1];
};

struct SolveCtl {
    uint32_t joined;     // CTAs that came before the team was closed (then kTeamClosed is set)
    uint32_t team;       // CTAs of the run, 0 until it is closed
    uint32_t arrive;     // barrier arrivals of the run
    uint32_t go;         // iterations whose barrier is open
    uint32_t err;        // a wait ran out
    uint32_t iter;       // iterations run
    double residual;     // res and aux sums of the last iteration
    double aux;
    unsigned long long count;   // for the Op's start (dangling vertices)
};

struct SolveArgs {
    const uint32_t *units;      // tile -> its first unit (128 places)
    const uint4 *idx;           // unit * 32 + lane: four ids of the lane
    const float4 *w;            // their weights (kWeighted)
    const uint32_t *seg_row, *seg_first;
    float2 *seg_sum;
    uint32_t *seg_done;
    double *partials;           // [2][grid + nlong] (res, aux) pairs, by iteration parity
    SolveCtl *ctl;
    uint32_t nrows, max_it;
    double tol;
    RowClassTable cls;
};

// Reordered structure (device).  perm: new -> old id, newid: old -> new.
struct SolvePlan {
    DevBuf perm, newid, units, idx, pos, seg_row, seg_first, seg_sum, seg_done, partials, ctl;
    RowClassTable cls = {};
    uint32_t n = 0, nlong = 0, nsegs = 0, grid = 1;
    bool cluster = false;       // small: one cluster, else the whole GPU
    uint64_t entries = 0;       // places for entries (units * 128)
    void release() {
        perm.release(); newid.release(); units.release(); idx.release(); pos.release();
        seg_row.release(); seg_first.release(); seg_sum.release(); seg_done.release();
        partials.release(); ctl.release();
    }
    SolveArgs args(uint32_t max_it, double tol, const DevBuf *weights = nullptr) const {
        SolveArgs a = {};
        a.units = units.as<uint32_t>();
        a.idx = idx.as<uint4>();
        if (weights) a.w = weights->as<float4>();
        a.seg_row = seg_row.as<uint32_t>();
        a.seg_first = seg_first.as<uint32_t>();
        a.seg_sum = seg_sum.as<float2>();
        a.seg_done = seg_done.as<uint32_t>();
        a.partials = partials.as<double>();
        a.ctl = ctl.as<SolveCtl>();
        a.nrows = n;
        a.max_it = max_it;
        a.tol = tol;
        a.cls = cls;
        return a;
    }
};

// rowplan.cu.  Rows of a device structure (ptr[n + 1]) by length, longest first,
// equal lengths in the order of their ids: perm, newid (n entries) and the
// offsets in the new order (n + 1).
int sort_rows(const uint32_t *ptr, uint32_t n, cudaStream_t s, uint32_t *perm, uint32_t *newid,
              uint32_t *new_ptr);
// Offsets (n + 1) of the rows perm[0], perm[1], ... of the structure ptr.
int permuted_offsets(const uint32_t *ptr, const uint32_t *perm, uint32_t n, cudaStream_t s,
                     uint32_t *new_ptr);
// Rows longer than bounds[i], i < nb <= 8, of rows sorted by length (sorted_ptr).
int rows_longer(const uint32_t *sorted_ptr, uint32_t n, const uint32_t *bounds, int nb,
                cudaStream_t s, uint32_t *counts);
// Whether a solve plan of n rows and nnz entries takes the lanes_u it is given; smaller
// ones choose their own (at most four entries per lane, or a cluster's).
inline bool solve_lanes_free(uint64_t nnz, uint32_t n, int num_sms) {
    return !(n <= kClusterRows && nnz <= kClusterEntries) &&
           nnz >= (uint64_t)num_sms * kSolveMinBlocks * kBlock * 4;
}
// The whole plan.  lanes_u: entries per lane the grouping aims at (rows get the
// fewest lanes G with G * lanes_u >= length; fewer entries per lane where that
// leaves SMs idle); with_pos: keep each entry's position in the structure
// (eid[position] when eid is set), ~0 for places without an entry, to permute
// weights.
int build_solve_plan(const uint32_t *ptr, const uint32_t *idx, const uint32_t *eid, uint32_t n,
                     uint64_t nnz, uint32_t lanes_u, bool with_pos, int num_sms, cudaStream_t s,
                     SolvePlan &p);

// Whether the stream may use every SM (it does not belong to a green context).
bool stream_has_whole_gpu(cudaStream_t s);

// After a solve of plan p on stream s has ended with control block c.  A run that gave up
// may have left segments counted: the next one starts from zero again.
inline int solve_error(const SolveCtl &c, const SolvePlan &p, cudaStream_t s, const char *what) {
    if (!c.err) return OLV_OK;
    OLV_CUDA(cudaMemsetAsync(p.seg_done.p, 0, (size_t)p.nlong * 4, s));
    set_error("%s: a grid barrier ran out of time", what);
    return OLV_ERR_TIMEOUT;
}

#ifdef __CUDACC__

// Polls allowed in a grid barrier: seconds, far above any iteration.
constexpr uint32_t kBarrierPolls = 1u << 25;

// The CTAs that run a whole-GPU solve: those that are there when it starts.  A grid
// barrier needs every CTA that waits at it to run at once, and on part of a GPU (a
// green context, an MPS share) or beside another stream's kernels the launch may
// not fit.  So a CTA joins by a counter; when all of the grid have joined, or
// kJoinNs after the first, the team is closed, and a CTA that comes later leaves.
// Every member was running when it joined, so the barriers end whatever runs
// beside them.  The grid's shares of the work go to the members in turn and the sums
// of a share have a place of their own, so results do not depend on the team.
// A cooperative launch instead fails where the grid does not fit and waits until
// all of it does.
constexpr uint32_t kTeamClosed = 1u << 31;
constexpr uint64_t kJoinNs = 100000;

// One thread per CTA.  False: too late, or (err set) the wait ran out.
__device__ __forceinline__ bool join_team(SolveCtl *ctl, uint32_t grid, uint32_t &rank,
                                          uint32_t &team) {
    rank = atomicAdd(&ctl->joined, 1u);
    if (rank & kTeamClosed) return false;
    auto close = [&] {
        const uint32_t n = atomicOr(&ctl->joined, kTeamClosed);
        if (!(n & kTeamClosed))
            asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(&ctl->team), "r"(n) : "memory");
    };
    uint64_t start, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
    if (rank + 1 == grid) close();
    for (uint32_t i = 0; i < kBarrierPolls; i++) {
        asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(team) : "l"(&ctl->team) : "memory");
        if (team) return true;
        if (rank == 0) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (now - start >= kJoinNs) close();
        }
        if (i > 64) __nanosleep(64);
    }
    ctl->err = 1;
    return false;
}

// Value of id j, 0 for a place without an entry (id none), by one predicated load:
// no request for such a place, no branch, several in flight.
__device__ __forceinline__ float row_value(const float *in, uint32_t j, uint32_t none) {
    float v;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %1, %2;\n\t"
        "mov.f32 %0, 0f00000000;\n\t"
        "@p ld.global.ca.f32 %0, [%3];\n\t}"
        : "=f"(v)
        : "r"(j), "r"(none), "l"(in + j));
    return v;
}

// kCluster: the launch is one cluster, gathered values in shared memory.
template <class Op, bool kCluster>
__global__ void __launch_bounds__(kCluster ? kClusterThreads : kBlock, kCluster ? 1 : kSolveMinBlocks)
k_row_solve(SolveArgs a, Op op) {
    constexpr int kThreads = kCluster ? kClusterThreads : kBlock, kWarps = kThreads / 32;
    extern __shared__ __align__(16) float s_val[];   // kCluster: values by id, then a zero
    __shared__ double s_red[2][kWarps];
    __shared__ double s_sum[2];
    __shared__ double s_part[2][2];   // kCluster: this CTA's sums, by iteration parity
    __shared__ uint32_t s_state;   // barrier: 0 out of time, 1 open, 2 this CTA is the last
    __shared__ uint32_t s_rank, s_team;   // !kCluster: this CTA in its team, CTAs in it
    __shared__ uint2 s_first[kWarps];     // !kCluster: units of the warps' first tiles
    constexpr unsigned kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t nw = gridDim.x * kWarps;
    const uint32_t ntiles = a.cls.tile0[kRowClasses], nfull = a.cls.tile0[kRowClasses - 1];
    const uint32_t nlong = a.cls.row0[1];
    uint32_t rank = blockIdx.x;
    if constexpr (!kCluster && Op::kStore) {
        if (threadIdx.x == 0) {
            uint32_t r, n = 0;
            s_team = join_team(a.ctl, gridDim.x, r, n) ? n : 0;
            // a full team by CTA number: neighbours are on different SMs, so each SM gets
            // its share of the CTAs with a tile more (by order of arrival: 5-9 % slower)
            s_rank = n == gridDim.x ? blockIdx.x : r;
        }
        __syncthreads();
        if (s_team == 0) return;
        rank = s_rank;
    }
    double sum_res = 0, sum_aux = op.first_aux();
    uint32_t it = 0;
    // the first tile's units (the same in every iteration); kCluster: the ids of a
    // tile's first two units are loaded while the tile before it is summed, those
    // of the first tile before the barrier
    uint32_t first_u = 0, first_ue = 0;
    if (rank * kWarps + wid < nfull) {
        first_u = __ldg(&a.units[rank * kWarps + wid]);
        first_ue = __ldg(&a.units[rank * kWarps + wid + 1]);
    }
    if constexpr (!kCluster) s_first[wid] = make_uint2(first_u, first_ue);   // not in registers
    __syncwarp();
    const uint4 none4 = make_uint4(a.nrows, a.nrows, a.nrows, a.nrows);
    auto ids = [&](uint32_t x, uint32_t end) {
        return x < end ? __ldg(&a.idx[(size_t)x * 32 + lane]) : none4;
    };
    uint4 k0 = none4, k1 = none4;
    if constexpr (Op::kGather && kCluster) {
        k0 = ids(first_u, first_ue);
        k1 = ids(first_u + 1, first_ue);
    }
    while (it < a.max_it) {
        op.begin(it, sum_aux);
        const float *in = nullptr;
        if constexpr (Op::kGather) in = op.in();
        if constexpr (Op::kGather && kCluster) {
            const float4 *in4 = reinterpret_cast<const float4 *>(in);
            for (uint32_t b = 0; b < a.nrows / 4; b += 4 * kThreads) {   // four in flight
                float4 v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t i = b + q * kThreads + threadIdx.x;
                    if (i < a.nrows / 4) v[q] = __ldcg(&in4[i]);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t i = b + q * kThreads + threadIdx.x;
                    if (i < a.nrows / 4) reinterpret_cast<float4 *>(s_val)[i] = v[q];
                }
            }
            for (uint32_t i = (a.nrows & ~3u) + threadIdx.x; i <= a.nrows; i += kThreads)
                s_val[i] = i < a.nrows ? __ldcg(&in[i]) : 0.0f;
            __syncthreads();
        }
        double *part = a.partials + (size_t)(it & 1) * 2 * (gridDim.x + nlong);
        auto end_row = [&](uint32_t r, float s, float c, const typename Op::Row &rd, double &rr,
                           double &ra) {
            const float v = op.finish(r, s, c, rd, rr, ra);
            if constexpr (Op::kStore) op.out()[r] = v;
        };
        // the CTA's sums: a tree over each warp, then over the warps
        auto cta_sum = [&](double &x, double &y) {
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                x += __shfl_down_sync(kFull, x, o);
                y += __shfl_down_sync(kFull, y, o);
            }
            if (lane == 0) {
                s_red[0][wid] = x;
                s_red[1][wid] = y;
            }
            __syncthreads();
            if (wid == 0) {   // lane 0 gets the sums
                x = lane < kWarps ? s_red[0][lane] : 0.0;
                y = lane < kWarps ? s_red[1][lane] : 0.0;
#pragma unroll
                for (int o = kWarps / 2; o; o >>= 1) {
                    x += __shfl_down_sync(kFull, x, o);
                    y += __shfl_down_sync(kFull, y, o);
                }
            }
        };
        // this CTA's shares of the grid's work (one, in a full team)
        double res, aux;
        for (uint32_t share = rank;;) {
            const uint32_t gw = share * kWarps + wid;
            res = 0;
            aux = 0;
            uint32_t k = 0;   // class of tile t
            uint32_t u = first_u, ue = first_ue;
            if constexpr (!kCluster) {
                u = s_first[wid].x;
                ue = s_first[wid].y;
                if (Op::kStore && share >= s_team && gw < nfull) {   // not this CTA's first share
                    u = __ldg(&a.units[gw]);
                    ue = __ldg(&a.units[gw + 1]);
                }
            }
            for (uint32_t t = gw; t < nfull; t += nw) {
                while (t >= a.cls.tile0[k + 1]) k++;
                const uint32_t lg = k == 0 ? 5 : 6 - k;
                const uint32_t G = 1u << lg;
                uint32_t r;
                bool mine;
                if (k == 0) {
                    r = __ldg(&a.seg_row[t]);
                    mine = false;
                } else {
                    r = a.cls.row0[k] + (((t - a.cls.tile0[k]) << 5) >> lg) + (lane >> lg);
                    mine = r < a.cls.row0[k + 1] && (lane & (G - 1)) == 0;
                }
                typename Op::Row rd{};
                if (mine) rd = op.row(r);
                uint32_t nu = 0, nue = 0;   // the next tile's units, one tile ahead
                if (t + (uint64_t)nw < nfull) {
                    nu = __ldg(&a.units[t + nw]);
                    nue = __ldg(&a.units[t + nw + 1]);
                }
                uint4 n0 = none4, n1 = none4;
                if constexpr (Op::kGather && kCluster) {
                    const bool wrap = t + (uint64_t)nw >= nfull;
                    const uint32_t x = wrap ? first_u : nu, xe = wrap ? first_ue : nue;
                    n0 = ids(x, xe);
                    n1 = ids(x + 1, xe);
                }
                Sum2 acc{0, 0};
                for (; u < ue; u += 2) {   // two units: eight gathers in flight
                    const bool two = u + 1 < ue;   // the same in the whole warp
                    const size_t at = (size_t)u * 32 + lane;
                    float x[8];
                    float4 w0, w1;
                    if constexpr (Op::kGather && kCluster) {
                        const uint4 j0 = k0, j1 = k1;
                        k0 = ids(u + 2, ue);
                        k1 = ids(u + 3, ue);
                        x[0] = s_val[j0.x];
                        x[1] = s_val[j0.y];
                        x[2] = s_val[j0.z];
                        x[3] = s_val[j0.w];
                        x[4] = s_val[j1.x];
                        x[5] = s_val[j1.y];
                        x[6] = s_val[j1.z];
                        x[7] = s_val[j1.w];
                    } else if constexpr (Op::kGather) {
                        const uint4 j0 = __ldcs(&a.idx[at]);
                        uint4 j1 = none4;
                        if (two) j1 = __ldcs(&a.idx[at + 32]);
                        x[0] = row_value(in, j0.x, a.nrows);
                        x[1] = row_value(in, j0.y, a.nrows);
                        x[2] = row_value(in, j0.z, a.nrows);
                        x[3] = row_value(in, j0.w, a.nrows);
                        if (two) {
                            x[4] = row_value(in, j1.x, a.nrows);
                            x[5] = row_value(in, j1.y, a.nrows);
                            x[6] = row_value(in, j1.z, a.nrows);
                            x[7] = row_value(in, j1.w, a.nrows);
                        }
                    }
                    if constexpr (Op::kWeighted) {
                        w0 = __ldcs(&a.w[at]);
                        if (two) w1 = __ldcs(&a.w[at + 32]);
                    }
                    auto add4 = [&](const float *v, const float4 &w) {
                        if constexpr (Op::kGather && Op::kWeighted) {
                            acc.add(v[0] * w.x, v[1] * w.y);
                            acc.add(v[2] * w.z, v[3] * w.w);
                        } else if constexpr (Op::kWeighted) {
                            acc.add(w.x, w.y);
                            acc.add(w.z, w.w);
                        } else {
                            acc.add(v[0], v[1]);
                            acc.add(v[2], v[3]);
                        }
                    };
                    add4(x, w0);
                    if (two) add4(x + 4, w1);
                }
                u = nu;
                ue = nue;
                if constexpr (Op::kGather && kCluster) {
                    k0 = n0;
                    k1 = n1;
                }
                // even and odd steps, then a fixed tree over the row's G lanes
                float s = low2(acc.s), c = low2(acc.c);
                pair_add(s, c, high2(acc.s), high2(acc.c));
                for (uint32_t o = G >> 1; o; o >>= 1) {
                    const float s2 = __shfl_down_sync(kFull, s, o, G);
                    const float c2 = __shfl_down_sync(kFull, c, o, G);
                    pair_add(s, c, s2, c2);
                }
                if (k != 0) {
                    if (mine) end_row(r, s, c, rd, res, aux);
                    continue;
                }
                // a segment: the last one of its row to finish folds them, lane l
                // segments l, l + 32, ..., then a fixed tree; the row's partials have
                // a place of their own (which warp is last is not fixed)
                const uint32_t first = __ldg(&a.seg_first[r]);
                const uint32_t nseg = __ldg(&a.seg_first[r + 1]) - first;
                uint32_t last = 0;
                if (lane == 0) {
                    // released by the count itself: a full fence would empty this SM's
                    // L1 at every segment; only the last segment's warp acquires
                    __stcg(&a.seg_sum[t], make_float2(s, c));
                    asm volatile("atom.release.gpu.global.inc.u32 %0, [%1], %2;"
                                 : "=r"(last)
                                 : "l"(&a.seg_done[r]), "r"(nseg - 1)
                                 : "memory");
                    last = last == nseg - 1;
                    if (last) __threadfence();
                }
                if (!__shfl_sync(kFull, last, 0)) continue;
                __syncwarp();   // lane 0 acquired; a shuffle orders no memory for the others
                s = 0.0f;
                c = 0.0f;
                for (uint32_t q = lane; q < nseg; q += 32) {
                    const float2 v = __ldcg(&a.seg_sum[first + q]);
                    pair_add(s, c, v.x, v.y);
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    const float s2 = __shfl_down_sync(kFull, s, o);
                    const float c2 = __shfl_down_sync(kFull, c, o);
                    pair_add(s, c, s2, c2);
                }
                if (lane == 0) {
                    double rr = 0, ra = 0;
                    end_row(r, s, c, op.row(r), rr, ra);
                    part[2 * (gridDim.x + r)] = rr;
                    part[2 * (gridDim.x + r) + 1] = ra;
                }
            }
            // rows without entries, 32 per tile
            for (uint32_t t = nfull + gw; t < ntiles; t += nw) {
                const uint32_t r = a.cls.row0[kRowClasses - 1] + (t - nfull) * 32 + lane;
                if (r < a.nrows) end_row(r, 0.0f, 0.0f, op.row(r), res, aux);
            }
            if constexpr (!Op::kStore) return;   // one pass: no barrier, no sums
            cta_sum(res, aux);
            if constexpr (kCluster) break;
            if (threadIdx.x == 0) {
                part[2 * share] = res;
                part[2 * share + 1] = aux;
            }
            share += s_team;
            if (share >= gridDim.x) break;
            __syncthreads();
        }
        it++;
        if constexpr (kCluster) {
            cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
            double(&mine)[2] = s_part[it & 1];
            if (threadIdx.x == 0) {
                mine[0] = res;
                mine[1] = aux;
            }
            cl.sync();
            // every CTA adds the CTAs' sums and the long rows' in the same order
            if (wid == 0) {
                double x = 0, y = 0;
                if (lane < gridDim.x) {
                    const double *p = cl.map_shared_rank(&mine[0], lane);
                    x = p[0];
                    y = p[1];
                }
                for (uint32_t i = lane; i < nlong; i += 32) {
                    x += __ldcg(&part[2 * (gridDim.x + i)]);
                    y += __ldcg(&part[2 * (gridDim.x + i) + 1]);
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    x += __shfl_xor_sync(kFull, x, o);
                    y += __shfl_xor_sync(kFull, y, o);
                }
                if (lane == 0) {
                    s_sum[0] = x;
                    s_sum[1] = y;
                }
            }
            __syncthreads();
            sum_res = s_sum[0];
            sum_aux = s_sum[1];
            if (sum_res < a.tol) break;
            continue;
        }
        // grid barrier: the last CTA to arrive folds all partials in a fixed order
        // and opens it
        if (threadIdx.x == 0) {
            __threadfence();
            const uint32_t before = atomicAdd(&a.ctl->arrive, 1u);
            s_state = before + 1 == it * s_team ? 2 : 1;
            __threadfence();
        }
        __syncthreads();
        if (s_state == 2) {
            double x = 0, y = 0;
            for (uint32_t i = threadIdx.x; i < gridDim.x + nlong; i += kThreads) {
                x += __ldcg(&part[2 * i]);
                y += __ldcg(&part[2 * i + 1]);
            }
            cta_sum(x, y);
            if (threadIdx.x == 0) {
                s_sum[0] = x;
                s_sum[1] = y;
                a.ctl->residual = x;
                a.ctl->aux = y;
                a.ctl->iter = it;
                __threadfence();
                asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(&a.ctl->go), "r"(it) : "memory");
            }
        } else if (threadIdx.x == 0) {
            uint32_t ok = 0;
            for (uint32_t i = 0; i < kBarrierPolls; i++) {
                uint32_t v;
                asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(&a.ctl->go) : "memory");
                if (v == it) {
                    ok = 1;
                    break;
                }
                if (i > 256) __nanosleep(64);
            }
            __threadfence();
            if (ok) {
                s_sum[0] = __ldcg(&a.ctl->residual);
                s_sum[1] = __ldcg(&a.ctl->aux);
            } else {
                a.ctl->err = 1;
                s_state = 0;
            }
        }
        __syncthreads();
        if (s_state == 0) return;
        sum_res = s_sum[0];
        sum_aux = s_sum[1];
        if (sum_res < a.tol) break;
    }
    if constexpr (kCluster) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.ctl->iter = it;
            a.ctl->residual = sum_res;
            a.ctl->aux = sum_aux;
        }
        cooperative_groups::this_cluster().sync();   // no CTA leaves while its sums are read
    }
}

inline void cluster_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr, size_t smem,
                           cudaStream_t s) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterCTAs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(kClusterCTAs);
    cfg->blockDim = dim3(kClusterThreads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = s;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
}

// Whether the GPU runs the cluster form of Op at its largest.  (Its shared memory stays
// below the 48 KB that need no attribute: one set to each handle's size belongs to the
// kernel, and threads undid each other's.)
template <class Op>
bool cluster_runs() {
    const void *fn = (const void *)k_row_solve<Op, true>;
    constexpr size_t smem = Op::kGather ? (kClusterRows + 4) * 4 : 0;
    static_assert(smem <= 47 * 1024, "one set of launch attributes for all plans");
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    cluster_config(&cfg, attr, smem, nullptr);
    int n = 0;
    const bool ok =
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= 1;
    if (!ok) cudaGetLastError();
    return ok;
}

// The form a plan's solves take, decided once, when it is built: a cluster where the
// plan is small and the GPU runs one for every Op it is used with.
template <class... Ops>
void choose_form(SolvePlan &p) {
    if (p.cluster) p.cluster = (cluster_runs<Ops>() && ...);
}

// Launch a solve.  *ctl must be zero but for count.  Part of a GPU may have no 16 SMs
// that can hold a cluster: a small plan takes the other form there.
template <class Op>
int launch_solve(const SolvePlan &p, SolveArgs a, Op op, cudaStream_t s) {
    if (p.cluster && stream_has_whole_gpu(s)) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        cluster_config(&cfg, attr, Op::kGather ? ((size_t)p.n + 4) * 4 : 0, s);
        OLV_CUDA(cudaLaunchKernelEx(&cfg, k_row_solve<Op, true>, a, op));
        return OLV_OK;
    }
    k_row_solve<Op, false><<<p.grid, kBlock, 0, s>>>(a, op);
    OLV_CUDA(cudaGetLastError());
    return OLV_OK;
}

#endif
}  // namespace olv
