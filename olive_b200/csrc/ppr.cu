// K personalised PageRank vectors on a general graph, advanced together as a
// sparse x dense-K product (no reference counterpart; each vector follows
// PageRank.cu:51-75 with the teleport to its own seed).
//
// Result contract, per vector k with seed s_k (K <= 32), from r_k = e_{s_k}:
//   r_k'[v] = alpha * (sum_{u->v} r_k[u] / outdeg(u)) + [v == s_k] * ((1-alpha) + alpha * d_k)
// with d_k the dangling mass of r_k (it returns to the seed); stop after max_it
// iterations or when max_k sum_v |r_k' - r_k| < tol.  FP32 values, FP64
// residual and dangling sums.
//
// Layout: the reverse graph relabelled by in-degree (longest rows first,
// olv_rowtiles.cuh's plan), one 128-byte row of 32 floats per vertex for the
// values x and for the scaled contributions y = x / outdeg (ping-pong).
// Each iteration is one pull: a group of 8 lanes per row, each lane holding
// four vectors (a float4), walks the row's in-edges in order, gathers the
// 128-byte contribution row of every in-neighbour and adds it with
// compensated (two-sum) FP32 arithmetic, so the sums have a fixed order and
// about one rounding each.  Rows longer than kPprLong are summed in fixed
// kPprSeg-edge segments first and the segments folded in a fixed order, a
// warp per row.  The same pass writes x', y' and per-CTA FP64 partials of
// |x' - x| and of the new dangling mass; a one-CTA kernel folds the partials
// in a fixed order and decides convergence on the device, inside a CUDA graph.
//
// What bounds it is the latency of the chain row offsets -> indices -> 128-byte
// rows from L2 and HBM, so every group keeps eight gathers per lane in flight
// and loads the next indices, and the next row's offsets and first indices,
// before it waits for them.  Rows without in-edges (the last ones; about half
// of an RMAT graph) hold zeros that no iteration changes, except the seeds
// among them, which the folding kernel updates: the pass does not visit them.
// RMAT-21, 32 vectors, 20 iterations: 43.0 -> 11.8 ms (before: four gathers in
// flight, no index prefetch, 1024-edge segments folded one by one, scalar adds,
// every row visited); 0.59 ms an iteration, 7.0 TB/s of gathered rows, L2 at
// 35-39% and HBM at 15-28% of their peaks.
#include <algorithm>
#include <vector>

#include "olive_b200/olv_advance.cuh"
#include "olv_graphexec.cuh"
#include "olv_internal.cuh"
#include "olv_rowtiles.cuh"

namespace olv {

constexpr int kPprK = 32;                // vectors per row (K is padded to 32)
constexpr uint32_t kPprLong = 256;       // rows with more in-edges are segmented
constexpr uint32_t kPprSeg = 256;        // in-edges per segment (32 rounds of 8 gathers)
// 4 CTAs per SM at 64 registers (a few spills): 11.8 ms; 3 at 80: 12.3; 5: 14.4
constexpr int kPprMinBlocks = 4;
constexpr uint32_t kPprCTAs = 148 * kPprMinBlocks;   // fixed grid: fixed partial order

struct PprCtl {
    double res[kPprK];      // residual of the last completed iteration, per vector
    double dang[kPprK];     // dangling mass of the current iterate, per vector
    uint32_t seed[kPprK];   // seeds in the relabelled ids (0xffffffff: padding)
    double alpha;
    double tol;
    double max_res;
    float a_hi, a_lo;       // alpha as an unevaluated FP32 pair
    uint32_t iter;
    uint32_t max_it;
    uint32_t done;
};

// Compensated accumulation of a lane's four vectors (Knuth's two-sum), two per
// instruction: 14 instructions per in-edge and lane instead of 28 (the pass
// was issue bound: 0.7 warp instructions per cycle and scheduler).
struct Acc4 {
    ulonglong2 s, c;
    __device__ __forceinline__ void zero() {
        s = make_ulonglong2(0, 0);
        c = s;
    }
    __device__ __forceinline__ static void add1(unsigned long long &s, unsigned long long &c,
                                                unsigned long long x) {
        const unsigned long long t = add2(s, x);
        const unsigned long long bp = sub2(t, s);
        c = add2(c, add2(sub2(s, sub2(t, bp)), sub2(x, bp)));
        s = t;
    }
    __device__ __forceinline__ void add(ulonglong2 x) {
        add1(s.x, c.x, x.x);
        add1(s.y, c.y, x.y);
    }
    __device__ __forceinline__ void add_pair(ulonglong2 xs, ulonglong2 xc) {
        add(xs);
        c.x = add2(c.x, xc.x);
        c.y = add2(c.y, xc.y);
    }
    __device__ __forceinline__ float4 value() const {
        const unsigned long long a = add2(s.x, c.x), b = add2(s.y, c.y);
        return make_float4(__uint_as_float((uint32_t)a), __uint_as_float((uint32_t)(a >> 32)),
                           __uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32)));
    }
};

// The next 8 in-neighbour ids of a group's row, one per lane; past the end the
// row `none` of y, which holds zeros.
__device__ __forceinline__ uint32_t ppr_ids(const uint32_t *__restrict__ idx, uint32_t j,
                                            uint32_t e, uint32_t none) {
    return j < e ? __ldcs(&idx[j]) : none;
}

// Sum of y rows over in-edges [b, e) of the four rows of a warp, one row per
// 8-lane group: lane q of a group holds vectors 4q..4q+3; the group reads 8
// in-neighbour ids at a time (one per lane; u: the first ones) and broadcasts
// them.  The warp stays together for the longest of its rows (neighbours in
// the in-degree order are equally long); an in-edge that a row does not have
// adds the zero row, which changes neither part of the sum and needs no test.
__device__ __forceinline__ void ppr_row_sum(const uint32_t *__restrict__ idx,
                                            const ulonglong2 *__restrict__ y, uint32_t b,
                                            uint32_t e, uint32_t u, uint32_t none, uint32_t q,
                                            int gbase, Acc4 &acc) {
    constexpr unsigned kFull = 0xffffffffu;
    const uint32_t longest = __reduce_max_sync(kFull, e - b);
    for (uint32_t k = 0; k < longest; k += 8) {
        ulonglong2 v[8];
#pragma unroll
        for (int t = 0; t < 4; t++)
            v[t] = __ldg(&y[(size_t)__shfl_sync(kFull, u, gbase + t) * (kPprK / 4) + q]);
        const bool more = k + 4 < longest;   // the same in the whole warp
        if (more) {
#pragma unroll
            for (int t = 4; t < 8; t++)
                v[t] = __ldg(&y[(size_t)__shfl_sync(kFull, u, gbase + t) * (kPprK / 4) + q]);
        }
        u = ppr_ids(idx, b + k + 8 + q, e, none);   // the next round's ids, behind the gathers
#pragma unroll
        for (int t = 0; t < 4; t++) acc.add(v[t]);
        if (more) {
#pragma unroll
            for (int t = 4; t < 8; t++) acc.add(v[t]);
        }
    }
}

// Long rows: segment s of the list sums its in-edges into (sum, comp) rows.
__global__ void __launch_bounds__(kBlock, kPprMinBlocks)
k_ppr_segments(const uint32_t *__restrict__ idx, const uint2 *__restrict__ segs,
               uint32_t nsegs, uint32_t none, const PprCtl *ctl,
               const ulonglong2 *__restrict__ y0, const ulonglong2 *__restrict__ y1,
               ulonglong2 *__restrict__ seg_sum, ulonglong2 *__restrict__ seg_comp) {
    if (ctl->done) return;
    const ulonglong2 *y = (ctl->iter & 1) ? y1 : y0;
    const uint32_t lane = threadIdx.x & 31, g = lane >> 3, q = lane & 7;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t stride = ((gridDim.x * blockDim.x) >> 5) * 4;
    // this segment's range and first ids, the next one's range
    uint32_t s = warp * 4 + g;
    uint2 r = s < nsegs ? __ldg(&segs[s]) : make_uint2(0u, 0u);
    uint32_t u = ppr_ids(idx, r.x + q, r.y, none);
    uint2 rn = s + stride < nsegs ? __ldg(&segs[s + stride]) : make_uint2(0u, 0u);
    for (uint32_t s0 = warp * 4; s0 < nsegs; s0 += stride) {
        const uint32_t un = ppr_ids(idx, rn.x + q, rn.y, none);
        const uint32_t s2 = s + 2 * stride;
        const uint2 r2 = s2 < nsegs ? __ldg(&segs[s2]) : make_uint2(0u, 0u);
        Acc4 acc;
        acc.zero();
        ppr_row_sum(idx, y, r.x, r.y, u, none, q, (int)(8 * g), acc);
        if (s < nsegs) {
            seg_sum[(size_t)s * 8 + q] = acc.s;
            seg_comp[(size_t)s * 8 + q] = acc.c;
        }
        s += stride;
        r = rn;
        u = un;
        rn = r2;
    }
}

// What a lane needs to finish a row.  Seeds, their constant terms ((1-alpha) +
// alpha d_k) and the rarely touched dangling sums stay in shared memory (each
// lane adds to places of its own), which leaves the registers to the gathers
// of four CTAs per SM.
struct PprEndShared {
    uint32_t seed[kPprK];
    float term[kPprK];
    double dang[kBlock][4];
};

struct PprRowEnd {
    PprEndShared *sh;
    float a_hi, a_lo;
    double res[4];
    // Row r (sums sv, values before the iteration old, out-degree d): x' and y'
    __device__ __forceinline__ void finish(uint32_t r, uint32_t q, float4 sv, float4 old,
                                           uint32_t d, float4 *__restrict__ x,
                                           float4 *__restrict__ yout) {
        const uint4 sd = reinterpret_cast<const uint4 *>(sh->seed)[q];
        float4 base = make_float4(0, 0, 0, 0);
        if (sd.x == r || sd.y == r || sd.z == r || sd.w == r) {
            const float4 st = reinterpret_cast<const float4 *>(sh->term)[q];
            if (sd.x == r) base.x = st.x;
            if (sd.y == r) base.y = st.y;
            if (sd.z == r) base.z = st.z;
            if (sd.w == r) base.w = st.w;
        }
        float4 nv;
        nv.x = fmaf(a_hi, sv.x, fmaf(a_lo, sv.x, base.x));
        nv.y = fmaf(a_hi, sv.y, fmaf(a_lo, sv.y, base.y));
        nv.z = fmaf(a_hi, sv.z, fmaf(a_lo, sv.z, base.z));
        nv.w = fmaf(a_hi, sv.w, fmaf(a_lo, sv.w, base.w));
        res[0] += fabs((double)nv.x - (double)old.x);
        res[1] += fabs((double)nv.y - (double)old.y);
        res[2] += fabs((double)nv.z - (double)old.z);
        res[3] += fabs((double)nv.w - (double)old.w);
        __stcs(&x[(size_t)r * 8 + q], nv);
        if (d) {
            const float fd = (float)d;
            yout[(size_t)r * 8 + q] = make_float4(__fdiv_rn(nv.x, fd), __fdiv_rn(nv.y, fd),
                                                  __fdiv_rn(nv.z, fd), __fdiv_rn(nv.w, fd));
        } else {
            yout[(size_t)r * 8 + q] = make_float4(0, 0, 0, 0);
            double *dang = sh->dang[threadIdx.x];
            dang[0] += (double)nv.x;
            dang[1] += (double)nv.y;
            dang[2] += (double)nv.z;
            dang[3] += (double)nv.w;
        }
    }
};

// One pull over the rows with in-edges [0, n): folded segments for the first
// nlong, sums for the others; the update, the next contributions, and per-CTA
// FP64 partials of |x' - x| and the dangling mass.
__global__ void __launch_bounds__(kBlock, kPprMinBlocks)
k_ppr_rows(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ idx,
           const uint32_t *__restrict__ outdeg, uint32_t n, uint32_t none, uint32_t nlong,
           const uint32_t *__restrict__ seg_first, const ulonglong2 *__restrict__ seg_sum,
           const ulonglong2 *__restrict__ seg_comp, const PprCtl *ctl, float4 *__restrict__ x,
           float4 *__restrict__ y0, float4 *__restrict__ y1, double *__restrict__ partials) {
    __shared__ double s_part[kBlock / 32][2 * kPprK];
    if (ctl->done) return;
    constexpr unsigned kFull = 0xffffffffu;
    const bool odd = ctl->iter & 1;
    const ulonglong2 *yin = reinterpret_cast<const ulonglong2 *>(odd ? y1 : y0);
    float4 *yout = odd ? y0 : y1;
    const uint32_t lane = threadIdx.x & 31, g = lane >> 3, q = lane & 7;
    const uint32_t wl = threadIdx.x >> 5;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    __shared__ __align__(16) PprEndShared sh;
    PprRowEnd end;
    end.sh = &sh;
    end.a_hi = ctl->a_hi;
    end.a_lo = ctl->a_lo;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        end.res[t] = 0;
        sh.dang[threadIdx.x][t] = 0;
    }
    if (threadIdx.x < kPprK) {
        const uint32_t k = threadIdx.x;
        sh.seed[k] = ctl->seed[k];
        sh.term[k] = (float)((1.0 - ctl->alpha) + ctl->alpha * ctl->dang[k]);
    }
    __syncthreads();
    // long rows: a warp each, group g folds segments g, g + 4, ... in order,
    // then the four groups' sums by a fixed tree
    for (uint32_t r = warp; r < nlong; r += nwarps) {
        const uint32_t s1 = __ldg(&seg_first[r + 1]);
        Acc4 acc;
        acc.zero();
        for (uint32_t s = __ldg(&seg_first[r]) + g; s < s1; s += 16) {
            ulonglong2 a[4], c[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t k = s + 4 * t;
                a[t] = k < s1 ? seg_sum[(size_t)k * 8 + q] : make_ulonglong2(0, 0);
                c[t] = k < s1 ? seg_comp[(size_t)k * 8 + q] : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int t = 0; t < 4; t++) acc.add_pair(a[t], c[t]);
        }
        __syncwarp();
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
            ulonglong2 s2, c2;
            s2.x = __shfl_down_sync(kFull, acc.s.x, o);
            s2.y = __shfl_down_sync(kFull, acc.s.y, o);
            c2.x = __shfl_down_sync(kFull, acc.c.x, o);
            c2.y = __shfl_down_sync(kFull, acc.c.y, o);
            acc.add_pair(s2, c2);
        }
        if (g == 0)
            end.finish(r, q, acc.value(), __ldcs(&x[(size_t)r * 8 + q]), __ldg(&outdeg[r]), x, yout);
        __syncwarp();
    }
    // the others: four per warp; this row's range and first ids, the next
    // row's range
    const uint32_t stride = nwarps * 4;
    uint32_t r = nlong + warp * 4 + g;
    uint32_t b = 0, e = 0, bn = 0, en = 0;
    if (r < n) {
        b = __ldg(&ptr[r]);
        e = __ldg(&ptr[r + 1]);
    }
    uint32_t u = ppr_ids(idx, b + q, e, none);
    if (r + stride < n) {
        bn = __ldg(&ptr[r + stride]);
        en = __ldg(&ptr[r + stride + 1]);
    }
    for (uint32_t r0 = nlong + warp * 4; r0 < n; r0 += stride) {
        const uint32_t un = ppr_ids(idx, bn + q, en, none);
        uint32_t b2 = 0, e2 = 0, d = 0;
        if (r + 2 * stride < n) {
            b2 = __ldg(&ptr[r + 2 * stride]);
            e2 = __ldg(&ptr[r + 2 * stride + 1]);
        }
        float4 old = make_float4(0, 0, 0, 0);
        if (r < n) {
            old = __ldcs(&x[(size_t)r * 8 + q]);
            d = __ldg(&outdeg[r]);
        }
        Acc4 acc;
        acc.zero();
        ppr_row_sum(idx, yin, b, e, u, none, q, (int)(8 * g), acc);
        if (r < n) end.finish(r, q, acc.value(), old, d, x, yout);
        r += stride;
        b = bn;
        e = en;
        u = un;
        bn = b2;
        en = e2;
    }
    // fixed-order reduction: the warp's four groups, then the CTA's warps
    double dang[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        dang[t] = sh.dang[threadIdx.x][t];
        end.res[t] += __shfl_xor_sync(kFull, end.res[t], 8);
        end.res[t] += __shfl_xor_sync(kFull, end.res[t], 16);
        dang[t] += __shfl_xor_sync(kFull, dang[t], 8);
        dang[t] += __shfl_xor_sync(kFull, dang[t], 16);
    }
    if (g == 0) {
#pragma unroll
        for (int t = 0; t < 4; t++) {
            s_part[wl][4 * q + t] = end.res[t];
            s_part[wl][kPprK + 4 * q + t] = dang[t];
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * kPprK) {
        double a = 0;
        for (int w = 0; w < kBlock / 32; w++) a += s_part[w][threadIdx.x];
        partials[(size_t)blockIdx.x * 2 * kPprK + threadIdx.x] = a;
    }
}

// Fold the per-CTA partials in a fixed order (16 threads per vector and sum,
// then those in order: 45 -> 5 us against one thread each), update the seeds
// whose rows have no in-edges (rows from n on; their sum is zero), publish
// residuals and dangling masses, decide convergence.
constexpr int kPprFold = 16;

__global__ void __launch_bounds__(2 * kPprK * kPprFold)
k_ppr_reduce(PprCtl *ctl, const double *__restrict__ partials, uint32_t nparts, uint32_t n,
             const uint32_t *__restrict__ outdeg, float *__restrict__ x, float *__restrict__ y0,
             float *__restrict__ y1, cudaGraphConditionalHandle h, int use_cond) {
    if (ctl->done) {
        if (use_cond && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    __shared__ double s_sum[kPprFold][2 * kPprK];
    const uint32_t k = threadIdx.x % (2 * kPprK), f = threadIdx.x / (2 * kPprK);
    double a = 0;
    for (uint32_t i = f; i < nparts; i += kPprFold) a += partials[(size_t)i * 2 * kPprK + k];
    s_sum[f][k] = a;
    __syncthreads();
    if (threadIdx.x >= kPprK) return;
    double res = 0, dang = 0;
    for (int i = 0; i < kPprFold; i++) {
        res += s_sum[i][k];
        dang += s_sum[i][kPprK + k];
    }
    const uint32_t s = ctl->seed[k];
    if (s != 0xffffffffu && s >= n) {
        const float nv = (float)((1.0 - ctl->alpha) + ctl->alpha * ctl->dang[k]);
        float *yout = (ctl->iter & 1) ? y0 : y1;
        const size_t at = (size_t)s * kPprK + k;
        const uint32_t d = outdeg[s];
        res += fabs((double)nv - (double)x[at]);
        x[at] = nv;
        yout[at] = d ? __fdiv_rn(nv, (float)d) : 0.0f;
        if (!d) dang += (double)nv;
    }
    ctl->res[k] = res;
    ctl->dang[k] = dang;
    double m = res;
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (k == 0) {
        ctl->max_res = m;
        ctl->iter++;
        if (m < ctl->tol || ctl->iter >= ctl->max_it) ctl->done = 1;
        if (use_cond) cudaGraphSetConditional(h, ctl->done ? 0u : 1u);
    }
}

// Start state: x = e_{s_k}, y = x / outdeg, d_k = [outdeg(s_k) == 0].
__global__ void k_ppr_init_seeds(PprCtl *ctl, const uint32_t *__restrict__ outdeg, float *x,
                                 float *y0, double alpha, double tol, uint32_t max_it) {
    const int k = threadIdx.x;   // kPprK threads
    const uint32_t s = ctl->seed[k];
    if (s != 0xffffffffu) {
        const uint32_t d = outdeg[s];
        x[(size_t)s * kPprK + k] = 1.0f;
        y0[(size_t)s * kPprK + k] = d ? __fdiv_rn(1.0f, (float)d) : 0.0f;
        ctl->dang[k] = d ? 0.0 : 1.0;
    } else {
        ctl->dang[k] = 0.0;
    }
    ctl->res[k] = 0.0;
    if (k == 0) {
        ctl->alpha = alpha;
        ctl->a_hi = (float)alpha;
        ctl->a_lo = (float)(alpha - (double)ctl->a_hi);
        ctl->tol = tol;
        ctl->max_it = max_it;
        ctl->iter = 0;
        ctl->max_res = 0;
        ctl->done = max_it == 0;
    }
}

__global__ void k_ppr_set_seeds(PprCtl *ctl, const uint32_t *__restrict__ seeds, int K,
                                const uint32_t *__restrict__ newid) {
    const int k = threadIdx.x;
    ctl->seed[k] = k < K ? newid[seeds[k]] : 0xffffffffu;
}

// out[v][k] = x[newid[v]][k] for k < K (the caller's ids and width).
__global__ void k_ppr_unpermute(const float *__restrict__ x, const uint32_t *__restrict__ newid,
                                uint32_t V, int K, float *__restrict__ out) {
    const uint64_t total = (uint64_t)V * K;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = i / K, k = i - v * K;
        out[i] = x[(size_t)newid[v] * kPprK + k];
    }
}

// The same for K = 32 and a 16-byte aligned output: whole 128-byte rows, eight
// lanes each, four rows in flight (RMAT-21: 220 -> 108 us).
__global__ void __launch_bounds__(kBlock)
k_ppr_unpermute32(const float4 *__restrict__ x, const uint32_t *__restrict__ newid, uint32_t V,
                  float4 *__restrict__ out) {
    const uint64_t total = (uint64_t)V * 8, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (uint64_t i = tid; i < total; i += 4 * stride) {
        float4 t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint64_t k = i + j * stride;
            if (k < total) t[j] = __ldcs(&x[(size_t)__ldg(&newid[k >> 3]) * 8 + (k & 7)]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (i + j * stride < total) __stcs(&out[i + j * stride], t[j]);
    }
}

__global__ void k_outdeg_in_order(const uint32_t *__restrict__ rowptr,
                                  const uint32_t *__restrict__ perm, uint32_t V, uint32_t *d) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = perm[i];
        d[i] = rowptr[v + 1] - rowptr[v];
    }
}

// ------------------------------------------------------------------ host --
struct PprState {
    TilePlan tp;                       // relabelled reverse graph (rows by in-degree)
    DevBuf outdeg, x, y, ctl, partials, segs, seg_first, seg_sum, seg_comp, seeds, out;
    uint32_t nlong = 0, nsegs = 0;
    uint32_t nrows = 0;                // rows with in-edges (a prefix)
    WhileGraph graph;
    ~PprState() {
        graph.destroy();
        tp.release(); outdeg.release(); x.release(); y.release(); ctl.release();
        partials.release(); segs.release(); seg_first.release(); seg_sum.release();
        seg_comp.release(); seeds.release(); out.release();
    }
};

static int build_ppr_state(olv_graph *g, PprState &p) {
    const uint32_t V = g->V;
    cudaStream_t s = g->stream;
    OLV_TRY(build_tile_plan(g->colptr.as<uint32_t>(), g->rowidx.as<uint32_t>(), V, s, p.tp));
    OLV_TRY(p.outdeg.ensure((size_t)V * 4 + 16));
    k_outdeg_in_order<<<g->num_sms * 8, kBlock, 0, s>>>(
        g->rowptr.as<uint32_t>(), p.tp.perm.as<uint32_t>(), V, p.outdeg.as<uint32_t>());
    // long rows are a prefix of the in-degree order: their segments
    std::vector<uint32_t> ptr((size_t)V + 1);
    OLV_CUDA(cudaMemcpyAsync(ptr.data(), p.tp.ptr.p, ((size_t)V + 1) * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    uint32_t nlong = 0;
    while (nlong < V && ptr[nlong + 1] - ptr[nlong] > kPprLong) nlong++;
    uint32_t nrows = nlong;
    while (nrows < V && ptr[nrows + 1] > ptr[nrows]) nrows++;
    p.nrows = nrows;
    std::vector<uint2> segs;
    std::vector<uint32_t> first((size_t)nlong + 1, 0);
    for (uint32_t r = 0; r < nlong; r++) {
        first[r] = (uint32_t)segs.size();
        for (uint32_t b = ptr[r]; b < ptr[r + 1]; b += kPprSeg)
            segs.push_back(make_uint2(b, std::min(ptr[r + 1], b + kPprSeg)));
    }
    first[nlong] = (uint32_t)segs.size();
    p.nlong = nlong;
    p.nsegs = (uint32_t)segs.size();
    const size_t rows = (size_t)V * kPprK * 4;
    OLV_TRY(p.x.ensure(rows + 64));
    OLV_TRY(p.y.ensure(2 * (rows + kPprK * 4) + 64));   // each with a last row of zeros
    OLV_TRY(p.ctl.ensure(sizeof(PprCtl)));
    OLV_TRY(p.partials.ensure((size_t)kPprCTAs * 2 * kPprK * 8));
    OLV_TRY(p.segs.ensure(segs.size() * 8 + 16));
    OLV_TRY(p.seg_first.ensure(first.size() * 4 + 16));
    OLV_TRY(p.seg_sum.ensure(segs.size() * kPprK * 4 + 16));
    OLV_TRY(p.seg_comp.ensure(segs.size() * kPprK * 4 + 16));
    OLV_TRY(p.seeds.ensure(kPprK * 4));
    if (!segs.empty())
        OLV_CUDA(cudaMemcpyAsync(p.segs.p, segs.data(), segs.size() * 8, cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaMemcpyAsync(p.seg_first.p, first.data(), first.size() * 4, cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaStreamSynchronize(s));   // the host vectors die here
    return OLV_OK;
}

template <class Sink>
static int ppr_iteration(olv_graph *g, PprState &p, Sink &&sink, cudaGraphConditionalHandle h,
                         int use_cond) {
    PprCtl *ctl = p.ctl.as<PprCtl>();
    const uint32_t *idx = p.tp.idx.as<uint32_t>(), *ptr = p.tp.ptr.as<uint32_t>();
    const uint32_t *outdeg = p.outdeg.as<uint32_t>();
    const uint32_t *seg_first = p.seg_first.as<uint32_t>();
    const uint2 *segs = p.segs.as<uint2>();
    float4 *x = p.x.as<float4>();
    float4 *y0 = p.y.as<float4>();
    float4 *y1 = y0 + ((size_t)g->V + 1) * (kPprK / 4);
    float4 *seg_sum = p.seg_sum.as<float4>(), *seg_comp = p.seg_comp.as<float4>();
    double *partials = p.partials.as<double>();
    uint32_t n = p.nrows, none = g->V, nlong = p.nlong, nsegs = p.nsegs, nparts = kPprCTAs;
    float *xf = p.x.as<float>(), *y0f = p.y.as<float>(), *y1f = y0f + ((size_t)g->V + 1) * kPprK;
    if (nsegs) {
        void *a_seg[] = {&idx, &segs, &nsegs, &none, &ctl, &y0, &y1, &seg_sum, &seg_comp};
        OLV_TRY(sink((const void *)k_ppr_segments, dim3(kPprCTAs), dim3(kBlock), a_seg));
    }
    void *a_rows[] = {&ptr, &idx, &outdeg, &n, &none, &nlong, &seg_first, &seg_sum, &seg_comp,
                      &ctl, &x, &y0, &y1, &partials};
    OLV_TRY(sink((const void *)k_ppr_rows, dim3(kPprCTAs), dim3(kBlock), a_rows));
    void *a_red[] = {&ctl, &partials, &nparts, &n, &outdeg, &xf, &y0f, &y1f, &h, &use_cond};
    OLV_TRY(sink((const void *)k_ppr_reduce, dim3(1), dim3(2 * kPprK * kPprFold), a_red));
    return OLV_OK;
}

}  // namespace olv

using namespace olv;

static PprState *ppr_state(olv_graph *g) { return static_cast<PprState *>(g->ppr_state); }

void olv::release_ppr_state(olv_graph *g) {
    delete ppr_state(g);
    g->ppr_state = nullptr;
}

extern "C" int olv_ppr_batch(olv_graph *g, const uint32_t *seeds, int K, double alpha,
                             int max_it, double tol, float *out, olv_stats *st) {
    OLV_CHECK_ARG(g && seeds && out, "olv_ppr_batch: null pointer");
    BufferScope scope(g->stream);
    OLV_CHECK_ARG(K >= 1 && K <= kPprK, "olv_ppr_batch: K must be in [1, %d]", kPprK);
    OLV_CHECK_ARG(alpha >= 0.0 && alpha < 1.0, "olv_ppr_batch: alpha must be in [0,1)");
    OLV_CHECK_ARG(max_it >= 0, "olv_ppr_batch: max_it must be >= 0");
    OLV_CHECK_ARG(g->V > 0, "olv_ppr_batch: empty graph");
    cudaStream_t s = g->stream;
    const bool dev_seeds = is_device_ptr(seeds);
    std::vector<uint32_t> hs(K);
    if (dev_seeds) {
        OLV_CUDA(cudaMemcpyAsync(hs.data(), seeds, (size_t)K * 4, cudaMemcpyDeviceToHost, s));
        OLV_CUDA(cudaStreamSynchronize(s));
    } else {
        std::copy(seeds, seeds + K, hs.begin());
    }
    for (int k = 0; k < K; k++)
        OLV_CHECK_ARG(hs[k] < g->V, "olv_ppr_batch: seed %u out of range (V=%u)", hs[k], g->V);
    PprState *ps = ppr_state(g);
    if (!ps) {
        ps = new PprState();
        g->ppr_state = ps;
        int r = build_ppr_state(g, *ps);
        if (r != OLV_OK) {
            release_ppr_state(g);
            return r;
        }
    }
    PprState &p = *ps;
    const size_t rows = (size_t)g->V * kPprK * 4;
    const bool dev_out = is_device_ptr(out);
    if (!dev_out) OLV_TRY(p.out.ensure((size_t)g->V * K * 4 + 16));
    float *dst = dev_out ? out : p.out.as<float>();
    OLV_CUDA(cudaEventRecord(g->ev0, s));
    OLV_CUDA(cudaMemcpyAsync(p.seeds.p, hs.data(), (size_t)K * 4, cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaMemsetAsync(p.x.p, 0, rows, s));
    // y0, and the rows of y1 that no iteration writes (the others are written
    // before they are read)
    const size_t ybytes = rows + kPprK * 4, skip = (size_t)p.nrows * kPprK * 4;
    OLV_CUDA(cudaMemsetAsync(p.y.p, 0, ybytes, s));
    OLV_CUDA(cudaMemsetAsync(p.y.as<char>() + ybytes + skip, 0, ybytes - skip, s));
    k_ppr_set_seeds<<<1, kPprK, 0, s>>>(p.ctl.as<PprCtl>(), p.seeds.as<uint32_t>(), K,
                                        p.tp.newid.as<uint32_t>());
    k_ppr_init_seeds<<<1, kPprK, 0, s>>>(p.ctl.as<PprCtl>(), p.outdeg.as<uint32_t>(),
                                         p.x.as<float>(), p.y.as<float>(), alpha, tol,
                                         (uint32_t)max_it);
    OLV_CUDA(cudaGetLastError());
    bool launched = false;
    if (g->tune.use_graphs && max_it > 0) {
        if (!p.graph.ready) {
            int r = p.graph.begin();
            auto sink = [&](const void *f, dim3 gr, dim3 bl, void **args) {
                return p.graph.add(f, gr, bl, args);
            };
            if (r == OLV_OK) r = ppr_iteration(g, p, sink, p.graph.handle, 1);
            if (r == OLV_OK) r = p.graph.finish();
            if (r != OLV_OK) p.graph.destroy();
        }
        if (p.graph.ready) {
            OLV_TRY(p.graph.launch(s));
            launched = true;
        }
    }
    if (!launched) {
        auto launch = [&](const void *f, dim3 gr, dim3 bl, void **args) {
            OLV_CUDA(cudaLaunchKernel(f, gr, bl, args, 0, s));
            return OLV_OK;
        };
        for (int it = 0; it < max_it; it++) OLV_TRY(ppr_iteration(g, p, launch, 0, 0));
    }
    if (K == kPprK && ((uintptr_t)dst & 15) == 0)
        k_ppr_unpermute32<<<g->num_sms * 8, kBlock, 0, s>>>(
            p.x.as<float4>(), p.tp.newid.as<uint32_t>(), g->V, reinterpret_cast<float4 *>(dst));
    else
        k_ppr_unpermute<<<g->num_sms * 8, kBlock, 0, s>>>(
            p.x.as<float>(), p.tp.newid.as<uint32_t>(), g->V, K, dst);
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaEventRecord(g->ev1, s));
    PprCtl hc;
    OLV_CUDA(cudaMemcpyAsync(&hc, p.ctl.p, sizeof hc, cudaMemcpyDeviceToHost, s));
    if (!dev_out)
        OLV_CUDA(cudaMemcpyAsync(out, dst, (size_t)g->V * K * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    // seeds, start, the iterations, map back
    g->launches = 3 + (p.nsegs ? 3ull : 2ull) * (launched ? hc.iter : (uint32_t)max_it);
    if (st) {
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        st->iterations = hc.iter;
        st->pull_steps = 0;
        st->vertices_reached = g->V;
        st->edges_traversed = g->E * (uint64_t)hc.iter;
        st->edges_relaxed = g->E * (uint64_t)hc.iter * (uint64_t)K;
        st->residual = hc.max_res;
        st->device_ms = ms;
    }
    return OLV_OK;
}
