// Batched traversal of many small graphs packed block-diagonally in one CSR,
// run by ONE persistent kernel with a device-side work queue (no reference
// counterpart; each instance's result equals its solo run, bit for bit).
//
// Work items are (instance, task) pairs handed out by atomic counters,
// largest instances first; the CTA or cluster that takes one runs it to completion:
//   BFS from the instance's local vertex 0 (testBFS.cu semantics, levels
//     relative to the instance, 0x7fffffff unreached).  The visited, current
//     and next frontier bitmaps of the instance live in shared memory
//     (3 x 8 KB for up to 65,536 vertices); a thread per vertex expands the
//     frontier with shared-memory atomicOr claims.
//   PPR: K <= 32 personalised PageRank vectors with one-hot seeds (the
//     oracle's orc_ppr definition: dangling mass returns to the seed), pulled
//     over the in-edges, summed in CSC order per vertex and vector.  K = 4, 8,
//     16 or 32: a lane owns four vectors, so one warp gathers for 32 / (K / 4)
//     vertices at a time; any other K: one warp per vertex, lane k = vector k.
//     The dangling mass is summed while the new vectors are written, in an
//     order-free or a fixed way, so results do not depend on which CTA runs
//     the item or when.  Stops after max_it iterations or when every vector's
//     L1 change (FP64) is below tol.
#include <algorithm>
#include <numeric>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "olive_b200/olv_advance.cuh"
#include "olv_internal.cuh"

namespace cg = cooperative_groups;

namespace olv {

constexpr int kBatchThreads = 512;
constexpr uint32_t kBatchMaxV = 65536;
constexpr int kBatchWarps = kBatchThreads / 32;
constexpr int kBatchMaxWarps = 32;
// PPR items of at most this many vertices can take one CTA, larger ones take a
// cluster (choose_large() below): a sweep of a small instance on 16 CTAs is mostly its
// barrier, while a larger one on a CTA is left running alone at the end.
constexpr uint32_t kCtaItem = 2048;

struct BatchArgs {
    const uint32_t *rowptr, *col, *colptr, *rowidx;
    const uint32_t *inst_off;
    const uint32_t *order;       // instances, largest first
    const uint32_t *seeds;       // [count][K] local ids
    int count, K, max_it, tasks; // tasks: 1 = BFS only / PPR only, 2 = both
    int do_bfs, do_ppr;
    float alpha;
    double tol;
    int32_t *levels;             // [V]
    float *ppr, *ppr_tmp;        // [V][K]
    float *inv_deg;              // [V] 1 / out-degree (0: dangling), written per PPR item
    uint2 *ew;                   // rows of four vectors: [E] in-edges as (local source, its inverse degree)
    uint32_t n_large;            // items order[0 .. n_large) are a cluster's, the rest a CTA's
    uint32_t *counter;           // work queue head
    uint32_t *ppr_iters;         // [count]
    unsigned long long *stats;   // [0] BFS edges traversed, [1] PPR edge visits, [2] error bits
};

__device__ void cta_bfs(const BatchArgs &a, uint32_t inst, uint32_t *bm) {
    const uint32_t base = a.inst_off[inst], n = a.inst_off[inst + 1] - base;
    const uint32_t words = (n + 31) / 32;
    uint32_t *vis = bm, *cur = bm + kBatchMaxV / 32, *nxt = bm + 2 * (kBatchMaxV / 32);
    __shared__ int s_any;
    __shared__ unsigned long long s_edges;
    for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) {
        vis[w] = 0;
        cur[w] = 0;
    }
    for (uint32_t v = threadIdx.x; v < n; v += blockDim.x) a.levels[base + v] = kInf;
    __syncthreads();
    if (threadIdx.x == 0) {
        vis[0] = 1u;
        cur[0] = 1u;
        a.levels[base] = 0;
        s_edges = 0;
    }
    unsigned long long edges = 0;
    for (int L = 0;; L++) {
        for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) nxt[w] = 0;
        if (threadIdx.x == 0) s_any = 0;
        __syncthreads();
        int any = 0;
        for (uint32_t u = threadIdx.x; u < n; u += blockDim.x) {
            if (!((cur[u >> 5] >> (u & 31)) & 1u)) continue;
            const uint32_t b = a.rowptr[base + u], e = a.rowptr[base + u + 1];
            edges += e - b;
            for (uint32_t i = b; i < e; i++) {
                const uint32_t v = a.col[i] - base;
                if (v >= n) {   // edge leaves the instance: not block-diagonal
                    atomicOr((unsigned int *)&a.stats[2], 1u);
                    continue;
                }
                const uint32_t bit = 1u << (v & 31);
                if (vis[v >> 5] & bit) continue;
                if (!(atomicOr(&vis[v >> 5], bit) & bit)) {
                    atomicOr(&nxt[v >> 5], bit);
                    a.levels[base + v] = L + 1;
                    any = 1;
                }
            }
        }
        if (any) s_any = 1;
        __syncthreads();
        uint32_t *t = cur;
        cur = nxt;
        nxt = t;
        const int go = s_any;
        __syncthreads();
        if (!go) break;
    }
    atomicAdd(&s_edges, edges);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&a.stats[0], s_edges);
    __syncthreads();
}

// Rows gathered per round of one warp's in-edge walk: the loads of a round
// are issued together, then folded in CSC order.
constexpr int kPprRound = 8;

// What one warp sees of a PPR item.
struct PprView {
    uint32_t base, n, seed;
    int K;
    bool lk;          // lane < K: the lane carries vector `lane`
    float alpha;
    float *r0, *r1;   // the item's vectors, ping-pong
    float *inv;       // 1 / out-degree, 0 for a dangling vertex
};

__device__ __forceinline__ PprView ppr_view(const BatchArgs &a, uint32_t inst, uint32_t lane) {
    PprView p;
    p.base = a.inst_off[inst];
    p.n = a.inst_off[inst + 1] - p.base;
    p.K = a.K;
    p.lk = (int)lane < p.K;
    p.seed = p.lk ? a.seeds[(size_t)inst * p.K + lane] : 0xffffffffu;
    p.alpha = a.alpha;
    p.r0 = a.ppr + (size_t)p.base * p.K;
    p.r1 = a.ppr_tmp + (size_t)p.base * p.K;
    p.inv = a.inv_deg + p.base;
    return p;
}

// Start vectors and inverse out-degrees of the vertices v = w0, w0 + nw, ...;
// returns this warp's dangling mass of the start vectors (per lane), summed
// in vertex order.
__device__ __forceinline__ float ppr_init_warp(const BatchArgs &a, const PprView &p, uint32_t lane,
                                               uint32_t w0, uint32_t nw) {
    float dpart = 0.0f;
    for (uint32_t v = w0; v < p.n; v += nw) {
        const uint32_t deg = a.rowptr[p.base + v + 1] - a.rowptr[p.base + v];
        if (lane == 0) p.inv[v] = deg ? __fdiv_rn(1.0f, (float)deg) : 0.0f;
        const float x = (v == p.seed) ? 1.0f : 0.0f;
        if (p.lk) p.r0[(size_t)v * p.K + lane] = x;
        if (!deg) dpart += x;
    }
    return dpart;
}

// One sweep over the vertices v = w0, w0 + nw, ... (one warp each): pull
// src over the in-edges, write dst; accumulates the warp's dangling mass of
// the new vectors, its FP64 L1 change and its in-edge visits.
__device__ __forceinline__ void ppr_sweep_warp(const BatchArgs &a, const PprView &p, uint32_t lane,
                                               uint32_t w0, uint32_t nw, const float *src,
                                               float *dst, float dk, float &dpart, double &res,
                                               unsigned long long &visits) {
    const uint32_t base = p.base, n = p.n;
    const int K = p.K;
    for (uint32_t v = w0; v < n; v += nw) {
        const uint32_t b = a.colptr[base + v], e = a.colptr[base + v + 1];
        float acc = 0.0f;
        // 32 in-edges at a time: lane j fetches source j and its inverse
        // degree, then the warp gathers the sources' rows kPprRound at a
        // time (lane k = vector k) and folds them in CSC order.  Padding
        // slots carry weight 0 and add exactly 0.
        for (uint32_t c0 = b; c0 < e; c0 += 32) {
            const uint32_t cnt = min(32u, e - c0);
            uint32_t u = 0;
            float w = 0.0f;
            if (lane < cnt) {
                u = a.rowidx[c0 + lane] - base;
                if (u >= n) {   // edge enters from outside the instance
                    atomicOr((unsigned int *)&a.stats[2], 2u);
                    u = 0;
                } else {
                    w = p.inv[u];
                }
            }
            for (uint32_t t = 0; t < cnt; t += kPprRound) {
                float x[kPprRound], ww[kPprRound];
#pragma unroll
                for (int j = 0; j < kPprRound; j++) {
                    const uint32_t uj = __shfl_sync(0xffffffffu, u, (t + j) & 31);
                    ww[j] = __shfl_sync(0xffffffffu, w, (t + j) & 31);
                    x[j] = (p.lk && t + j < cnt) ? src[(size_t)uj * K + lane] : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < kPprRound; j++)
                    if (t + j < cnt) acc = fmaf(x[j], ww[j], acc);
            }
        }
        visits += e - b;
        if (p.lk) {
            const float tele = (v == p.seed) ? fmaf(p.alpha, dk, 1.0f - p.alpha) : 0.0f;
            const float nv = fmaf(p.alpha, acc, tele);
            res += fabs((double)nv - (double)src[(size_t)v * K + lane]);
            dst[(size_t)v * K + lane] = nv;
            if (p.inv[v] == 0.0f) dpart += nv;
        }
    }
}

// ---- rows of four vectors per lane (K = 4, 8, 16 or 32) --------------------
// L = K / 4 lanes per vertex, a float4 of vectors per lane, so a warp sweeps
// 32 / L vertices at once.  In-edges are read as (source, inverse degree) pairs
// laid out once per item: every lane of a vertex loads the pair itself (one
// broadcast load, no index arithmetic or shuffles), four pairs ahead of the four
// rows being gathered.  A place past a vertex's in-edges
// weighs zero.  Every vertex's in-edges are folded in CSC order.  The dangling
// mass is summed in 64-bit fixed point (units of 2^-62; the masses of a vector
// sum to at most one), so it does not depend on which warp adds what when; the
// L1 change (FP64, only with a tolerance to compare it with) is combined in a
// fixed order.
// The sweep this replaces (one chunk of indices per vertex, sources and weights
// by shuffles, K = 32 only) took 690 warp instructions per four vertices of eight
// in-edges and was bound by them: 96 uniform digraphs of 1024..65536 vertices,
// K = 32, 20 sweeps 18.0 -> 11.6 ms; K = 8 (a lane per vector before) 30.4 -> 5.8 ms.
constexpr double kDangOne = 4611686018427387904.0;   // 2^62

struct alignas(16) RowsShared {
    unsigned long long dang[3][32];       // this CTA's dangling mass, by sweep modulo 3
    double warp_res[2][kBatchMaxWarps][32];   // per warp and vector, by sweep parity
    double res[2][32];                    // this CTA's L1 change, by sweep parity
    alignas(16) uint32_t seed[32];
    alignas(16) float tele[32];           // what a seed gets in this sweep
    int stop;
};

// One sweep of one warp over the vertex groups g = w0, w0 + nw, ...; adds the new
// dangling mass to dang (shared) and, kRes, the L1 change to res: a group's by a fixed
// tree over its vertices, then the groups in order.
template <int L, bool kRes>
__device__ __forceinline__ void ppr_sweep_rows(const BatchArgs &a, const PprView &p,
                                               const RowsShared &sh, uint32_t lane, uint32_t w0,
                                               uint32_t nw, const float *src, float *dst,
                                               unsigned long long *dang, double (&res)[4]) {
    constexpr uint32_t kVerts = 32 / L;
    const uint32_t slot = lane / L, q = lane % L, n = p.n;
    const float4 *src4 = reinterpret_cast<const float4 *>(src) + q;
    float4 *dst4 = reinterpret_cast<float4 *>(dst) + q;
    for (uint32_t g = w0; g * kVerts < n; g += nw) {
        const uint32_t v = g * kVerts + slot;
        const bool valid = v < n;
        uint32_t b = 0, deg = 0;
        float inv = 1.0f;
        float4 old;
        if (valid) {
            b = a.colptr[p.base + v];
            deg = a.colptr[p.base + v + 1] - b;
            inv = p.inv[v];
            if (kRes) old = src4[(size_t)v * L];
        }
        const uint32_t longest = __reduce_max_sync(0xffffffffu, deg);
        const uint2 *ew = a.ew + b;
        uint2 e[4];
#pragma unroll
        for (uint32_t r = 0; r < 4; r++) e[r] = r < deg ? ew[r] : make_uint2(0u, 0u);
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t c = 0; c < longest; c += 4) {
            float4 x[4];
            float w[4];
#pragma unroll
            for (uint32_t r = 0; r < 4; r++) {
                x[r] = src4[(size_t)e[r].x * L];
                w[r] = __uint_as_float(e[r].y);
            }
#pragma unroll
            for (uint32_t r = 0; r < 4; r++)
                e[r] = c + 4 + r < deg ? ew[c + 4 + r] : make_uint2(0u, 0u);
#pragma unroll
            for (uint32_t r = 0; r < 4; r++) {
                acc.x = fmaf(x[r].x, w[r], acc.x);
                acc.y = fmaf(x[r].y, w[r], acc.y);
                acc.z = fmaf(x[r].z, w[r], acc.z);
                acc.w = fmaf(x[r].w, w[r], acc.w);
            }
        }
        double change[4] = {0.0, 0.0, 0.0, 0.0};
        if (valid) {
            const uint4 sd = reinterpret_cast<const uint4 *>(sh.seed)[q];
            float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (sd.x == v || sd.y == v || sd.z == v || sd.w == v) {
                const float4 s = reinterpret_cast<const float4 *>(sh.tele)[q];
                t = make_float4(sd.x == v ? s.x : 0.0f, sd.y == v ? s.y : 0.0f,
                                sd.z == v ? s.z : 0.0f, sd.w == v ? s.w : 0.0f);
            }
            const float4 nv = make_float4(fmaf(p.alpha, acc.x, t.x), fmaf(p.alpha, acc.y, t.y),
                                          fmaf(p.alpha, acc.z, t.z), fmaf(p.alpha, acc.w, t.w));
            if (kRes) {
                change[0] = fabs((double)nv.x - (double)old.x);
                change[1] = fabs((double)nv.y - (double)old.y);
                change[2] = fabs((double)nv.z - (double)old.z);
                change[3] = fabs((double)nv.w - (double)old.w);
            }
            dst4[(size_t)v * L] = nv;
            if (inv == 0.0f) {   // a dangling vertex: rare enough for shared atomics
                atomicAdd(&dang[4 * q], __double2ull_rn((double)nv.x * kDangOne));
                atomicAdd(&dang[4 * q + 1], __double2ull_rn((double)nv.y * kDangOne));
                atomicAdd(&dang[4 * q + 2], __double2ull_rn((double)nv.z * kDangOne));
                atomicAdd(&dang[4 * q + 3], __double2ull_rn((double)nv.w * kDangOne));
            }
        }
        if (kRes) {
#pragma unroll
            for (int o = L; o < 32; o <<= 1)
#pragma unroll
                for (int c = 0; c < 4; c++)
                    change[c] += __shfl_xor_sync(0xffffffffu, change[c], o);
#pragma unroll
            for (int c = 0; c < 4; c++) res[c] += change[c];
        }
    }
}

// A PPR item by a team of C CTAs (this is CTA `rank`); sync(): the team's barrier,
// at(p, r): CTA r's copy of a shared variable.
template <int L, class Sync, class At>
__device__ void team_ppr(const BatchArgs &a, uint32_t inst, uint32_t C, uint32_t rank, Sync sync,
                         At at, RowsShared &sh) {
    constexpr unsigned kFull = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t gw = rank * warps + wid, nw = C * warps, q = lane % L;
    const PprView p = ppr_view(a, inst, lane);
    const bool with_res = a.tol > 0.0;   // nothing is below a tolerance of zero
    // a cluster's warps have a group each of an item that can be a CTA's: the L1 change is
    // added up as that CTA's warps would (each its groups in order), so that the sweep
    // at which an item stops does not depend on the team
    const bool as_cta = C > 1 && p.n <= kCtaItem;
    // start vectors and inverse degrees, then the in-edges as pairs
    const uint32_t tid = rank * blockDim.x + threadIdx.x, nt = C * blockDim.x;
    for (uint32_t v = tid; v < p.n; v += nt) {
        const uint32_t deg = a.rowptr[p.base + v + 1] - a.rowptr[p.base + v];
        p.inv[v] = deg ? __fdiv_rn(1.0f, (float)deg) : 0.0f;
    }
    for (uint32_t i = tid; i < p.n * L; i += nt) {
        const uint32_t v = i / L, k = 4 * (i % L);
        const uint32_t *sd = a.seeds + (size_t)inst * p.K + k;
        reinterpret_cast<float4 *>(p.r0)[i] =
            make_float4(v == sd[0] ? 1.0f : 0.0f, v == sd[1] ? 1.0f : 0.0f,
                        v == sd[2] ? 1.0f : 0.0f, v == sd[3] ? 1.0f : 0.0f);
    }
    // dangling mass of the start: the seeds without out-edges (counted by CTA 0)
    if (threadIdx.x < 32) {
        unsigned long long d = 0;
        if (rank == 0 && (int)lane < p.K) {
            const uint32_t s = p.base + p.seed;
            if (a.rowptr[s + 1] == a.rowptr[s]) d = (unsigned long long)kDangOne;
        }
        sh.dang[0][lane] = d;
        sh.dang[1][lane] = 0;
        sh.seed[lane] = p.seed;   // ~0 past the K vectors
    }
    sync();
    const uint64_t e0 = a.colptr[p.base], e1 = a.colptr[p.base + p.n];
    for (uint64_t e = e0 + tid; e < e1; e += nt) {
        uint32_t u = a.rowidx[e] - p.base;
        float w = 0.0f;
        if (u >= p.n) {   // edge enters from outside the instance
            atomicOr((unsigned int *)&a.stats[2], 2u);
            u = 0;
        } else {
            w = p.inv[u];
        }
        a.ew[e] = make_uint2(u, __float_as_uint(w));
    }
    sync();
    int it = 0;
    while (it < a.max_it) {
        const int pb = it & 1;
        if (threadIdx.x < 32) {   // every CTA adds the team's masses (integers: in any order)
            unsigned long long t = 0;
            for (uint32_t r = 0; r < C; r++) t += at(&sh.dang[it % 3][0], r)[lane];
            sh.tele[lane] = fmaf(p.alpha, (float)((double)t / kDangOne), 1.0f - p.alpha);
            sh.dang[(it + 2) % 3][lane] = 0;   // read in the last sweep, added to in the next
        }
        __syncthreads();
        const float *src = pb ? p.r1 : p.r0;
        float *dst = pb ? p.r0 : p.r1;
        unsigned long long *dang = sh.dang[(it + 1) % 3];
        double res[4] = {0.0, 0.0, 0.0, 0.0};
        if (with_res)
            ppr_sweep_rows<L, true>(a, p, sh, lane, gw, nw, src, dst, dang, res);
        else
            ppr_sweep_rows<L, false>(a, p, sh, lane, gw, nw, src, dst, dang, res);
        if (with_res) {
            if (lane < L)
#pragma unroll
                for (int c = 0; c < 4; c++) sh.warp_res[pb][wid][4 * q + c] = res[c];
            if (!as_cta) {   // this CTA's warps in order
                __syncthreads();
                if (wid == 0) {
                    double t = 0.0;
                    if ((int)lane < p.K)
                        for (uint32_t w = 0; w < warps; w++) t += sh.warp_res[pb][w][lane];
                    sh.res[pb][lane] = t;
                }
            }
        }
        // orders this sweep's writes (vectors and sums) before the next sweep's reads
        sync();
        it++;
        if (with_res) {   // stop test: the same on every CTA
            if (as_cta) {   // (no CTA reads the last sweep's sums any more)
                double t = 0.0;
                for (uint32_t r = 0; r < C; r++) t += at(&sh.warp_res[pb][wid][0], r)[lane];
                sh.warp_res[pb ^ 1][wid][lane] = t;
                __syncthreads();
            }
            if (wid == 0) {
                double t = 0.0;
                if (as_cta)
                    for (uint32_t w = 0; w < warps; w++) t += sh.warp_res[pb ^ 1][w][lane];
                else
                    for (uint32_t r = 0; r < C; r++) t += at(&sh.res[pb][0], r)[lane];
                double mx = (int)lane < p.K ? t : 0.0;
#pragma unroll
                for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(kFull, mx, o));
                if (lane == 0) sh.stop = mx < a.tol;
            }
            __syncthreads();
            if (sh.stop) break;
        }
    }
    if (it & 1) {   // result is in the scratch copy
        for (uint32_t i = tid; i < p.n * L; i += nt)
            reinterpret_cast<float4 *>(p.r0)[i] = reinterpret_cast<const float4 *>(p.r1)[i];
    }
    if (tid == 0) {
        a.ppr_iters[inst] = it;
        atomicAdd(&a.stats[1], (unsigned long long)(e1 - e0) * (unsigned long long)it *
                                   (unsigned long long)p.K);
    }
    sync();   // shared state and vectors are the next item's
}

// The same by this CTA alone.
template <int L>
__device__ __forceinline__ void cta_rows_ppr(const BatchArgs &a, uint32_t inst, RowsShared &sh) {
    team_ppr<L>(
        a, inst, 1, 0, [] { __syncthreads(); }, [](auto *p, uint32_t) { return p; }, sh);
}

__device__ void cta_ppr(const BatchArgs &a, uint32_t inst) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const PprView p = ppr_view(a, inst, lane);
    const uint32_t n = p.n;
    const int K = p.K;
    __shared__ float s_d[kBatchWarps][32];
    __shared__ double s_res[kBatchWarps][32];
    __shared__ float s_dang[32];
    __shared__ int s_stop;
    // Dangling mass is always summed in the same order: each warp over its
    // vertices (v = wid, wid + W, ...), then warps 0..W-1.
    s_d[wid][lane] = ppr_init_warp(a, p, lane, wid, kBatchWarps);
    __syncthreads();
    int it = 0;
    unsigned long long visits = 0;
    while (it < a.max_it) {
        const float *src = (it & 1) ? p.r1 : p.r0;
        float *dst = (it & 1) ? p.r0 : p.r1;
        if (wid == 0) {
            float t = 0.0f;
            for (int w = 0; w < kBatchWarps; w++) t += s_d[w][lane];
            s_dang[lane] = t;
        }
        __syncthreads();
        const float dk = s_dang[lane];
        double res = 0.0;
        float dpart = 0.0f;
        ppr_sweep_warp(a, p, lane, wid, kBatchWarps, src, dst, dk, dpart, res, visits);
        s_d[wid][lane] = dpart;
        s_res[wid][lane] = res;
        __syncthreads();
        if (threadIdx.x == 0) {
            double mx = 0.0;
            for (int k = 0; k < K; k++) {
                double t = 0.0;
                for (int w = 0; w < kBatchWarps; w++) t += s_res[w][k];
                mx = t > mx ? t : mx;
            }
            s_stop = mx < a.tol;
        }
        __syncthreads();
        it++;
        if (s_stop) break;
    }
    if (it & 1) {   // result is in the scratch copy
        for (uint32_t v = wid; v < n; v += kBatchWarps)
            if (p.lk) p.r0[(size_t)v * K + lane] = p.r1[(size_t)v * K + lane];
    }
    if (threadIdx.x == 0) a.ppr_iters[inst] = it;
    if (lane == 0 && visits) atomicAdd(&a.stats[1], visits * (unsigned long long)K);
    __syncthreads();
}

// L (here and below): lanes per vertex of the rows of four vectors per lane, 0: a lane
// per vector.  Kernels of their own: with all sweeps in one, the registers of the
// others made the lane-per-vector sweep spill (K = 1 and 12: up to 1.4x slower).
template <int L>
__global__ void __launch_bounds__(kBatchThreads, 2) k_batch(BatchArgs a) {
    __shared__ union {
        uint32_t bm[3 * (kBatchMaxV / 32)];
        std::conditional_t<L != 0, RowsShared, char> rows;
    } mem;
    __shared__ uint32_t s_item;
    const uint32_t n_items = (uint32_t)a.count * a.tasks;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        __syncthreads();
        if (item >= n_items) break;
        const uint32_t inst = a.order[item / a.tasks];
        const bool bfs = a.tasks == 2 ? (item % 2 == 0) : (a.do_bfs != 0);
        if (bfs) {
            cta_bfs(a, inst, mem.bm);
        } else if constexpr (L != 0) {
            cta_rows_ppr<L>(a, inst, mem.rows);
        } else {
            cta_ppr(a, inst);
        }
    }
}

// ---- cluster version ------------------------------------------------------
// The same items, with the larger PPR items run by a whole thread-block cluster
// (16 CTAs of 1024 threads where the GPU allows it, else 8): the cluster's
// 512 (256) warps split the instance's vertices, and the per-iteration
// reductions go through distributed shared memory with one cluster barrier
// per iteration.  Only a handful of instances are in flight at a time, so
// their PPR vectors (2 x V_i x 128 B each) stay in L2 and the row gathers
// hit L2 instead of DRAM.  A solo run with the same cluster size is bitwise
// equal: nothing depends on scheduling.
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;

struct ClusterShared {
    float d[kClusterWarps][32];      // per-warp dangling mass
    double res[kClusterWarps][32];   // per-warp L1 change
    float dc[2][32];                 // CTA dangling mass, by iteration parity
    double rc[2][32];                // CTA L1 change, by iteration parity
    int stop;
};

__device__ void cluster_ppr(const BatchArgs &a, uint32_t inst, cg::cluster_group &cl,
                            ClusterShared &sh) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t C = cl.num_blocks(), crank = cl.block_rank();
    const uint32_t gw = crank * kClusterWarps + wid, nw = C * kClusterWarps;
    const PprView p = ppr_view(a, inst, lane);
    const int K = p.K;
    // dangling mass: each warp in vertex order, then warps 0..31 of a CTA,
    // then CTAs 0..C-1 (every CTA forms the same sum)
    sh.d[wid][lane] = ppr_init_warp(a, p, lane, gw, nw);
    __syncthreads();
    if (wid == 0) {
        float t = 0.0f;
        for (int w = 0; w < kClusterWarps; w++) t += sh.d[w][lane];
        sh.dc[0][lane] = t;
    }
    cl.sync();
    int it = 0;
    unsigned long long visits = 0;
    while (it < a.max_it) {
        const int pb = it & 1;
        float dk = 0.0f;
        for (uint32_t r = 0; r < C; r++) dk += cl.map_shared_rank(&sh.dc[pb][0], r)[lane];
        const float *src = pb ? p.r1 : p.r0;
        float *dst = pb ? p.r0 : p.r1;
        double res = 0.0;
        float dpart = 0.0f;
        ppr_sweep_warp(a, p, lane, gw, nw, src, dst, dk, dpart, res, visits);
        sh.d[wid][lane] = dpart;
        sh.res[wid][lane] = res;
        __syncthreads();
        if (wid == 0) {
            float t = 0.0f;
            double q = 0.0;
            for (int w = 0; w < kClusterWarps; w++) {
                t += sh.d[w][lane];
                q += sh.res[w][lane];
            }
            sh.dc[pb ^ 1][lane] = t;
            sh.rc[pb ^ 1][lane] = q;
        }
        // orders this sweep's writes (vectors and partials) before every
        // CTA's reads of the next sweep, cluster wide
        cl.sync();
        if (wid == 0) {   // stop test: the same on every CTA
            double tot = 0.0;
            for (uint32_t r = 0; r < C; r++) tot += cl.map_shared_rank(&sh.rc[pb ^ 1][0], r)[lane];
            double mx = (int)lane < K ? tot : 0.0;
#pragma unroll
            for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) sh.stop = mx < a.tol;
        }
        __syncthreads();
        it++;
        if (sh.stop) break;
    }
    if (it & 1) {   // result is in the scratch copy
        for (uint32_t v = gw; v < p.n; v += nw)
            if (p.lk) p.r0[(size_t)v * K + lane] = p.r1[(size_t)v * K + lane];
    }
    if (crank == 0 && threadIdx.x == 0) a.ppr_iters[inst] = it;
    if (lane == 0 && visits) atomicAdd(&a.stats[1], visits * (unsigned long long)K);
}

template <int L>
__global__ void __launch_bounds__(kClusterThreads, 1) k_batch_cluster(BatchArgs a) {
    __shared__ union {
        std::conditional_t<L != 0, RowsShared, ClusterShared> sh;
        uint32_t bm[3 * (kBatchMaxV / 32)];   // BFS, after the PPR items
    } mem;
    auto &sh = mem.sh;
    __shared__ uint32_t s_item;
    cg::cluster_group cl = cg::this_cluster();
    // the cluster's items first, largest first (counter[1], taken by CTA 0), then
    // the CTA's, then BFS: the smaller ones level the CTAs' ends
    if (a.do_ppr) {
        for (;;) {
            if (cl.block_rank() == 0 && threadIdx.x == 0) s_item = atomicAdd(&a.counter[1], 1u);
            cl.sync();
            const uint32_t item = *cl.map_shared_rank(&s_item, 0);
            if (item >= a.n_large) break;
            if constexpr (L != 0)
                team_ppr<L>(
                    a, a.order[item], cl.num_blocks(), cl.block_rank(), [&] { cl.sync(); },
                    [&](auto *p, uint32_t r) { return cl.map_shared_rank(p, r); }, sh);
            else
                cluster_ppr(a, a.order[item], cl, sh);
        }
        cl.sync();   // the last item's number has been read by every CTA
        if constexpr (L != 0) {
            for (;;) {
                __syncthreads();
                if (threadIdx.x == 0) s_item = a.n_large + atomicAdd(&a.counter[2], 1u);
                __syncthreads();
                const uint32_t item = s_item;
                if (item >= (uint32_t)a.count) break;
                cta_rows_ppr<L>(a, a.order[item], sh);
            }
            __syncthreads();
        }
    }
    if (a.do_bfs) {   // BFS items: one CTA each (counter[0])
        for (;;) {
            if (threadIdx.x == 0) s_item = atomicAdd(&a.counter[0], 1u);
            __syncthreads();
            const uint32_t item = s_item;
            __syncthreads();
            if (item >= (uint32_t)a.count) break;
            cta_bfs(a, a.order[item], mem.bm);
        }
    }
    cl.sync();   // no CTA leaves while another may still read its shared memory
}

using BatchKernel = void (*)(BatchArgs);
static BatchKernel batch_kernel(const BatchArgs &a, BatchKernel k32, BatchKernel k16, BatchKernel k8,
                                BatchKernel k4, BatchKernel other) {
    if (!a.ew) return other;
    return a.K == 32 ? k32 : a.K == 16 ? k16 : a.K == 8 ? k8 : k4;
}

// Which of the items (sizes, largest first) the clusters take: those above kCtaItem,
// and of the others the largest ones where that ends the call earlier.  The times are
// estimates in ns a sweep.  An item takes a cluster a barrier, a chain of loads of its
// row's length, and a thirtieth of its work; a CTA its work, per vertex and per in-edge
// (measured: K = 4..32, 60..4000 vertices, 2..24 in-edges each, within about 30 %).  The
// clusters' items come first, then the CTAs take the rest, which ends with the largest
// or when all CTAs have had their share.  20 sweeps, K = 32, equal items of eight
// in-edges a vertex, all on clusters / all on CTAs, us: one of 250 vertices 152 / 151, of
// 2000 166 / 769; 28 of 250 424 / 167, of 2000 514 / 788; 96 of 2000 1471 / 801.
static uint32_t choose_large(const std::vector<uint32_t> &sizes, double deg, int K, int C,
                             int clusters) {
    const size_t count = sizes.size();
    size_t m = 0;
    while (m < count && sizes[m] > kCtaItem) m++;
    // the smaller ones' sums need a group of vertices a warp (team_ppr)
    if ((uint64_t)C * (kClusterThreads / 32) * (128 / K) < kCtaItem) return (uint32_t)m;
    auto cta = [&](size_t i) { return sizes[i] * (0.22 * K + (0.4 + 0.025 * K) * deg); };
    auto cluster = [&](size_t i) { return 3000.0 + deg * (130.0 + 1200.0 / K) + cta(i) / 30; };
    std::vector<double> busy(clusters, 0.0);   // until when each cluster is
    auto give = [&](size_t i) { *std::min_element(busy.begin(), busy.end()) += cluster(i); };
    double rest = 0, best = 0;
    for (size_t i = 0; i < m; i++) give(i);
    for (size_t i = m; i < count; i++) rest += cta(i);
    uint32_t at = (uint32_t)m;
    for (size_t i = m;; i++) {   // items [0, i) on clusters
        const double end = *std::max_element(busy.begin(), busy.end()) +
                           (i < count ? std::max(cta(i), rest / (clusters * C)) : 0.0);
        if (i == m || end < best) {
            best = end;
            at = (uint32_t)i;
        }
        if (i == count) return at;
        give(i);
        rest -= cta(i);
    }
}

// Launch k_batch_cluster with `want` CTAs per cluster (8 or 16), or with the
// largest size the GPU runs when want = 1; one CTA per SM.  *launched =
// false when no wanted size is available.
static int launch_batch_cluster(BatchArgs a, const std::vector<uint32_t> &sizes, double deg,
                                int num_sms, cudaStream_t s, int want, bool *launched,
                                int *cluster_size) {
    *launched = false;
    const auto kernel = batch_kernel(a, k_batch_cluster<8>, k_batch_cluster<4>, k_batch_cluster<2>,
                                     k_batch_cluster<1>, k_batch_cluster<0>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
        cudaSuccess)
        cudaGetLastError();
    for (int C : {16, 8}) {
        if (want != 1 && want != C) continue;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = C;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(C * std::max(1, num_sms / C));
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int ncl = 0;
        if (cudaOccupancyMaxActiveClusters(&ncl, kernel, &cfg) != cudaSuccess || ncl < 1) {
            cudaGetLastError();
            continue;
        }
        ncl = std::min(ncl, std::max(1, num_sms / C));
        cfg.gridDim = dim3(C * ncl);
        a.n_large = a.ew ? choose_large(sizes, deg, a.K, C, ncl) : (uint32_t)a.count;
        OLV_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
        *launched = true;
        *cluster_size = C;
        return OLV_OK;
    }
    return OLV_OK;
}

// Device buffers of olv_batch_run, kept with the graph between calls (they
// only grow), so a call allocates nothing once the sizes have been seen.
struct BatchState {
    DevBuf off, order, seeds, tmp, inv, ew, counter, iters, stats, levels, ppr;
    ~BatchState() {
        off.release(); order.release(); seeds.release(); tmp.release(); inv.release(); ew.release();
        counter.release();
        iters.release(); stats.release(); levels.release(); ppr.release();
    }
};

void release_batch_state(olv_graph *g) {
    delete static_cast<BatchState *>(g->batch_state);
    g->batch_state = nullptr;
}

}  // namespace olv

using namespace olv;

extern "C" int olv_batch_run(olv_graph *g, const uint32_t *inst_offsets, int count, int K,
                             const uint32_t *seeds, double alpha, int max_it, double tol,
                             int32_t *levels_out, float *ppr_out, uint32_t *ppr_iters_out,
                             olv_stats *st) {
    OLV_CHECK_ARG(g && inst_offsets, "olv_batch_run: null pointer");
    BufferScope scope(g->stream);
    OLV_CHECK_ARG(count >= 1, "olv_batch_run: count must be >= 1");
    OLV_CHECK_ARG(levels_out || ppr_out, "olv_batch_run: nothing to compute");
    OLV_CHECK_ARG(!ppr_out || (seeds && K >= 1 && K <= 32),
                  "olv_batch_run: PPR needs seeds and 1 <= K <= 32");
    OLV_CHECK_ARG(alpha >= 0 && alpha < 1 && max_it >= 0, "olv_batch_run: bad alpha / max_it");
    std::vector<uint32_t> off(count + 1);
    if (is_device_ptr(inst_offsets))
        OLV_CUDA(cudaMemcpy(off.data(), inst_offsets, (count + 1) * 4, cudaMemcpyDeviceToHost));
    else
        memcpy(off.data(), inst_offsets, (count + 1) * 4);
    OLV_CHECK_ARG(off[count] <= g->V, "olv_batch_run: offsets exceed the graph");
    for (int i = 0; i < count; i++) {
        OLV_CHECK_ARG(off[i + 1] > off[i], "olv_batch_run: empty or decreasing instance %d", i);
        if (off[i + 1] - off[i] > kBatchMaxV) {
            set_error("olv_batch_run: instance %d has %u vertices (limit %u)", i,
                      off[i + 1] - off[i], kBatchMaxV);
            return OLV_ERR_LIMIT;
        }
    }
    const int K_ = ppr_out ? K : 0;
    std::vector<uint32_t> hseeds;
    if (ppr_out) {
        hseeds.resize((size_t)count * K);
        if (is_device_ptr(seeds))
            OLV_CUDA(cudaMemcpy(hseeds.data(), seeds, hseeds.size() * 4, cudaMemcpyDeviceToHost));
        else
            memcpy(hseeds.data(), seeds, hseeds.size() * 4);
        for (int i = 0; i < count; i++)
            for (int k = 0; k < K; k++)
                OLV_CHECK_ARG(hseeds[(size_t)i * K + k] < off[i + 1] - off[i],
                              "olv_batch_run: seed %d of instance %d out of range", k, i);
    }
    // largest instances first
    std::vector<uint32_t> order(count);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
        return off[x + 1] - off[x] > off[y + 1] - off[y];
    });
    if (!g->batch_state) g->batch_state = new BatchState();
    BatchState &bs = *static_cast<BatchState *>(g->batch_state);
    cudaStream_t s = g->stream;
    const size_t V = off[count];
    OLV_TRY(bs.off.ensure((count + 1) * 4));
    OLV_TRY(bs.order.ensure(count * 4));
    OLV_TRY(bs.counter.ensure(16));
    OLV_TRY(bs.iters.ensure(count * 4 + 16));
    OLV_TRY(bs.stats.ensure(32));
    OLV_CUDA(cudaMemcpyAsync(bs.off.p, off.data(), (count + 1) * 4, cudaMemcpyHostToDevice, s));
    OLV_CUDA(cudaMemcpyAsync(bs.order.p, order.data(), count * 4, cudaMemcpyHostToDevice, s));
    const bool dev_lv = levels_out && is_device_ptr(levels_out);
    const bool dev_pr = ppr_out && is_device_ptr(ppr_out);
    if (levels_out && !dev_lv) OLV_TRY(bs.levels.ensure(V * 4));
    if (ppr_out) {
        OLV_TRY(bs.seeds.ensure(hseeds.size() * 4));
        OLV_CUDA(cudaMemcpyAsync(bs.seeds.p, hseeds.data(), hseeds.size() * 4,
                                 cudaMemcpyHostToDevice, s));
        OLV_TRY(bs.tmp.ensure(V * K * 4));
        OLV_TRY(bs.inv.ensure(V * 4));
        if (!dev_pr) OLV_TRY(bs.ppr.ensure(V * K * 4));
    }
    BatchArgs a;
    a.rowptr = g->rowptr.as<uint32_t>();
    a.col = g->col.as<uint32_t>();
    a.colptr = g->colptr.as<uint32_t>();
    a.rowidx = g->rowidx.as<uint32_t>();
    a.inst_off = bs.off.as<uint32_t>();
    a.order = bs.order.as<uint32_t>();
    a.seeds = bs.seeds.as<uint32_t>();
    a.count = count;
    a.K = K_;
    a.max_it = max_it;
    a.do_bfs = levels_out != nullptr;
    a.do_ppr = ppr_out != nullptr;
    a.tasks = a.do_bfs + a.do_ppr;
    a.alpha = (float)alpha;
    a.tol = tol;
    a.levels = levels_out ? (dev_lv ? levels_out : bs.levels.as<int32_t>()) : nullptr;
    a.ppr = ppr_out ? (dev_pr ? ppr_out : bs.ppr.as<float>()) : nullptr;
    a.ppr_tmp = bs.tmp.as<float>();
    a.inv_deg = bs.inv.as<float>();
    // rows of four vectors per lane need whole 16-byte rows
    bool rows = ppr_out && (K == 4 || K == 8 || K == 16 || K == 32) &&
                (((uintptr_t)a.ppr | (uintptr_t)a.ppr_tmp) & 15) == 0;
    if (rows && bs.ew.ensure(g->E * 8 + 16) != OLV_OK) {   // no room for the pairs
        cudaGetLastError();
        rows = false;
    }
    a.ew = rows ? bs.ew.as<uint2>() : nullptr;
    std::vector<uint32_t> sizes(count);
    for (int i = 0; i < count; i++) sizes[i] = off[order[i] + 1] - off[order[i]];
    a.counter = bs.counter.as<uint32_t>();
    a.ppr_iters = bs.iters.as<uint32_t>();
    a.stats = bs.stats.as<unsigned long long>();
    OLV_CUDA(cudaEventRecord(g->ev0, s));
    OLV_CUDA(cudaMemsetAsync(bs.counter.p, 0, 16, s));
    OLV_CUDA(cudaMemsetAsync(bs.stats.p, 0, 32, s));
    bool launched = false;
    int csize = 0;
    if (g->tune.batch_cluster)
        OLV_TRY(launch_batch_cluster(a, sizes, (double)g->E / g->V, g->num_sms, s,
                                     g->tune.batch_cluster, &launched, &csize));
    if (!launched) {   // one CTA per item
        const auto kernel = batch_kernel(a, k_batch<8>, k_batch<4>, k_batch<2>, k_batch<1>, k_batch<0>);
        int per_sm = 0;
        OLV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBatchThreads, 0));
        const int grid = std::max(1, per_sm) * g->num_sms;
        kernel<<<grid, kBatchThreads, 0, s>>>(a);
    }
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaEventRecord(g->ev1, s));
    unsigned long long hst[3];
    OLV_CUDA(cudaMemcpyAsync(hst, bs.stats.p, 24, cudaMemcpyDeviceToHost, s));
    if (levels_out && !dev_lv)
        OLV_CUDA(cudaMemcpyAsync(levels_out, a.levels, V * 4, cudaMemcpyDeviceToHost, s));
    if (ppr_out && !dev_pr)
        OLV_CUDA(cudaMemcpyAsync(ppr_out, a.ppr, V * K * 4, cudaMemcpyDeviceToHost, s));
    if (ppr_iters_out)
        OLV_CUDA(cudaMemcpyAsync(ppr_iters_out, bs.iters.p, count * 4, cudaMemcpyDefault, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    g->launches = 1;
    if (hst[2]) {
        set_error("olv_batch_run: the graph is not block-diagonal under inst_offsets "
                  "(edges cross instances; code %llu)", hst[2]);
        return OLV_ERR_ARG;
    }
    if (st) {
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        st->iterations = (uint32_t)count;
        st->pull_steps = 0;
        st->vertices_reached = V;
        st->edges_traversed = hst[0];   // BFS: out-edges of reached vertices, all instances
        st->edges_relaxed = hst[1];     // PPR: in-edge visits x K, all iterations
        st->residual = 0;
        st->device_ms = ms;
    }
    return OLV_OK;
}
