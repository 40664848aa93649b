// PageRank: deterministic FP32 pull over the reverse graph.
//
// Result contract: PageRank.cu:89-147 / testPageRank.cu:41-115 -- ranks start
// at 1/N; each iteration r'[v] = (1-alpha)/N + alpha * sum_{u->v} r[u]/outdeg(u)
// (+ alpha * d/N with d the dangling mass when it is redistributed); stop when
// the L1 change sum|r' - r| < tol or after max_it iterations.
//
// The reference pushes rank/outdeg along out-edges with an FP64 CAS atomicAdd
// (PageRank.cu:51-61, common.h:141-150), refills the V accumulators on the host
// every iteration (oliver.h:127) and copies all vertex values back to sum the
// residual on the host (oliver.h:176-183).  Here:
//   * the solve runs on a relabelled copy of the reverse graph (CSC): vertices
//     renumbered by in-degree, longest rows first, built once per graph.  Ranks,
//     contributions r/outdeg and out-degrees live in the new order; the ranks
//     are mapped back to the caller's ids once, at the end of the solve;
//   * each iteration is one pull pass over the in-edges: a group of 1..32
//     lanes per row (by row length) sums the row's contributions in a fixed
//     order with compensated (two-sum) FP32 arithmetic, so results do not
//     depend on scheduling and carry ~1 rounding per vertex;
//   * the same pass writes the next iteration's contributions r/outdeg and
//     per-CTA FP64 partial sums of |r' - r| and of the dangling mass, which are
//     folded in a fixed order and decide convergence on the device.
//
// Two ways to run the iterations.  All of them in one launch (olv_rowsolve.cuh)
// where launches and the loop around them were most of the time, and on graphs
// without a segmented row that have work enough per row; else an iteration is a tile
// pass and a one-CTA fold inside a CUDA graph (olv_rowtiles.cuh), which reads the hubs'
// rows faster (no counts and fences among the gathers) and passes over rows of few
// entries faster.  The line is one_launch()'s.
#include <algorithm>
#include <vector>

#include "olive_b200/olv_advance.cuh"
#include "olv_graphexec.cuh"
#include "olv_internal.cuh"
#include "olv_rowsolve.cuh"
#include "olv_rowtiles.cuh"

namespace olv {

constexpr int kRedThreads = 1024;   // 32 warps: one more tree over them

struct PrCtl {
    double base;        // (1-alpha)/N + alpha*d/N for the running iteration
    double residual;    // L1 change of the last completed iteration
    double dangling;
    uint32_t iter;      // completed iterations
    uint32_t done;
    uint32_t max_it;
    uint32_t leak;
    double tol;
    double alpha;
    double inv_n;
};

// r' = alpha * (s + c) + base, with alpha split into hi + lo FP32 parts.
__device__ __forceinline__ float pr_update(float s, float c, float a_hi, float a_lo, float base) {
    const float t = fmaf(a_lo, s, fmaf(a_hi, c, base));
    return fmaf(a_hi, s, t);
}

// Row sums over in-edges of the contributions r[u]/outdeg(u); the row update
// writes the rank, the next contribution and FP64 |r'-r| / dangling partials
// (olv_rowtiles.cuh).
struct PrTileOp {
    const uint32_t *done;
    const PrCtl *ctl;
    const float *c0, *c1;
    float *rank;
    const uint32_t *outdeg;
    const float *cin;
    float *cout;
    float a_hi, a_lo;   // alpha as an unevaluated FP32 pair: the update carries FP64-level
                        // alpha (parameters: read from the control block they took two
                        // registers more and were no faster)
    float base;

    __device__ __forceinline__ void begin() {
        const bool odd = ctl->iter & 1;
        cin = odd ? c1 : c0;
        cout = const_cast<float *>(odd ? c0 : c1);
        base = (float)ctl->base;
    }
    __device__ __forceinline__ float term(uint32_t, uint32_t j) const { return __ldg(&cin[j]); }
    struct Row {
        float old;       // rank before this iteration
        uint32_t deg;    // out-degree
    };
    __device__ __forceinline__ Row row(uint32_t v) const { return Row{rank[v], __ldg(&outdeg[v])}; }
    __device__ __forceinline__ void finish(uint32_t v, float s, float c, const Row &r, double &res,
                                           double &dang) const {
        const float nr = pr_update(s, c, a_hi, a_lo, base);
        rank[v] = nr;
        res += fabs((double)nr - (double)r.old);
        if (r.deg) {
            cout[v] = __fdiv_rn(nr, (float)r.deg);
        } else {
            cout[v] = 0.0f;
            dang += (double)nr;
        }
    }
};

// The same for a whole solve in one launch (olv_rowsolve.cuh).
struct PrOp {
    static constexpr bool kGather = true, kWeighted = false, kStore = true;
    float *c0, *c1;            // contributions, ping-pong
    float *rank;
    const uint32_t *outdeg;
    const SolveCtl *ctl;
    float a_hi, a_lo;
    double alpha, inv_n;
    int leak;
    float rank0;
    float base;
    uint32_t odd;

    // dangling mass of the start: an exact count, so that the first constant
    // term does not depend on the order of atomics
    __device__ __forceinline__ double first_aux() const {
        return (double)ctl->count * (double)rank0;
    }
    __device__ __forceinline__ void begin(uint32_t it, double dang) {
        odd = it & 1;
        base = (float)((1.0 - alpha) * inv_n + (leak ? 0.0 : alpha * dang * inv_n));
    }
    __device__ __forceinline__ const float *in() const { return odd ? c1 : c0; }
    __device__ __forceinline__ float *out() const { return odd ? c0 : c1; }
    struct Row {
        float old;       // rank before this iteration
        uint32_t deg;    // out-degree
    };
    __device__ __forceinline__ Row row(uint32_t v) const { return Row{rank[v], __ldg(&outdeg[v])}; }
    __device__ __forceinline__ float finish(uint32_t v, float s, float c, const Row &r, double &res,
                                            double &dang) const {
        const float nr = pr_update(s, c, a_hi, a_lo, base);
        rank[v] = nr;
        res += fabs((double)nr - (double)r.old);
        if (r.deg) return __fdiv_rn(nr, (float)r.deg);
        dang += (double)nr;
        return 0.0f;
    }
};

// Fold the per-CTA partials (fixed order), publish residual and the next
// iteration's constant term, decide convergence.
__global__ void __launch_bounds__(kRedThreads)
k_pr_reduce(PrCtl *ctl, const double *__restrict__ partials, uint32_t nparts,
            cudaGraphConditionalHandle h, int use_cond) {
    __shared__ double s[2][kRedThreads / 32];
    if (ctl->done) {
        if (use_cond && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    double a = 0, b = 0;
    for (uint32_t i = threadIdx.x; i < nparts; i += kRedThreads) {
        const double2 p = reinterpret_cast<const double2 *>(partials)[i];
        a += p.x;
        b += p.y;
    }
    // a tree over each warp, then over the warps (one barrier)
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s[0][threadIdx.x >> 5] = a;
        s[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    a = s[0][threadIdx.x];
    b = s[1][threadIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (threadIdx.x == 0) {
        const double res = a, dang = b;
        ctl->residual = res;
        ctl->dangling = dang;
        ctl->iter++;
        ctl->base = (1.0 - ctl->alpha) * ctl->inv_n +
                    (ctl->leak ? 0.0 : ctl->alpha * dang * ctl->inv_n);
        if (res < ctl->tol || ctl->iter >= ctl->max_it) ctl->done = 1;
        if (use_cond) cudaGraphSetConditional(h, ctl->done ? 0u : 1u);
    }
}

// r = 1/N, contributions r/outdeg, count of dangling vertices (exact integer
// count, so the first constant term does not depend on atomic ordering).
__global__ void k_pr_init(const uint32_t *__restrict__ outdeg, uint32_t V, float *rank, float *c0,
                          unsigned long long *ndang) {
    const float r = __fdiv_rn(1.0f, (float)V);
    unsigned long long nd = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
         v += (uint64_t)gridDim.x * blockDim.x) {
        rank[v] = r;
        const uint32_t d = outdeg[v];
        c0[v] = d ? __fdiv_rn(r, (float)d) : 0.0f;
        nd += d == 0;
    }
    warp_add64(nd, ndang);
}

__global__ void k_pr_ctl_init(PrCtl *ctl, const unsigned long long *ndang, uint32_t V,
                              double alpha, uint32_t max_it, double tol, uint32_t leak) {
    PrCtl c = {};
    c.alpha = alpha;
    c.inv_n = 1.0 / (double)V;
    c.tol = tol;
    c.max_it = max_it;
    c.leak = leak;
    const double dang = (double)(*ndang) * (double)__fdiv_rn(1.0f, (float)V);
    c.dangling = dang;
    c.base = (1.0 - alpha) * c.inv_n + (leak ? 0.0 : alpha * dang * c.inv_n);
    c.residual = 0;
    c.done = max_it == 0;
    *ctl = c;
}

// out-degree of every vertex, in the relabelled order
__global__ void k_outdeg_perm(const uint32_t *__restrict__ rowptr,
                              const uint32_t *__restrict__ perm, uint32_t V, uint32_t *d) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = perm[i];
        d[i] = rowptr[v + 1] - rowptr[v];
    }
}

// rank[v] = rank of v's new id (coalesced writes, gathers from an L2-sized array)
__global__ void k_pr_unpermute(const float *__restrict__ rank_new,
                               const uint32_t *__restrict__ newid, uint32_t V,
                               float *__restrict__ rank) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
         v += (uint64_t)gridDim.x * blockDim.x)
        rank[v] = rank_new[newid[v]];
}

// ------------------------------------------------------------------ host --
struct PrPlan {
    bool solve = false;        // one launch for all iterations
    SolvePlan sp;              // ... its structure,
    TilePlan tp;               // or that of the tile pass
    DevBuf outdeg, contrib, rank, ctl, dang;   // outdeg, contrib, rank: new order
    const uint32_t *perm() const { return (solve ? sp.perm : tp.perm).as<uint32_t>(); }
    const uint32_t *newid() const { return (solve ? sp.newid : tp.newid).as<uint32_t>(); }
    ~PrPlan() {
        sp.release(); tp.release(); outdeg.release(); contrib.release(); rank.release();
        ctl.release(); dang.release();
    }
};

// One launch for all iterations, or a pass each.  Measured from one build, us for 20
// iterations, one launch / a pass each:
//   uniform digraphs, edges a vertex: 2^17 vertices, 2: 211 / 268, 8: 273 / 307;
//   262,144, 1: 310 / 285, 3: 345 / 304, 4: 328 / 329, 8: 358 / 408; 524,288, 1: 399 /
//   332, 4: 413 / 430, 12: 726 / 773; 1,000,003, 1: 579 / 418, 2: 559 / 496, 4: 613 /
//   603, 8: 861 / 875; 2,000,003, 1: 903 / 620, 2: 891 / 739; 2^21, 16: 2932 / 3181;
//   grids of 490,000 and 4 M vertices 265 / 342, 929 / 1265;
//   RMAT, edges drawn a vertex: 2^16, 16: 346 / 420; 2^17, 4: 308 / 451, 16: 497 / 519,
//   24 (2.9 M edges): 516 / 456; 200,003, 8: 475 / 446; 2^18, 1: 314 / 426, 8: 534 / 513,
//   12 (3 M): 611 / 563; 300,007, 1: 436 / 330, 8 (1.3 M): 393 / 501, 16: 580 / 481;
//   370,001, 4 (1 M): 541 / 452, 8 (2 M): 430 / 527, 16: 621 / 538; 440,009, 8 (2.9 M):
//   732 / 595; 2^19, 2: 647 / 560, 8: 817 / 638; 2^20, 16: 1611 / 1117.
static bool one_launch(const olv_graph *g) {
    const bool few = g->E < 2u << 20;
    if (few && g->V <= 1u << 18) return true;
    const bool rows_long_enough = 2 * g->E >= 7 * (uint64_t)g->V;
    return rows_long_enough && (g->max_in_degree <= kRowLong || (few && g->V <= 3u << 17));
}

bool pr_tile_u_matters(const olv_graph *g) {
    return !one_launch(g) || solve_lanes_free(g->E, g->V, g->num_sms);
}

static int build_pr_plan(olv_graph *g, PrPlan &p) {
    const uint32_t V = g->V;
    p.solve = one_launch(g);
    if (p.solve) {
        OLV_TRY(build_solve_plan(g->colptr.as<uint32_t>(), g->rowidx.as<uint32_t>(), nullptr, V,
                                 g->E, g->tune.pr_tile_u, false, g->num_sms, g->stream, p.sp));
        choose_form<PrOp>(p.sp);
    } else {
        OLV_TRY(build_tile_plan(g->colptr.as<uint32_t>(), g->rowidx.as<uint32_t>(), V, g->stream,
                                p.tp, g->tune.pr_tile_u));
    }
    OLV_TRY(p.outdeg.ensure((size_t)V * 4 + 16));
    k_outdeg_perm<<<g->num_sms * 8, kBlock, 0, g->stream>>>(g->rowptr.as<uint32_t>(), p.perm(), V,
                                                           p.outdeg.as<uint32_t>());
    OLV_TRY(p.contrib.ensure((size_t)V * 8 + 64));
    OLV_TRY(p.rank.ensure((size_t)V * 4 + 16));
    OLV_TRY(p.ctl.ensure(sizeof(PrCtl)));
    OLV_TRY(p.dang.ensure(16));
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaStreamSynchronize(g->stream));
    return OLV_OK;
}

template <class Sink>
static int pr_iteration(olv_graph *g, PrPlan &p, double alpha, Sink &&sink, cudaGraphConditionalHandle h,
                        int use_cond) {
    PrCtl *ctl = p.ctl.as<PrCtl>();
    PrTileOp op;
    op.done = &ctl->done;
    op.ctl = ctl;
    op.c0 = p.contrib.as<float>();
    op.c1 = p.contrib.as<float>() + g->V;
    op.rank = p.rank.as<float>();
    op.outdeg = p.outdeg.as<uint32_t>();
    op.cin = nullptr;
    op.cout = nullptr;
    op.a_hi = (float)alpha;
    op.a_lo = (float)(alpha - (double)op.a_hi);
    op.base = 0;
    OLV_TRY(tile_pass(p.tp, op, sink));
    const double *cpart = p.tp.partials.as<double>();
    uint32_t nparts = kTileCTAs;
    void *a_red[] = {&ctl, &cpart, &nparts, &h, &use_cond};
    OLV_TRY(sink((const void *)k_pr_reduce, dim3(1), dim3(kRedThreads), a_red));
    return OLV_OK;
}

}  // namespace olv

using namespace olv;

struct PrState {
    PrPlan plan;
    WhileGraph graph;
    double graph_alpha = -1;   // the graph's kernels have alpha as a parameter
};

static PrState *pr_state(olv_graph *g) { return static_cast<PrState *>(g->pr_state); }

void olv::release_pr_state(olv_graph *g) {
    PrState *s = pr_state(g);
    if (s) {
        s->graph.destroy();
        delete s;
    }
    g->pr_state = nullptr;
}

extern "C" int olv_pagerank(olv_graph *g, double alpha, int max_it, double tol, int dangling_mode,
                            float *rank_out, olv_stats *st) {
    OLV_CHECK_ARG(g && rank_out, "olv_pagerank: null pointer");
    BufferScope scope(g->stream);
    OLV_CHECK_ARG(alpha >= 0.0 && alpha < 1.0, "olv_pagerank: alpha must be in [0,1)");
    OLV_CHECK_ARG(max_it >= 0, "olv_pagerank: max_it must be >= 0");
    OLV_CHECK_ARG(dangling_mode == OLV_DANGLING_UNIFORM || dangling_mode == OLV_DANGLING_LEAK,
                  "olv_pagerank: bad dangling_mode %d", dangling_mode);
    cudaStream_t s = g->stream;
    PrState *ps = pr_state(g);
    if (!ps) {
        ps = new PrState();
        g->pr_state = ps;
        int r = build_pr_plan(g, ps->plan);
        if (r != OLV_OK) {
            release_pr_state(g);
            return r;
        }
    }
    PrPlan &p = ps->plan;
    const double ad = alpha;
    const bool dev_out = is_device_ptr(rank_out);
    if (!dev_out) OLV_TRY(g->ws.level.ensure((size_t)g->V * 4 + 16));
    float *rank = dev_out ? rank_out : g->ws.level.as<float>();
    float *rank_new = p.rank.as<float>();

    const uint32_t leak = dangling_mode == OLV_DANGLING_LEAK ? 1u : 0u;
    SolveCtl *sctl = p.sp.ctl.as<SolveCtl>();
    bool launched = false;   // the passes as one graph
    OLV_CUDA(cudaEventRecord(g->ev0, s));
    if (p.solve)
        OLV_CUDA(cudaMemsetAsync(sctl, 0, sizeof(SolveCtl), s));
    else
        OLV_CUDA(cudaMemsetAsync(p.dang.p, 0, 8, s));
    k_pr_init<<<g->num_sms * 8, kBlock, 0, s>>>(
        p.outdeg.as<uint32_t>(), g->V, rank_new, p.contrib.as<float>(),
        p.solve ? &sctl->count : p.dang.as<unsigned long long>());
    OLV_CUDA(cudaGetLastError());
    if (p.solve) {
        PrOp op = {};
        op.c0 = p.contrib.as<float>();
        op.c1 = op.c0 + (((size_t)g->V + 3) & ~(size_t)3);   // 16-byte aligned
        op.rank = rank_new;
        op.outdeg = p.outdeg.as<uint32_t>();
        op.ctl = sctl;
        op.alpha = ad;
        op.a_hi = (float)ad;
        op.a_lo = (float)(ad - (double)op.a_hi);
        op.inv_n = 1.0 / (double)g->V;
        op.leak = (int)leak;
        op.rank0 = 1.0f / (float)g->V;
        OLV_TRY(launch_solve(p.sp, p.sp.args((uint32_t)max_it, tol), op, s));
    } else {
        k_pr_ctl_init<<<1, 1, 0, s>>>(p.ctl.as<PrCtl>(), p.dang.as<unsigned long long>(), g->V, ad,
                                      (uint32_t)max_it, tol, leak);
        OLV_CUDA(cudaGetLastError());
        if (g->tune.use_graphs && max_it > 0) {
            if (ps->graph.ready && ps->graph_alpha != ad) ps->graph.destroy();
            if (!ps->graph.ready) {
                ps->graph_alpha = ad;
                int r = ps->graph.begin();
                auto sink = [&](const void *f, dim3 gr, dim3 bl, void **args) {
                    return ps->graph.add(f, gr, bl, args);
                };
                if (r == OLV_OK) r = pr_iteration(g, p, ad, sink, ps->graph.handle, 1);
                if (r == OLV_OK) r = ps->graph.finish();
                if (r != OLV_OK) ps->graph.destroy();
            }
            if (ps->graph.ready) {
                OLV_TRY(ps->graph.launch(s));
                launched = true;
            }
        }
        if (!launched) {
            auto launch = [&](const void *f, dim3 gr, dim3 bl, void **args) {
                OLV_CUDA(cudaLaunchKernel(f, gr, bl, args, 0, s));
                return OLV_OK;
            };
            for (int it = 0; it < max_it; it++) OLV_TRY(pr_iteration(g, p, ad, launch, 0, 0));
        }
    }
    k_pr_unpermute<<<g->num_sms * 8, kBlock, 0, s>>>(rank_new, p.newid(), g->V, rank);
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaEventRecord(g->ev1, s));
    PrCtl hc = {};
    SolveCtl hs = {};
    if (p.solve)
        OLV_CUDA(cudaMemcpyAsync(&hs, sctl, sizeof hs, cudaMemcpyDeviceToHost, s));
    else
        OLV_CUDA(cudaMemcpyAsync(&hc, p.ctl.p, sizeof hc, cudaMemcpyDeviceToHost, s));
    if (!dev_out)
        OLV_CUDA(cudaMemcpyAsync(rank_out, rank, (size_t)g->V * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    OLV_TRY(solve_error(hs, p.sp, s, "olv_pagerank"));
    g->launches = 3;   // init, one solve, map back
    if (p.solve) {
        hc.iter = hs.iter;
        hc.residual = hs.residual;
    } else {   // init, control, the passes, map back
        g->launches += (p.tp.nsegs ? 3ull : 2ull) * (launched ? hc.iter : (uint32_t)max_it);
    }
    if (st) {
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        st->iterations = hc.iter;
        st->pull_steps = 0;
        st->vertices_reached = g->V;
        st->edges_traversed = g->E * (uint64_t)hc.iter;
        st->edges_relaxed = g->E * (uint64_t)hc.iter;
        st->residual = hc.residual;
        st->device_ms = ms;
    }
    return OLV_OK;
}
