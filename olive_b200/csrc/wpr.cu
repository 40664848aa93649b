// Differentiable weighted PageRank (no reference counterpart).
//
//   W_u = sum_v w_uv,  P_uv = w_uv / W_u  (rows without out-edges are zero)
//   forward:  r = (1-alpha) p + alpha P^T r        (pull over the CSC)
//   adjoint:  lambda = g + alpha P lambda           (pull over the CSR: the
//             same row-sum engine over the reversed edges)
//   dL/dw_uv = alpha r_u (lambda_v - t_u) / W_u,   t_u = sum_x P_ux lambda_x
//   dL/dp    = (1-alpha) lambda                     for L = sum_v g_v r_v.
// Both solves are Jacobi sweeps with deterministic compensated FP32 row sums
// and FP64 residual norms, each solve one launch; the gradient is implicit at the
// fixed point, so memory is O(V + E) with no tape.
//
// The row sums run on relabelled, row-sorted copies of the CSC (forward) and the
// CSR (adjoint, W, t), a whole solve in one launch (olv_rowsolve.cuh); their
// vectors are in each copy's numbering (hub values together, rows read and
// written as runs) and the edge weights are permuted into each copy's entry
// order at the start of every forward solve.  RMAT-20, 100 sweeps and their
// adjoint: 20.2 -> 12.7 ms (before: rows reordered but ids and vectors in the
// caller's numbering, L1 hits 21%, rows updated by scattered accesses).
#include "olv_internal.cuh"
#include "olv_rowsolve.cuh"

struct olv_wpr_ctx {
    olv_graph *g = nullptr;
    double alpha = 0.85;
    float a_hi = 0, a_lo = 0;
    olv::DevBuf W, r, coef, lam, t, gbuf;      // [V], the caller's ids
    olv::DevBuf fW, fr, ftp, fs2;              // forward (tcsc ids); fs2: ping-pong
    olv::DevBuf aW, ag, alam2;                 // adjoint (tcsr ids); alam2: ping-pong
};

namespace olv {

struct WprPlans {
    SolvePlan tcsc, tcsr;      // row-sorted CSC and CSR
    DevBuf wc, wr;             // weights in tcsc / tcsr entry order
    DevBuf erow;               // gradient: row of every kGradEdges-th CSR entry
    ~WprPlans() {
        tcsc.release();
        tcsr.release();
        wc.release();
        wr.release();
        erow.release();
    }
};

// --- row-sum ops (row ids are the plan's) ----------------------------------
struct WsumOp {   // W_u = sum of out-weights (CSR), to the caller's ids
    static constexpr bool kGather = false, kWeighted = true, kStore = false;
    const uint32_t *perm;
    float *W;
    __device__ __forceinline__ double first_aux() const { return 0; }
    __device__ __forceinline__ void begin(uint32_t, double) {}
    __device__ __forceinline__ const float *in() const { return nullptr; }
    __device__ __forceinline__ float *out() const { return nullptr; }
    struct Row {
        uint32_t v;
    };
    __device__ __forceinline__ Row row(uint32_t r) const { return Row{__ldg(&perm[r])}; }
    __device__ __forceinline__ float finish(uint32_t, float s, float c, const Row &q, double &,
                                            double &) const {
        W[q.v] = s + c;
        return 0.0f;
    }
};

struct WfwdOp {   // r'[v] = (1-alpha) p[v] + alpha sum_{u->v} w_uv r[u]/W_u
    static constexpr bool kGather = true, kWeighted = true, kStore = true;
    float *s0, *s1;       // r/W ping-pong
    const float *W, *tp;  // tp = (1-alpha) p
    float *r;
    float a_hi, a_lo;
    uint32_t odd;
    __device__ __forceinline__ double first_aux() const { return 0; }
    __device__ __forceinline__ void begin(uint32_t it, double) { odd = it & 1; }
    __device__ __forceinline__ const float *in() const { return odd ? s1 : s0; }
    __device__ __forceinline__ float *out() const { return odd ? s0 : s1; }
    struct Row {
        float tp, r, W;
    };
    __device__ __forceinline__ Row row(uint32_t v) const {
        return Row{__ldg(&tp[v]), r[v], __ldg(&W[v])};
    }
    __device__ __forceinline__ float finish(uint32_t v, float s, float c, const Row &q, double &res,
                                            double &) const {
        const float t = fmaf(a_lo, s, fmaf(a_hi, c, q.tp));
        const float nr = fmaf(a_hi, s, t);
        res += fabs((double)nr - (double)q.r);
        r[v] = nr;
        return q.W > 0.0f ? __fdiv_rn(nr, q.W) : 0.0f;
    }
};

struct WadjOp {   // lambda'[u] = g[u] + alpha sum_{u->v} w_uv lambda[v] / W_u
    static constexpr bool kGather = true, kWeighted = true, kStore = true;
    float *l0, *l1;        // lambda ping-pong
    const float *W, *gv;
    float a_hi, a_lo;
    uint32_t odd;
    __device__ __forceinline__ double first_aux() const { return 0; }
    __device__ __forceinline__ void begin(uint32_t it, double) { odd = it & 1; }
    __device__ __forceinline__ const float *in() const { return odd ? l1 : l0; }
    __device__ __forceinline__ float *out() const { return odd ? l0 : l1; }
    struct Row {
        float W, g, lam;
    };
    __device__ __forceinline__ Row row(uint32_t u) const {
        return Row{__ldg(&W[u]), __ldg(&gv[u]), __ldcg(&in()[u])};
    }
    __device__ __forceinline__ float finish(uint32_t, float s, float c, const Row &q, double &res,
                                            double &) const {
        const float tu = q.W > 0.0f ? __fdiv_rn(s + c, q.W) : 0.0f;
        const float nl = fmaf(a_hi, tu, fmaf(a_lo, tu, q.g));
        res += fabs((double)nl - (double)q.lam);
        return nl;
    }
};

// One pass over the final lambda: t_u, lambda, dL/dp = (1-alpha) lambda and the
// gradient's row factor alpha r_u / W_u, all in the caller's ids.
struct WtOp {
    static constexpr bool kGather = true, kWeighted = true, kStore = false;
    const float *l0, *l1;
    const uint32_t *sweeps;   // adjoint sweeps run: which buffer holds lambda
    const uint32_t *perm;
    const float *W, *r;       // W in row ids, r in the caller's
    float *t, *lam, *coef, *dp;
    float alpha, one_minus_alpha;
    const float *l;
    __device__ __forceinline__ double first_aux() const { return 0; }
    __device__ __forceinline__ void begin(uint32_t, double) { l = (*sweeps & 1) ? l1 : l0; }
    __device__ __forceinline__ const float *in() const { return l; }
    __device__ __forceinline__ float *out() const { return nullptr; }
    struct Row {
        float W, lam, r;
        uint32_t v;
    };
    __device__ __forceinline__ Row row(uint32_t u) const {
        const uint32_t v = __ldg(&perm[u]);
        return Row{__ldg(&W[u]), __ldg(&l[u]), __ldg(&r[v]), v};
    }
    __device__ __forceinline__ float finish(uint32_t, float s, float c, const Row &q, double &,
                                            double &) const {
        t[q.v] = q.W > 0.0f ? __fdiv_rn(s + c, q.W) : 0.0f;
        lam[q.v] = q.lam;
        coef[q.v] = q.W > 0.0f ? __fdiv_rn(alpha * q.r, q.W) : 0.0f;
        if (dp) dp[q.v] = one_minus_alpha * q.lam;
        return 0.0f;
    }
};

// Row of CSR entry e: the last one that begins at or before e.
__device__ __forceinline__ uint32_t row_of(const uint32_t *__restrict__ ptr, uint32_t V,
                                           uint64_t e) {
    uint32_t lo = 0, hi = V;   // ptr[lo] <= e < ptr[hi]
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (__ldg(&ptr[mid]) <= e)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

constexpr uint32_t kGradEdges = 256;   // entries a warp takes at a time

__global__ void k_grad_rows(const uint32_t *__restrict__ ptr, uint32_t V, uint64_t E,
                            uint32_t *__restrict__ erow) {
    const uint64_t n = (E + kGradEdges - 1) / kGradEdges;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        erow[i] = row_of(ptr, V, i * kGradEdges);
}

// dL/dw_e = coef[u] (lambda[col e] - t[u]), u the row of entry e.  A warp takes
// kGradEdges entries from a known first row; a lane's rows only go up, so each
// entry's row is found by stepping on from the last one's, or by a search in the
// rows left when they are many.
__global__ void __launch_bounds__(kBlock)
k_wpr_grad(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ col, uint32_t V,
           uint64_t E, const uint32_t *__restrict__ erow, const float *__restrict__ coef,
           const float *__restrict__ lam, const float *__restrict__ t, float *__restrict__ dw) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t n = (E + kGradEdges - 1) / kGradEdges;
    const uint64_t warp = (blockIdx.x * (uint64_t)kBlock + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * kBlock) >> 5;
    for (uint64_t i = warp; i < n; i += nwarps) {
        const uint32_t r0 = __ldg(&erow[i]), r1 = i + 1 < n ? __ldg(&erow[i + 1]) : V - 1;
        constexpr int kSteps = kGradEdges / 32;
        uint32_t c[kSteps], u[kSteps];
        float l[kSteps];
#pragma unroll
        for (int q = 0; q < kSteps; q++) {
            const uint64_t e = i * kGradEdges + q * 32 + lane;
            c[q] = e < E ? __ldg(&col[e]) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kSteps; q++) l[q] = __ldg(&lam[c[q]]);
        uint32_t lo = r0;
#pragma unroll
        for (int q = 0; q < kSteps; q++) {
            const uint64_t e = i * kGradEdges + q * 32 + lane;
            uint32_t hi = r1 + 1;
            while (hi - lo > 1) {   // the row lies in [lo, hi)
                const uint32_t mid = lo + (hi - lo) / 2;
                if (__ldg(&ptr[mid]) <= e)
                    lo = mid;
                else
                    hi = mid;
            }
            u[q] = lo;
        }
#pragma unroll
        for (int q = 0; q < kSteps; q++) {
            const uint64_t e = i * kGradEdges + q * 32 + lane;
            if (e < E) dw[e] = __ldg(&coef[u[q]]) * (l[q] - __ldg(&t[u[q]]));
        }
    }
}

// Weights in a plan's entry order; places without an entry weigh nothing.
__global__ void k_permute_entries(const float *__restrict__ in, const uint32_t *__restrict__ pos,
                                  uint64_t n, float *__restrict__ out) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t p = pos[k];
        out[k] = p != 0xffffffffu ? in[p] : 0.0f;
    }
}

// Start of a forward solve, in the plan's ids.
__global__ void k_wpr_init(uint32_t V, const float *__restrict__ p, const float *__restrict__ W,
                           const uint32_t *__restrict__ perm, float alpha, float *tp, float *r,
                           float *s0, float *Wp) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = perm[i];
        const float pv = p[v], wv = W[v];
        tp[i] = (1.0f - alpha) * pv;
        r[i] = pv;
        Wp[i] = wv;
        s0[i] = wv > 0.0f ? __fdiv_rn(pv, wv) : 0.0f;
    }
}

// Start of an adjoint solve, in the plan's ids.
__global__ void k_wadj_init(uint32_t V, const float *__restrict__ g, const float *__restrict__ W,
                            const uint32_t *__restrict__ perm, float *gp, float *l0, float *Wp) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < V;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = perm[i];
        gp[i] = g[v];
        l0[i] = g[v];
        Wp[i] = W[v];
    }
}

// out[v] = in[newid[v]]
__global__ void k_to_ids(const float *__restrict__ in, const uint32_t *__restrict__ newid,
                         uint32_t V, float *__restrict__ out) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
         v += (uint64_t)gridDim.x * blockDim.x)
        out[v] = in[newid[v]];
}

static WprPlans *wpr_plans(olv_graph *g) { return static_cast<WprPlans *>(g->wpr_state); }

static int ensure_wpr_plans(olv_graph *g) {
    if (g->wpr_state) return OLV_OK;
    WprPlans *p = new WprPlans();
    cudaStream_t s = g->stream;
    int r = build_solve_plan(g->colptr.as<uint32_t>(), g->rowidx.as<uint32_t>(),
                             g->csc_eid.as<uint32_t>(), g->V, g->E, g->tune.pr_tile_u, true,
                             g->num_sms, s, p->tcsc);
    if (r == OLV_OK)
        r = build_solve_plan(g->rowptr.as<uint32_t>(), g->col.as<uint32_t>(), nullptr, g->V, g->E,
                             g->tune.pr_tile_u, true, g->num_sms, s, p->tcsr);
    if (r == OLV_OK) r = p->wc.ensure(p->tcsc.entries * 4 + 16);
    if (r == OLV_OK) r = p->wr.ensure(p->tcsr.entries * 4 + 16);
    if (r == OLV_OK) r = p->erow.ensure((g->E / kGradEdges + 1) * 4);
    if (r != OLV_OK) {
        delete p;
        return r;
    }
    choose_form<WfwdOp>(p->tcsc);
    choose_form<WsumOp, WadjOp, WtOp>(p->tcsr);
    k_grad_rows<<<g->num_sms * 8, kBlock, 0, s>>>(g->rowptr.as<uint32_t>(), g->V, g->E,
                                                 p->erow.as<uint32_t>());
    g->wpr_state = p;
    return OLV_OK;
}

void release_wpr_state(olv_graph *g) {
    delete wpr_plans(g);
    g->wpr_state = nullptr;
}

static void split_alpha(double alpha, float &hi, float &lo) {
    hi = (float)alpha;
    lo = (float)(alpha - (double)hi);
}

static int copy_vec_in(DevBuf &dst, const float *src, size_t n, cudaStream_t s) {
    OLV_TRY(dst.ensure(n * 4 + 16));
    OLV_CUDA(cudaMemcpyAsync(dst.p, src, n * 4, cudaMemcpyDefault, s));
    return OLV_OK;
}

}  // namespace olv

using namespace olv;

extern "C" int olv_wpr_forward(olv_graph *g, const float *w, const float *p, double alpha,
                               int max_it, double tol, float *r_out, olv_wpr_ctx **ctx_out,
                               olv_stats *st) {
    OLV_CHECK_ARG(g && p && ctx_out, "olv_wpr_forward: null pointer");
    BufferScope scope(g->stream);
    OLV_CHECK_ARG(alpha >= 0 && alpha < 1 && max_it >= 0, "olv_wpr_forward: bad alpha / max_it");
    if (w) OLV_TRY(olv_graph_set_weights_f32(g, w));
    OLV_CHECK_ARG(g->weight_type == OLV_W_F32, "olv_wpr_forward: graph has no FP32 weights");
    OLV_TRY(ensure_wpr_plans(g));
    WprPlans &pl = *wpr_plans(g);
    olv_wpr_ctx *c = *ctx_out;
    if (!c) {
        c = new (std::nothrow) olv_wpr_ctx();
        if (!c) {
            set_error("olv_wpr_forward: host allocation failed");
            return OLV_ERR_NOMEM;
        }
        *ctx_out = c;
    }
    OLV_CHECK_ARG(c->g == nullptr || c->g == g, "olv_wpr_forward: context belongs to another graph");
    c->g = g;
    c->alpha = alpha;
    split_alpha(alpha, c->a_hi, c->a_lo);
    const size_t V = g->V;
    cudaStream_t s = g->stream;
    const size_t Va = (V + 3) & ~(size_t)3;   // ping-pong halves 16-byte aligned
    for (DevBuf *b : {&c->W, &c->r, &c->fW, &c->fr, &c->ftp}) OLV_TRY(b->ensure(V * 4 + 16));
    OLV_TRY(c->fs2.ensure(Va * 8 + 32));
    OLV_TRY(copy_vec_in(c->gbuf, p, V, s));   // p staged in gbuf during the forward
    SolveCtl *fctl = pl.tcsc.ctl.as<SolveCtl>(), *rctl = pl.tcsr.ctl.as<SolveCtl>();
    OLV_CUDA(cudaEventRecord(g->ev0, s));
    OLV_CUDA(cudaMemsetAsync(fctl, 0, sizeof(SolveCtl), s));
    OLV_CUDA(cudaMemsetAsync(rctl, 0, sizeof(SolveCtl), s));
    // the weights in the entry orders of the two copies
    k_permute_entries<<<g->num_sms * 8, kBlock, 0, s>>>(g->w.as<float>(),
                                                       pl.tcsc.pos.as<uint32_t>(), pl.tcsc.entries,
                                                       pl.wc.as<float>());
    k_permute_entries<<<g->num_sms * 8, kBlock, 0, s>>>(g->w.as<float>(),
                                                       pl.tcsr.pos.as<uint32_t>(), pl.tcsr.entries,
                                                       pl.wr.as<float>());
    // W = row sums of the weights (one pass, same deterministic engine)
    OLV_TRY(launch_solve(pl.tcsr, pl.tcsr.args(1, 0.0, &pl.wr),
                         WsumOp{pl.tcsr.perm.as<uint32_t>(), c->W.as<float>()}, s));
    k_wpr_init<<<g->num_sms * 8, kBlock, 0, s>>>(
        g->V, c->gbuf.as<float>(), c->W.as<float>(), pl.tcsc.perm.as<uint32_t>(), (float)alpha,
        c->ftp.as<float>(), c->fr.as<float>(), c->fs2.as<float>(), c->fW.as<float>());
    OLV_CUDA(cudaGetLastError());
    WfwdOp op = {};
    op.s0 = c->fs2.as<float>();
    op.s1 = op.s0 + Va;
    op.W = c->fW.as<float>();
    op.tp = c->ftp.as<float>();
    op.r = c->fr.as<float>();
    op.a_hi = c->a_hi;
    op.a_lo = c->a_lo;
    OLV_TRY(launch_solve(pl.tcsc, pl.tcsc.args((uint32_t)max_it, tol, &pl.wc), op, s));
    k_to_ids<<<g->num_sms * 8, kBlock, 0, s>>>(c->fr.as<float>(), pl.tcsc.newid.as<uint32_t>(),
                                              g->V, c->r.as<float>());
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaEventRecord(g->ev1, s));
    SolveCtl hc, hr;
    OLV_CUDA(cudaMemcpyAsync(&hc, fctl, sizeof hc, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaMemcpyAsync(&hr, rctl, sizeof hr, cudaMemcpyDeviceToHost, s));
    if (r_out) OLV_CUDA(cudaMemcpyAsync(r_out, c->r.p, V * 4, cudaMemcpyDefault, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    const int solved = solve_error(hc, pl.tcsc, s, "olv_wpr_forward");
    OLV_TRY(solve_error(hr, pl.tcsr, s, "olv_wpr_forward"));
    OLV_TRY(solved);
    g->launches = 6;   // two weight copies, their sums, init, one solve, map back
    if (st) {
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        st->iterations = hc.iter;
        st->pull_steps = 0;
        st->vertices_reached = V;
        st->edges_traversed = g->E * (uint64_t)hc.iter;
        st->edges_relaxed = st->edges_traversed;
        st->residual = hc.residual;
        st->device_ms = ms;
    }
    return OLV_OK;
}

extern "C" int olv_wpr_backward(olv_wpr_ctx *c, const float *gvec, int max_it, double tol,
                                float *dw_out, float *dp_out, olv_stats *st) {
    OLV_CHECK_ARG(c && c->g && gvec && dw_out, "olv_wpr_backward: null pointer or no forward");
    OLV_CHECK_ARG(max_it >= 0, "olv_wpr_backward: bad max_it");
    olv_graph *g = c->g;
    BufferScope scope(g->stream);
    if (!wpr_plans(g)) {   // the row plans were dropped (pr_tile_u changed) since the forward
        set_error("olv_wpr_backward: the graph's row plans changed since olv_wpr_forward; "
                  "run the forward again");
        return OLV_ERR_STATE;
    }
    WprPlans &pl = *wpr_plans(g);
    const size_t V = g->V;
    const uint64_t E = g->E;
    cudaStream_t s = g->stream;
    const size_t Va = (V + 3) & ~(size_t)3;
    for (DevBuf *b : {&c->coef, &c->lam, &c->t, &c->aW, &c->ag}) OLV_TRY(b->ensure(V * 4 + 16));
    OLV_TRY(c->alam2.ensure(Va * 8 + 32));
    OLV_TRY(copy_vec_in(c->gbuf, gvec, V, s));
    const bool dev_dw = is_device_ptr(dw_out);
    const bool dev_dp = dp_out && is_device_ptr(dp_out);
    DevBuf dwbuf, dpbuf;
    if (!dev_dw) OLV_TRY(dwbuf.ensure(E * 4 + 16));
    if (dp_out && !dev_dp) OLV_TRY(dpbuf.ensure(V * 4 + 16));
    float *dw = dev_dw ? dw_out : dwbuf.as<float>();
    float *dp = dp_out ? (dev_dp ? dp_out : dpbuf.as<float>()) : nullptr;
    SolveCtl *ctl = pl.tcsr.ctl.as<SolveCtl>();
    OLV_CUDA(cudaEventRecord(g->ev0, s));
    OLV_CUDA(cudaMemsetAsync(ctl, 0, sizeof(SolveCtl), s));
    k_wadj_init<<<g->num_sms * 8, kBlock, 0, s>>>(
        g->V, c->gbuf.as<float>(), c->W.as<float>(), pl.tcsr.perm.as<uint32_t>(),
        c->ag.as<float>(), c->alam2.as<float>(), c->aW.as<float>());
    OLV_CUDA(cudaGetLastError());
    WadjOp op = {};
    op.l0 = c->alam2.as<float>();
    op.l1 = op.l0 + Va;
    op.W = c->aW.as<float>();
    op.gv = c->ag.as<float>();
    op.a_hi = c->a_hi;
    op.a_lo = c->a_lo;
    OLV_TRY(launch_solve(pl.tcsr, pl.tcsr.args((uint32_t)max_it, tol, &pl.wr), op, s));
    SolveCtl hc, ht;
    OLV_CUDA(cudaMemcpyAsync(&hc, ctl, sizeof hc, cudaMemcpyDeviceToHost, s));
    // the last pass counts its own barrier and iteration in tcsc's block
    SolveCtl *tctl = pl.tcsc.ctl.as<SolveCtl>();
    OLV_CUDA(cudaMemsetAsync(tctl, 0, sizeof(SolveCtl), s));
    WtOp top = {};
    top.l0 = op.l0;
    top.l1 = op.l1;
    top.sweeps = &ctl->iter;
    top.perm = pl.tcsr.perm.as<uint32_t>();
    top.W = c->aW.as<float>();
    top.r = c->r.as<float>();
    top.t = c->t.as<float>();
    top.lam = c->lam.as<float>();
    top.coef = c->coef.as<float>();
    top.dp = dp;
    top.alpha = (float)c->alpha;
    top.one_minus_alpha = (float)(1.0 - c->alpha);
    SolveArgs ta = pl.tcsr.args(1, 0.0, &pl.wr);
    ta.ctl = tctl;
    OLV_TRY(launch_solve(pl.tcsr, ta, top, s));
    OLV_CUDA(cudaMemcpyAsync(&ht, tctl, sizeof ht, cudaMemcpyDeviceToHost, s));
    if (E)
        k_wpr_grad<<<g->num_sms * 8, kBlock, 0, s>>>(
            g->rowptr.as<uint32_t>(), g->col.as<uint32_t>(), g->V, E, pl.erow.as<uint32_t>(),
            c->coef.as<float>(), c->lam.as<float>(), c->t.as<float>(), dw);
    OLV_CUDA(cudaGetLastError());
    OLV_CUDA(cudaEventRecord(g->ev1, s));
    if (!dev_dw) OLV_CUDA(cudaMemcpyAsync(dw_out, dw, E * 4, cudaMemcpyDeviceToHost, s));
    if (dp_out && !dev_dp) OLV_CUDA(cudaMemcpyAsync(dp_out, dp, V * 4, cudaMemcpyDeviceToHost, s));
    OLV_CUDA(cudaStreamSynchronize(s));
    OLV_TRY(solve_error(hc, pl.tcsr, s, "olv_wpr_backward"));
    OLV_TRY(solve_error(ht, pl.tcsr, s, "olv_wpr_backward"));
    g->launches = 3 + (E ? 1 : 0);   // init, one solve, the last sums, the edges' gradient
    if (st) {
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        st->iterations = hc.iter;
        st->pull_steps = 0;
        st->vertices_reached = V;
        st->edges_traversed = E * (uint64_t)(hc.iter + 2);
        st->edges_relaxed = st->edges_traversed;
        st->residual = hc.residual;
        st->device_ms = ms;
    }
    return OLV_OK;
}

extern "C" int olv_wpr_ctx_destroy(olv_wpr_ctx *c) {
    if (!c) return OLV_OK;
    delete c;
    return OLV_OK;
}
