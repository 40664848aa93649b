// Autotuner (no reference counterpart; the reference fixed its launch shape
// in util::kernelConfig, utils.h:56-72, and took the edge-group size from the
// -g flag, BFS.cu:89).  Coordinate descent over the engine's tunables -- BFS
// hub split and push/pull switch points, SSSP bucket width, hub split and
// light sub-buckets, the PageRank / weighted-PageRank row grouping (entries
// per lane, which sets the lanes per row of the tile plans), the msBFS
// push/pull switch -- each candidate timed with CUDA events on the graph's
// own stream (BFS/SSSP from the highest out-degree vertex, msBFS from 16
// sources spread over the graph, PageRank 10 iterations); the winners are
// applied to the handle and, optionally,
// written to a JSON table keyed by GPU and graph shape, which olv_autotune_load
// re-applies when the key matches.  Tuning changes speed only: every result
// stays bit-exact (tests check it).
#include <stdio.h>
#include <string.h>

#include <string>
#include <vector>

#include "olv_internal.cuh"

namespace olv {

static int time_call(olv_graph *g, int (*fn)(olv_graph *, uint32_t, void *), uint32_t src,
                     void *out, int reps, double *ms_out) {
    OLV_TRY(fn(g, src, out));   // warm-up (also builds cached graphs)
    double best = 1e30;
    for (int r = 0; r < reps; r++) {
        olv_stats st;
        (void)st;
        OLV_TRY(fn(g, src, out));
        float ms = 0;
        OLV_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        best = ms < best ? ms : best;
    }
    *ms_out = best;
    return OLV_OK;
}

static int run_bfs(olv_graph *g, uint32_t src, void *out) {
    return olv_bfs(g, src, static_cast<int32_t *>(out), nullptr);
}
static int run_sssp(olv_graph *g, uint32_t src, void *out) {
    return olv_sssp(g, src, static_cast<uint32_t *>(out), nullptr);
}
static int run_pagerank(olv_graph *g, uint32_t, void *out) {
    return olv_pagerank(g, 0.85, 10, 0.0, OLV_DANGLING_UNIFORM, static_cast<float *>(out), nullptr);
}
// msBFS from kMsTuneSources sources spread over the vertices with out-edges
constexpr int kMsTuneSources = 16;
struct MsTune {
    std::vector<uint32_t> sources;
    DevBuf out;
};
static int run_msbfs(olv_graph *g, uint32_t, void *arg) {
    MsTune *m = static_cast<MsTune *>(arg);
    return olv_msbfs(g, m->sources.data(), (int)m->sources.size(), m->out.as<int32_t>(),
                     nullptr);
}

static std::string tune_key(olv_graph *g) {
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, g->device);
    char buf[512];
    snprintf(buf, sizeof buf, "%s|V=%u|E=%llu|maxout=%u|maxin=%u|w=%d", prop.name, g->V,
             (unsigned long long)g->E, g->max_out_degree, g->max_in_degree, g->weight_type);
    return buf;
}

}  // namespace olv

using namespace olv;

extern "C" int olv_autotune(olv_graph *g, const char *json_path, int reps) {
    OLV_CHECK_ARG(g, "olv_autotune: null graph");
    if (reps < 1) reps = 3;
    uint32_t src = 0, deg = 0;
    OLV_TRY(olv_graph_max_degree_vertex(g, &src, &deg));
    DevBuf out;
    OLV_TRY(out.ensure((size_t)g->V * 4 + 16));
    struct Cand {
        const char *key;
        std::vector<double> values;
        int (*fn)(olv_graph *, uint32_t, void *);
        void *arg;   // output buffer (or the msBFS set-up)
    };
    std::vector<Cand> plan = {
        {"hub_degree", {256, 1024, 4096}, run_bfs, out.p},
        {"alpha", {2, 6, 14, 30, 60}, run_bfs, out.p},
        {"beta", {6, 24, 100}, run_bfs, out.p},
    };
    if (g->weight_type == OLV_W_U32) {
        plan.push_back({"sssp_delta", {8, 16, 24, 32, 64, 128, 256}, run_sssp, out.p});
        plan.push_back({"sssp_tail_delta", {0, 256, 1024, 4096}, run_sssp, out.p});
        plan.push_back({"sssp_hub_degree", {128, 256, 1024}, run_sssp, out.p});
        plan.push_back({"sssp_piece", {256, 1024}, run_sssp, out.p});
        plan.push_back({"sssp_sub", {0, 8, 16}, run_sssp, out.p});
    }
    // PageRank / weighted PageRank row grouping (entries per lane per round), where the
    // plan follows it
    std::vector<double> lanes = {4, 8, 16};
    if (!pr_tile_u_matters(g)) lanes = {(double)g->tune.pr_tile_u};
    plan.push_back({"pr_tile_u", lanes, run_pagerank, out.p});
    // multi-source BFS push -> pull switch point
    std::vector<uint32_t> rp((size_t)g->V + 1);
    OLV_TRY(olv_graph_copy_csr(g, rp.data(), nullptr, nullptr));
    MsTune mst;
    for (uint32_t v = 0, seen = 0; v < g->V && (int)mst.sources.size() < kMsTuneSources; v++)
        if (rp[v + 1] > rp[v] && seen++ % (1 + g->V / (8 * kMsTuneSources)) == 0)
            mst.sources.push_back(v);
    if (!mst.sources.empty()) {
        OLV_TRY(mst.out.ensure((size_t)g->V * 4 * mst.sources.size() + 16));
        plan.push_back({"ms_alpha", {5, 10, 20, 40}, run_msbfs, &mst});
    }
    std::string log;
    for (auto &c : plan) {
        double best_ms = 1e30, best_v = 0;
        for (double v : c.values) {
            OLV_TRY(olv_tune_set(g, c.key, v));
            double ms = 0;
            OLV_TRY(time_call(g, c.fn, src, c.arg, reps, &ms));
            if (ms < best_ms) {
                best_ms = ms;
                best_v = v;
            }
        }
        OLV_TRY(olv_tune_set(g, c.key, best_v));
        char line[160];
        snprintf(line, sizeof line, "%s  \"%s\": %.6g", log.empty() ? "" : ",\n", c.key, best_v);
        log += line;
    }
    if (json_path) {
        FILE *f = fopen(json_path, "w");
        if (!f) {
            set_error("olv_autotune: cannot write %s", json_path);
            return OLV_ERR_ARG;
        }
        fprintf(f, "{\n  \"key\": \"%s\",\n%s\n}\n", tune_key(g).c_str(), log.c_str());
        fclose(f);
    }
    return OLV_OK;
}

extern "C" int olv_autotune_load(olv_graph *g, const char *json_path, int *applied) {
    OLV_CHECK_ARG(g && json_path, "olv_autotune_load: null pointer");
    if (applied) *applied = 0;
    FILE *f = fopen(json_path, "r");
    if (!f) {
        set_error("olv_autotune_load: cannot read %s", json_path);
        return OLV_ERR_ARG;
    }
    std::string text;
    char buf[4096];
    size_t n;
    while ((n = fread(buf, 1, sizeof buf, f)) > 0) text.append(buf, n);
    fclose(f);
    const std::string want = "\"key\": \"" + tune_key(g) + "\"";
    if (text.find(want) == std::string::npos) return OLV_OK;   // table is for another graph/GPU
    const char *keys[] = {"hub_degree",      "piece",      "alpha",           "beta",
                          "sssp_delta",      "sssp_piece", "sssp_hub_degree", "sssp_sub",
                          "sssp_tail_delta", "ms_alpha",   "pr_tile_u"};
    for (const char *k : keys) {
        const std::string pat = std::string("\"") + k + "\":";
        size_t pos = text.find(pat);
        if (pos == std::string::npos) continue;
        double v = atof(text.c_str() + pos + pat.size());
        OLV_TRY(olv_tune_set(g, k, v));
    }
    if (applied) *applied = 1;
    return OLV_OK;
}
