// Device buffers of the engine and the blocks kept for the next ones.
//
// A call on a new graph allocates some fifty buffers, half of them for the
// length of one step (sort keys, renumbering, plans).  The driver takes up to
// a millisecond to map or unmap a large one: a graph created from host arrays,
// one SSSP and its destruction (RMAT, 1 M vertices, 16 M edges) took 40 ms, 23
// of them there, and take 17 ms with the blocks kept (12 are the host-to-device
// copy).  A buffer takes the smallest kept block that fits without wasting a
// quarter of itself.
//
// Bounds and safety:
//   - at most 1/64 of a device's memory is kept in a context; past that the
//     blocks kept longest go back to the driver first (cudaFree, which may wait
//     for the device), and a block larger than the bound goes back at once;
//   - when the driver has no room for a new buffer, every kept block of the
//     context goes back and the allocation is tried again, so that keeping
//     blocks never makes one of the engine's allocations fail; other users of the
//     device get them with olv_release_memory();
//   - a block is kept only by a call on a handle (BufferScope), after the
//     handle's stream, the only one that uses the handle's buffers, has been
//     waited for, so its next owner may use it on any stream and from any
//     thread.  Keeping a block and handing it out again wait for no other
//     stream.  What is given up elsewhere is freed.  The lists are guarded by one
//     mutex;
//   - a block belongs to the context it was allocated in and is handed out there
//     only: a context's id is never used again, so that blocks which died with
//     their context (cudaDeviceReset, cuCtxDestroy) stay where they are.
#include <list>
#include <mutex>
#include <unordered_map>

#include "olv_driver.h"
#include "olv_internal.cuh"

namespace olv {

namespace {

constexpr size_t kSmallUnit = 512, kLargeUnit = 2u << 20;   // block sizes are multiples of these

struct Block {
    void *p;
    size_t bytes;
    uint64_t ctx;
};

struct PerContext {
    size_t bytes = 0, bound = 0;
};

struct Kept {
    std::mutex m;
    std::list<Block> blocks;   // kept longest first
    std::unordered_map<uint64_t, PerContext> by_ctx;
};

Kept &kept() {
    static Kept *k = new Kept;   // outlives every buffer, also those of static objects
    return *k;
}

// Id of the calling thread's context, 0 if it cannot be told (nothing is kept then).
uint64_t current_context() {
    static const auto get = driver_entry<PFN_cuCtxGetCurrent_v4000>("cuCtxGetCurrent", 4000);
    static const auto id_of = driver_entry<PFN_cuCtxGetId_v12000>("cuCtxGetId", 12000);
    if (!get || !id_of) return 0;
    CUcontext c = nullptr;
    if (get(&c) != CUDA_SUCCESS || !c) {
        // this thread's first call: the runtime has not made a context current yet
        if (cudaFree(nullptr) != cudaSuccess || get(&c) != CUDA_SUCCESS || !c) {
            cudaGetLastError();
            return 0;
        }
    }
    unsigned long long id = 0;
    return id_of(c, &id) == CUDA_SUCCESS ? id : 0;
}

size_t keep_bound() {
    size_t free_b = 0, total = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return total / 64;
}

// Blocks of the current context ctx, kept longest first, go back to the driver
// until at most `most` bytes are kept there.
void give_back(Kept &k, uint64_t ctx, size_t most) {
    const auto c = k.by_ctx.find(ctx);
    if (c == k.by_ctx.end()) return;
    for (auto it = k.blocks.begin(); it != k.blocks.end() && c->second.bytes > most;) {
        if (it->ctx != ctx) {
            ++it;
            continue;
        }
        cudaFree(it->p);
        c->second.bytes -= it->bytes;
        it = k.blocks.erase(it);
    }
}

cudaError_t take(Block *out, size_t n) {
    const size_t unit = n < kLargeUnit / 2 ? kSmallUnit : kLargeUnit;
    const size_t need = (n + unit - 1) / unit * unit;
    const uint64_t ctx = current_context();
    Kept &k = kept();
    std::lock_guard<std::mutex> lock(k.m);
    auto best = k.blocks.end();
    for (auto it = k.blocks.begin(); it != k.blocks.end(); ++it)
        if (it->ctx == ctx && it->bytes >= need && it->bytes - need <= it->bytes / 4 &&
            (best == k.blocks.end() || it->bytes < best->bytes))
            best = it;
    Block b{nullptr, need, ctx};
    if (best != k.blocks.end()) {
        b = *best;
        k.by_ctx.find(ctx)->second.bytes -= b.bytes;
        k.blocks.erase(best);
    } else {
        cudaError_t e = cudaMalloc(&b.p, need);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            give_back(k, ctx, 0);
            e = cudaMalloc(&b.p, need);
        }
        if (e != cudaSuccess) return e;
    }
    *out = b;
    return cudaSuccess;
}

// The scope this thread is in.
thread_local cudaStream_t t_stream = nullptr;
thread_local bool t_keep = false;

void put(const Block &b) {
    bool keep = t_keep && b.ctx && current_context() == b.ctx &&
                cudaStreamSynchronize(t_stream) == cudaSuccess;
    if (keep) {
        keep = false;
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.m);
        try {
            PerContext &c = k.by_ctx[b.ctx];
            if (c.bound == 0) c.bound = keep_bound();
            if (b.bytes <= c.bound) {
                give_back(k, b.ctx, c.bound - b.bytes);
                k.blocks.push_back(b);
                c.bytes += b.bytes;
                keep = true;
            }
        } catch (...) {   // no host memory for the list: not kept
        }
    }
    if (!keep) cudaFree(b.p);
}

}  // namespace

BufferScope::BufferScope(cudaStream_t s)
    : before(t_stream), kept_before(t_keep), errors_before(error_count()) {
    t_stream = s;
    t_keep = true;
}

void BufferScope::end() {
    if (ended) return;
    ended = true;
    if (error_count() != errors_before && cudaStreamSynchronize(t_stream) != cudaSuccess)
        cudaGetLastError();
    t_stream = before;
    t_keep = kept_before;
}

int DevBuf::ensure(size_t n) {
    if (n <= bytes && p) return OLV_OK;
    release();
    if (n == 0) n = 16;
    Block b;
    const cudaError_t e = take(&b, n);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc", __FILE__, __LINE__);
    p = b.p;
    bytes = b.bytes;
    ctx = b.ctx;
    return OLV_OK;
}

void DevBuf::release() {
    if (p) put(Block{p, bytes, ctx});
    p = nullptr;
    bytes = 0;
}

}  // namespace olv

using namespace olv;

extern "C" int olv_release_memory(uint64_t *bytes_out) {
    const uint64_t ctx = current_context();
    Kept &k = kept();
    std::lock_guard<std::mutex> lock(k.m);
    const auto c = k.by_ctx.find(ctx);
    if (bytes_out) *bytes_out = c == k.by_ctx.end() ? 0 : c->second.bytes;
    give_back(k, ctx, 0);
    return OLV_OK;
}
