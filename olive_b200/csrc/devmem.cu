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
//   - at most 1/64 of a device's memory is kept on it; past that the blocks
//     kept longest go back to the driver first, and a block larger than the
//     bound goes back at once;
//   - when the driver has no room for a new buffer, every kept block of the
//     device goes back and the allocation is tried again, so that keeping
//     blocks never makes one of the engine's allocations fail;
//   - a block is kept only by a call on a handle (BufferScope), after the
//     handle's stream, the only one that uses the handle's buffers, has been
//     waited for, so its next owner may use it on any stream and from any
//     thread; no other stream is waited for or looked at, so captures that
//     other threads have under way are not disturbed.  What is given up
//     elsewhere is freed.  The lists are guarded by one mutex.
#include <list>
#include <mutex>
#include <unordered_map>

#include "olv_internal.cuh"

namespace olv {

namespace {

constexpr size_t kSmallUnit = 512, kLargeUnit = 2u << 20;   // block sizes are multiples of these

struct Block {
    void *p;
    size_t bytes;
    int dev;
};

struct Kept {
    std::mutex m;
    std::list<Block> blocks;                    // kept longest first
    std::unordered_map<int, size_t> bytes;      // kept, by device
    std::unordered_map<int, size_t> bound;
};

Kept &kept() {
    static Kept *k = new Kept;   // outlives every buffer, also those of static objects
    return *k;
}

size_t keep_bound(Kept &k, int dev) {
    auto it = k.bound.find(dev);
    if (it != k.bound.end()) return it->second;
    size_t free_b = 0, total = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return k.bound[dev] = total / 64;
}

// Blocks of device dev, kept longest first, go back to the driver until at
// most `most` bytes are kept there.
void give_back(Kept &k, int dev, size_t most) {
    for (auto it = k.blocks.begin(); it != k.blocks.end() && k.bytes[dev] > most;) {
        if (it->dev != dev) {
            ++it;
            continue;
        }
        cudaFree(it->p);
        k.bytes[dev] -= it->bytes;
        it = k.blocks.erase(it);
    }
}

cudaError_t take(Block *out, size_t n) {
    const size_t unit = n < kLargeUnit / 2 ? kSmallUnit : kLargeUnit;
    const size_t need = (n + unit - 1) / unit * unit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    Kept &k = kept();
    std::lock_guard<std::mutex> lock(k.m);
    auto best = k.blocks.end();
    for (auto it = k.blocks.begin(); it != k.blocks.end(); ++it)
        if (it->dev == dev && it->bytes >= need && it->bytes - need <= it->bytes / 4 &&
            (best == k.blocks.end() || it->bytes < best->bytes))
            best = it;
    Block b{nullptr, need, dev};
    if (best != k.blocks.end()) {
        b = *best;
        k.bytes[dev] -= b.bytes;
        k.blocks.erase(best);
    } else {
        e = cudaMalloc(&b.p, need);
        if (e == cudaErrorMemoryAllocation && k.bytes[dev]) {
            cudaGetLastError();
            give_back(k, dev, 0);
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
    int dev = 0;
    bool keep = t_keep && cudaGetDevice(&dev) == cudaSuccess && dev == b.dev &&
                cudaStreamSynchronize(t_stream) == cudaSuccess;
    if (keep) {
        keep = false;
        Kept &k = kept();
        std::lock_guard<std::mutex> lock(k.m);
        try {
            const size_t bound = keep_bound(k, b.dev);
            if (b.bytes <= bound) {
                give_back(k, b.dev, bound - b.bytes);
                k.blocks.push_back(b);
                k.bytes[b.dev] += b.bytes;
                keep = true;
            }
        } catch (...) {   // no host memory for the list: not kept
        }
    }
    if (!keep) cudaFree(b.p);
}

}  // namespace

BufferScope::BufferScope(cudaStream_t s, bool keep) : before(t_stream), kept_before(t_keep) {
    t_stream = s;
    t_keep = keep;
}

BufferScope::~BufferScope() {
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
    dev = b.dev;
    return OLV_OK;
}

void DevBuf::release() {
    if (p) put(Block{p, bytes, dev});
    p = nullptr;
    bytes = 0;
}

}  // namespace olv
