// Device and pinned blocks of sessions and scratches, kept for the next one.
//
// A request makes and drops a session of a hundred buffers.  cudaMalloc and cudaFree map and unmap memory under a
// driver-wide lock and free waits for the whole device: 45 ms a request on an idle B200, several hundred beside other
// work, against 8 - 25 ms for the prompt itself.  Blocks that are given back are kept by size class (pool.cuh), at most
// kPoolBytes per device, the longest idle ones going first; all of them are given back when a model on the device is
// destroyed and when an allocation of this library fails, the pool's own or another (device_malloc, host_malloc: every
// allocation outside the pool goes through them).  Whoever gives a block back has waited for the work that uses it.
#include <algorithm>

#include "model.cuh"
#include "pool.cuh"

namespace dfl {

namespace {
constexpr size_t kPoolBytes = 8ull << 30, kPoolHostBytes = 256ull << 20;
constexpr size_t kPoolStreams = 64;

struct CudaSource : BlockSource {
    void* get(int place, size_t bytes) override {   // device blocks: on the current device, which is `place`
        void* p = nullptr;
        if ((place == POOL_HOST ? cudaMallocHost(&p, bytes) : cudaMalloc(&p, bytes)) == cudaSuccess) return p;
        cudaGetLastError();
        return nullptr;
    }
    void put(int place, void* p) override {
        if (place == POOL_HOST) { cudaFreeHost(p); return; }
        int cur = 0;
        cudaGetDevice(&cur);
        if (cur != place) cudaSetDevice(place);
        cudaFree(p);
        if (cur != place) cudaSetDevice(cur);
    }
};
struct Pool {
    CudaSource source;
    BlockPool blocks{source, kPoolBytes, kPoolHostBytes};
    std::mutex mu;   // of what follows
    std::map<int, std::vector<cudaStream_t>> streams;
    std::unordered_map<void*, size_t> lent;   // host blocks in callers' hands (dfl_host_alloc)
    size_t lent_bytes = 0;
};
// never destroyed: at process exit the driver may be gone before static destructors run
Pool& pool() { static Pool* p = new Pool(); return *p; }

cudaError_t again_after_trim(cudaError_t e, int place, cudaError_t (*get)(void**, size_t), void** p, size_t bytes) {
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    pool().blocks.trim(place);
    return get(p, bytes);
}
}  // namespace

void* pool_alloc(size_t bytes) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    return pool().blocks.take(device, bytes);
}
void* pool_alloc_host(size_t bytes) { return pool().blocks.take(POOL_HOST, bytes); }
void pool_free(void* p) { pool().blocks.give(p); }
cudaError_t device_malloc_bytes(void** p, size_t bytes) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    return e != cudaSuccess ? e : again_after_trim(cudaMalloc(p, bytes), device, [](void** q, size_t n) { return cudaMalloc(q, n); }, p, bytes);
}
cudaError_t host_malloc_bytes(void** p, size_t bytes) {
    return again_after_trim(cudaMallocHost(p, bytes), POOL_HOST, [](void** q, size_t n) { return cudaMallocHost(q, n); }, p, bytes);
}
// Streams the same way: making and dropping the four of a request costs 0.25 ms.  At most kPoolStreams idle ones a device.
cudaStream_t pool_stream() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        auto& idle = pool().streams[device];
        if (!idle.empty()) {
            cudaStream_t st = idle.back();
            idle.pop_back();
            return st;
        }
    }
    cudaStream_t st = nullptr;
    return cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess ? st : nullptr;
}
void pool_stream_free(cudaStream_t st) {
    if (!st) return;
    int device = 0;
    if (cudaStreamSynchronize(st) == cudaSuccess && cudaGetDevice(&device) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(pool().mu);
        auto& idle = pool().streams[device];
        if (idle.size() < kPoolStreams) {
            idle.push_back(st);
            return;
        }
    }
    cudaStreamDestroy(st);
}
void pool_trim(int device) {
    std::vector<cudaStream_t> streams;
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        streams.swap(pool().streams[device]);
    }
    for (cudaStream_t st : streams) cudaStreamDestroy(st);
    pool().blocks.trim(device);
    pool().blocks.trim(POOL_HOST);
}

}  // namespace dfl

// ---- result buffers ----------------------------------------------------------------------------------------------
// A block's logits are 10 MB: into fresh pageable memory they travel at 6 GB/s (a staging copy and a page fault every 4 KB), into a
// pinned block at the link's 55.  The blocks in use by callers are bounded like the idle ones; beyond that dfl_host_alloc
// gives nothing and the caller falls back to memory of its own.
extern "C" void* dfl_host_alloc(uint64_t n_bytes) {
    using namespace dfl;
    static_assert(kPoolHostBytes >= (64u << 20), "one result must fit");
    if (n_bytes > (64ull << 20)) return nullptr;
    Pool& p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        if (p.lent_bytes + n_bytes > kPoolHostBytes) return nullptr;
        p.lent_bytes += n_bytes;
    }
    void* b = pool_alloc_host(n_bytes);
    std::lock_guard<std::mutex> lock(p.mu);
    if (b) p.lent[b] = n_bytes;
    else p.lent_bytes -= n_bytes;
    return b;
}
extern "C" void dfl_host_free(void* p) {
    using namespace dfl;
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        auto it = pool().lent.find(p);
        if (it == pool().lent.end()) return;
        pool().lent_bytes -= it->second;
        pool().lent.erase(it);
    }
    pool_free(p);
}

// ---- the pool's rules over a source of `capacity` bytes that only counts ----------------------------------------------
extern "C" dfl_status dfl_pool_selftest(uint64_t limit, uint64_t capacity, int32_t host, const int64_t* ops, uint32_t n_ops, int64_t* trace) {
    using namespace dfl;
    if (!ops || !trace) return fail(DFL_ERR_BAD_ARG, "pool_selftest: null argument");
    struct Fake : BlockSource {
        uint64_t capacity = 0, held = 0, gets = 0, last = 0;
        std::unordered_map<void*, size_t> out;
        void* get(int, size_t bytes) override {
            if (held + bytes > capacity) return nullptr;
            held += bytes;
            ++gets;
            void* p = reinterpret_cast<void*>(static_cast<uintptr_t>(++last * 4096));
            out[p] = bytes;
            return p;
        }
        void put(int, void* p) override { held -= out.at(p); out.erase(p); }
    } fake;
    fake.capacity = capacity;
    BlockPool blocks(fake, limit, limit);
    const int place = host ? POOL_HOST : 0;
    std::vector<void*> taken;
    for (uint32_t i = 0; i < n_ops; ++i) {
        int64_t ok = 1;
        if (ops[i] > 0) {
            taken.push_back(blocks.take(place, (size_t)ops[i]));
            ok = taken.back() != nullptr;
        } else if (ops[i] < 0) {
            const uint64_t which = (uint64_t)(-ops[i] - 1);
            if (which >= taken.size()) return fail(DFL_ERR_BAD_ARG, "pool_selftest: no such block");
            blocks.give(taken[which]);
        } else {
            blocks.trim(place);
        }
        trace[3 * i] = ok;
        trace[3 * i + 1] = (int64_t)fake.held;
        trace[3 * i + 2] = (int64_t)fake.gets;
    }
    return DFL_OK;
}
