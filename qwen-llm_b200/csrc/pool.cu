// Device and pinned blocks of sessions and scratches, kept for the next one.
//
// A request makes and drops a session of a hundred buffers.  cudaMalloc and cudaFree map and unmap memory under a
// driver-wide lock and free waits for the whole device: 45 ms a request on an idle B200, several hundred beside other
// work, against 8 - 25 ms for the prompt itself.  Blocks that are given back are kept by size, at most
// kPoolBytes per device (the rest goes to the driver at once), and all of them are given back when a model on the device is
// destroyed or an allocation fails.  Whoever gives a block back has waited for the work that uses it.
#include <map>
#include <mutex>
#include <unordered_map>

#include "model.cuh"

namespace dfl {

namespace {
constexpr size_t kPoolBytes = 8ull << 30, kPoolHostBytes = 256ull << 20;
constexpr size_t kPoolStreams = 64;
constexpr int HOST = -1;   // "device" of pinned host blocks

struct Pool {
    struct Block { int device; size_t bytes; };
    std::mutex mu;
    std::multimap<std::pair<int, size_t>, void*> idle;
    std::map<int, size_t> idle_bytes;
    std::map<int, std::vector<cudaStream_t>> streams;
    std::unordered_map<void*, Block> live;
    std::unordered_map<void*, size_t> lent;   // host blocks in callers' hands (dfl_host_alloc)
    size_t lent_bytes = 0;

    static void release(int device, void* p) {
        if (device == HOST) { cudaFreeHost(p); return; }
        int cur = 0;
        cudaGetDevice(&cur);
        if (cur != device) cudaSetDevice(device);
        cudaFree(p);
        if (cur != device) cudaSetDevice(cur);
    }
    void trim(int device) {
        std::lock_guard<std::mutex> lock(mu);
        for (auto it = idle.begin(); it != idle.end();) {
            if (it->first.first != device) { ++it; continue; }
            release(device, it->second);
            it = idle.erase(it);
        }
        idle_bytes[device] = 0;
        for (cudaStream_t st : streams[device]) cudaStreamDestroy(st);
        streams[device].clear();
    }
    void* take(int device, size_t bytes) {
        bytes = (bytes + 511) / 512 * 512;
        if (bytes == 0) bytes = 512;
        if (device == HOST) {   // results of any row count: eight sizes an octave, so that requests find each other's blocks
            size_t step = 512;
            while (step * 16 <= bytes) step *= 2;
            bytes = (bytes + step - 1) / step * step;
        }
        {
            std::lock_guard<std::mutex> lock(mu);
            auto it = idle.find({device, bytes});
            if (it != idle.end()) {
                void* p = it->second;
                idle.erase(it);
                idle_bytes[device] -= bytes;
                live[p] = {device, bytes};
                return p;
            }
        }
        void* p = nullptr;
        auto get = [&] { return device == HOST ? cudaMallocHost(&p, bytes) : cudaMalloc(&p, bytes); };
        if (get() != cudaSuccess) {
            cudaGetLastError();
            trim(device);
            if (get() != cudaSuccess) return nullptr;
        }
        std::lock_guard<std::mutex> lock(mu);
        live[p] = {device, bytes};
        return p;
    }
    void give(void* p) {
        if (!p) return;
        Block b;
        {
            std::lock_guard<std::mutex> lock(mu);
            auto it = live.find(p);
            if (it == live.end()) return;
            b = it->second;
            live.erase(it);
            if (idle_bytes[b.device] + b.bytes <= (b.device == HOST ? kPoolHostBytes : kPoolBytes)) {
                idle_bytes[b.device] += b.bytes;
                idle.insert({{b.device, b.bytes}, p});
                return;
            }
        }
        release(b.device, p);
    }
};
// never destroyed: at process exit the driver may be gone before static destructors run
Pool& pool() { static Pool* p = new Pool(); return *p; }
}  // namespace

void* pool_alloc(size_t bytes) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    return pool().take(device, bytes);
}
void* pool_alloc_host(size_t bytes) { return pool().take(HOST, bytes); }
void pool_free(void* p) { pool().give(p); }
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
void pool_trim(int device) { pool().trim(device); pool().trim(HOST); }

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
    void* b = p.take(HOST, n_bytes);
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
    pool().give(p);
}
