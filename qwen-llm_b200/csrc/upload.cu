// Long host -> device uploads from pageable memory (a snapshot out of a prefix cache: 50 MB of state plus 40 - 170 KB a token).
//
// A copy from pageable memory runs at the speed of the one driver thread that moves it into a pinned buffer: 10 GB/s, where the
// link takes 55.  Here a few threads fill a ring of pinned 1 MiB slots and the caller queues each slot's copy as it fills,
// so the uploads of a restore are bound by host memory.  Four threads: more compete with each other and with other
// requests on the host.  90 MB restored: 8.5 -> 3.6 ms on 16 host cores.  Memory that is pinned already goes straight to the link.
#include <atomic>
#include <cstring>
#include <thread>

#include "model.cuh"

namespace dfl {

namespace {
constexpr size_t kChunk = 1 << 20, kSlots = 16, kWorthIt = 4 << 20;

dfl_status copy_directly(cudaStream_t st, const std::vector<Upload>& list) {
    for (const Upload& u : list) {
        DFL_CUDA(cudaMemcpyAsync(u.dst, u.src, u.bytes, cudaMemcpyHostToDevice, st));
        if (u.after) DFL_CHECK(u.after());
    }
    DFL_CUDA(cudaStreamSynchronize(st));
    return DFL_OK;
}
bool is_pinned(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeHost;
}
struct Chunk { size_t upload, offset, bytes; bool last; };
struct Ring {
    uint8_t* slots = nullptr;
    cudaEvent_t done[kSlots] = {};
    bool make() {
        if (!(slots = (uint8_t*)pool_alloc_host(kChunk * kSlots))) return false;
        for (cudaEvent_t& e : done)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { e = nullptr; cudaGetLastError(); return false; }
        return true;
    }
    ~Ring() {
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
        pool_free(slots);
    }
};
}  // namespace

dfl_status upload_all(cudaStream_t st, const std::vector<Upload>& list) {
    size_t total = 0;
    for (const Upload& u : list) total += u.bytes;
    const unsigned hw = std::thread::hardware_concurrency();
    Ring ring;
    if (total < kWorthIt || hw < 2 || is_pinned(list[0].src) || !ring.make()) return copy_directly(st, list);
    std::vector<Chunk> chunks;
    for (size_t i = 0; i < list.size(); ++i)
        for (size_t off = 0; off < list[i].bytes; off += kChunk) {
            const size_t bytes = std::min(kChunk, list[i].bytes - off);
            chunks.push_back({i, off, bytes, off + bytes == list[i].bytes});
        }
    std::vector<std::atomic<bool>> filled(chunks.size());
    for (auto& f : filled) f.store(false, std::memory_order_relaxed);
    std::atomic<size_t> next{0}, copied{0};   // chunks taken by a thread / whose copy to the device has finished
    std::atomic<bool> stop{false};
    auto fill = [&] {
        for (;;) {
            const size_t c = next.fetch_add(1);
            if (c >= chunks.size()) return;
            while (c >= copied.load(std::memory_order_acquire) + kSlots) {
                if (stop.load()) return;
                std::this_thread::yield();
            }
            memcpy(ring.slots + c % kSlots * kChunk, (const uint8_t*)list[chunks[c].upload].src + chunks[c].offset, chunks[c].bytes);
            filled[c].store(true, std::memory_order_release);
        }
    };
    std::vector<std::thread> threads;
    try {
        while (threads.size() < std::min(4u, hw - 1)) threads.emplace_back(fill);
    } catch (...) {
        if (threads.empty()) return copy_directly(st, list);   // no thread to be had
    }
    dfl_status status = DFL_OK;
    cudaError_t e = cudaSuccess;
    size_t oldest = 0;
    for (size_t c = 0; c < chunks.size() && status == DFL_OK && e == cudaSuccess; ++c) {
        while (!filled[c].load(std::memory_order_acquire)) {
            if (oldest < c && cudaEventQuery(ring.done[oldest % kSlots]) != cudaErrorNotReady) copied.store(++oldest, std::memory_order_release);
            else std::this_thread::yield();
        }
        const Chunk& k = chunks[c];
        const Upload& u = list[k.upload];
        e = cudaMemcpyAsync((uint8_t*)u.dst + k.offset, ring.slots + c % kSlots * kChunk, k.bytes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(ring.done[c % kSlots], st);
        if (e == cudaSuccess && k.last && u.after) status = u.after();
    }
    stop.store(true);
    for (std::thread& t : threads) t.join();
    const cudaError_t end = cudaStreamSynchronize(st);   // nothing reads the ring any more
    DFL_CHECK(status);
    DFL_CUDA(e);
    DFL_CUDA(end);
    return DFL_OK;
}

}  // namespace dfl
