// Blocks of memory that outlive their owner: what is kept, for whom, and what goes first.  The memory itself comes from a
// Source (cudaMalloc / cudaMallocHost in pool.cu, a fake one in dfl_pool_selftest).
//
// Sizes are rounded up to sixteen classes an octave (at most 1/16 more; eight for host blocks), so that owners whose sizes differ a
// little find each other's blocks.  Idle blocks of one place are bounded by bytes; the one returned longest ago goes first.
#pragma once
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace dfl {

constexpr int POOL_HOST = -1;   // place of pinned host blocks; other places are device numbers

struct BlockSource {
    virtual void* get(int place, size_t bytes) = 0;   // nullptr: no memory
    virtual void put(int place, void* p) = 0;
    virtual ~BlockSource() = default;
};

class BlockPool {
public:
    BlockPool(BlockSource& source, size_t device_limit, size_t host_limit) : src(source), limits{device_limit, host_limit} {}

    void* take(int place, size_t bytes) {
        const size_t exact = bytes ? (bytes + 511) / 512 * 512 : 512, size = size_class(place, exact);
        {
            std::lock_guard<std::mutex> lock(mu);
            auto it = idle.upper_bound({place, size});   // of several, the one returned last
            if (it != idle.begin() && (--it)->first == std::make_pair(place, size)) {
                void* p = it->second.p;
                idle.erase(it);
                idle_bytes[place] -= size;
                live[p] = {place, size, true};
                return p;
            }
        }
        size_t got = size;
        void* p = src.get(place, size);
        if (!p) {
            trim(place);
            p = src.get(place, size);
        }
        if (!p && exact < size) p = src.get(place, got = exact);   // what fits without the rounding is not refused for it
        if (!p) return nullptr;
        std::lock_guard<std::mutex> lock(mu);
        live[p] = {place, got, got == size};
        return p;
    }

    void give(void* p) {
        if (!p) return;
        std::vector<void*> out;
        int place;
        {
            std::lock_guard<std::mutex> lock(mu);
            auto l = live.find(p);
            if (l == live.end()) return;
            const Block b = l->second;
            live.erase(l);
            place = b.place;
            const size_t limit = limits[place == POOL_HOST];
            if (!b.keep || b.bytes > limit) {
                out.push_back(p);
            } else {
                while (idle_bytes[place] + b.bytes > limit) {
                    auto oldest = idle.end();
                    for (auto it = idle.lower_bound({place, 0}); it != idle.end() && it->first.first == place; ++it)
                        if (oldest == idle.end() || it->second.when < oldest->second.when) oldest = it;
                    idle_bytes[place] -= oldest->first.second;
                    out.push_back(oldest->second.p);
                    idle.erase(oldest);
                }
                idle.insert({{place, b.bytes}, {p, ++clock}});
                idle_bytes[place] += b.bytes;
            }
        }
        for (void* q : out) src.put(place, q);
    }

    // gives every idle block of the place back to its source
    void trim(int place) {
        std::vector<void*> out;
        {
            std::lock_guard<std::mutex> lock(mu);
            auto a = idle.lower_bound({place, 0}), b = a;
            for (; b != idle.end() && b->first.first == place; ++b) out.push_back(b->second.p);
            idle.erase(a, b);
            idle_bytes[place] = 0;
        }
        for (void* q : out) src.put(place, q);
    }

    static size_t size_class(int place, size_t bytes) {
        const size_t per_octave = place == POOL_HOST ? 8 : 16;
        size_t step = 512;
        while (step * 2 * per_octave <= bytes) step *= 2;
        return (bytes + step - 1) / step * step;
    }

private:
    struct Block { int place; size_t bytes; bool keep; };
    struct Idle { void* p; uint64_t when; };
    BlockSource& src;
    const size_t limits[2];   // device, host
    std::mutex mu;
    std::multimap<std::pair<int, size_t>, Idle> idle;   // equal keys in the order of their return
    std::map<int, size_t> idle_bytes;
    std::unordered_map<void*, Block> live;
    uint64_t clock = 0;
};

}  // namespace dfl
