// Device memory of the cache objects.  Host code only; of CUDA it uses cudaMalloc, cudaFree and cudaGetLastError.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <list>
#include <new>
#include <vector>

namespace tqb {

// Blocks of device memory that a cache object gives up (reset, growth) and takes again: cudaMalloc and cudaFree cost
// 80 to 500 us each and cudaFree waits for the whole device, so a request of 16 steps on 28 layers spent 18 of its 20 ms
// in them.  Small blocks come from slabs: the layers of a cache grow to the same size one after the other, so the first one
// asks for all that are as far behind (`blocks_ahead`; a new cache's 28 layers of 1,024 tokens stored: 9.1 -> 0.9 ms).
// The pool belongs to one cache object and is given back with the object or when an allocation fails.  Beyond kKeepBytes held, wholly
// unused slabs are freed, the oldest first, until no more than that is held: after a reset the bound is exact.  While the cache
// is in use, blocks that share a slab with a live one come on top; they go when that one does.  Every idle block is unused: its owner has synchronised the device before it was put here.  A block that a layer outgrows
// while work may still use it is retired: nothing takes it before settle(), which a reset calls after it has waited for the device.
class BlockPool {
    struct Slab {
        void* p;
        int blocks, used;   // used: not idle, not retired
    };

public:
    static constexpr size_t kKeepBytes = 512u << 20, kSlabBytes = 64u << 20;
    struct Block {
        void* p = nullptr;
        size_t bytes = 0;
        Slab* slab = nullptr;
    };

    // The smallest idle block that fits, unless it is more than twice as large; else a new one, out of a slab of up to
    // `alike` blocks of the size.  `use_idle` = false while the stream is being captured: whatever cudaMalloc answers there is the answer.
    cudaError_t take(size_t need, int alike, bool use_idle, Block* out) {
        if (use_idle && take_idle(need, out)) return cudaSuccess;
        int count = use_idle && need <= kSlabBytes / 2 ? (int)std::min<size_t>((size_t)alike, kSlabBytes / need) : 1;
        if (count < 1) count = 1;
        void* p = nullptr;
        cudaError_t e = cudaMalloc(&p, need * count);
        if (e == cudaErrorMemoryAllocation && (count > 1 || held_ > 0)) {
            cudaGetLastError();
            trim(0);
            count = 1;
            e = cudaMalloc(&p, need);
        }
        if (e != cudaSuccess) return e;
        try {   // room for every block in either list: hold() and settle() never allocate
            idle_.reserve(blocks_ + count);
            retired_.reserve(blocks_ + count);
            slabs_.push_back(Slab{p, count, count});
        } catch (const std::bad_alloc&) {
            cudaFree(p);
            return cudaErrorMemoryAllocation;
        }
        blocks_ += count;
        Slab* slab = &slabs_.back();
        for (int i = 1; i < count; ++i) put(Block{(char*)p + i * need, need, slab});
        *out = Block{p, need, slab};
        return cudaSuccess;
    }
    void put(const Block& b) { hold(b, idle_); }
    void retire(const Block& b) { hold(b, retired_); }
    // Nothing queued on the device uses a retired block any more.
    void settle() {
        idle_.insert(idle_.end(), retired_.begin(), retired_.end());
        retired_.clear();
    }
    // Frees slabs without a live block, the oldest first, until at most `keep` bytes are held (cudaFree waits for work that still uses
    // a retired block).
    void trim(size_t keep) {
        for (auto it = slabs_.begin(); it != slabs_.end() && held_ > keep;) {
            if (it->used > 0) {
                ++it;
                continue;
            }
            for (auto* list : {&idle_, &retired_})
                for (size_t k = list->size(); k-- > 0;)
                    if ((*list)[k].slab == &*it) {
                        held_ -= (*list)[k].bytes;
                        list->erase(list->begin() + k);
                    }
            cudaFree(it->p);
            blocks_ -= it->blocks;
            it = slabs_.erase(it);
        }
    }
    // Slabs that hold memory (the pool keeps no record of any other).
    size_t slabs() const { return slabs_.size(); }
    // With the object: live blocks too.
    void release() {
        for (auto& s : slabs_) cudaFree(s.p);
        slabs_.clear();
        idle_.clear();
        retired_.clear();
        held_ = blocks_ = 0;
    }

private:
    std::vector<Block> idle_, retired_;
    std::list<Slab> slabs_;   // by age; blocks point into it
    size_t held_ = 0;         // bytes of both lists
    size_t blocks_ = 0;       // of all slabs

    void hold(const Block& b, std::vector<Block>& list) {
        if (!b.p) return;
        list.push_back(b);
        held_ += b.bytes;
        --b.slab->used;
        if (held_ > kKeepBytes) trim(kKeepBytes);
    }

    bool take_idle(size_t need, Block* out) {
        size_t best = idle_.size();
        for (size_t i = 0; i < idle_.size(); ++i)
            if (idle_[i].bytes >= need && idle_[i].bytes / 2 <= need && (best == idle_.size() || idle_[i].bytes < idle_[best].bytes)) best = i;
        if (best == idle_.size()) return false;
        *out = idle_[best];
        held_ -= out->bytes;
        ++out->slab->used;
        idle_.erase(idle_.begin() + best);
        return true;
    }
};

// How many blocks of a size a growing layer asks for at once: its own, one for each layer in use that will need the same next, and of
// the layers never used all at the layer's own first growth (the first prompt of a new cache), later no more than are in use: a
// program that uses one layer of 80 holds a block more than it needs, not 79.
template <typename Layers>
int blocks_ahead(const Layers& layers, int64_t own_cap, int64_t needed) {
    int behind = 0, used = 0, unused = 0;
    for (const auto& o : layers) {
        if (o.cap == 0) {
            ++unused;
        } else {
            ++used;
            behind += o.cap < needed ? 1 : 0;
        }
    }
    return own_cap == 0 ? behind + unused : behind + std::min(unused, used);
}

inline size_t align256(size_t n) { return (n + 255) / 256 * 256; }

}  // namespace tqb
