// handle_heap.cuh -- memory whose address a caller may hold: blocks of slabs.
//
// Vectors and matrices give out their device addresses, so their memory has
// to be the driver's ordinary kind: a stream-ordered pool's cannot be
// exported to another process by cudaIpcGetMemHandle, and
// cudaDeviceEnablePeerAccess does not cover it.  But cudaMalloc and cudaFree
// of a few megabytes take 1 to 4 ms each (a 64^3 setup whose ten matrices are
// read out: 30 of both), so blocks are cut from slabs that stay (that setup
// 17.3 ms, with the matrices in the pool 17.4).  Only blocks
// of memory no kernel uses any more come back (the caller of free has waited
// for the device, as cudaFree does), so a block may be handed out again on
// any stream at once.
//
// Host code only: the slabs come from and go to the functions that a call
// passes in.  Not thread-safe by itself.
#pragma once

#include <cstddef>
#include <map>
#include <set>
#include <utility>

namespace rb {

class HandleHeap {
public:
    static constexpr size_t kAlign = 256;                     // as cudaMalloc's
    static constexpr size_t kSlab = (size_t)64 << 20;         // (arrays of 64 MB and more are the driver's)
    static constexpr size_t kKeep = (size_t)1 << 30;          // bytes of idle slabs kept

    // A block of at least `bytes`; a new slab of at least `bytes`, or `slab`
    // where that is more, comes from get(size), which may throw.
    template <class Get>
    void* alloc(size_t bytes, Get&& get, size_t slab = kSlab) {
        const size_t need = (bytes + kAlign - 1) / kAlign * kAlign;
        auto it = by_size_.lower_bound({need, nullptr});
        if (it == by_size_.end()) {
            const size_t size = need > slab ? need : slab;
            char* base = static_cast<char*>(get(size));
            slabs_[base] = size;
            add_free(base, size);
            idle_ += size;
            it = by_size_.lower_bound({need, nullptr});
        }
        char* p = it->second;
        const size_t size = it->first;
        if (whole_slab(p, size)) idle_ -= size;
        drop_free(p, size);
        if (size > need) add_free(p + need, size - need);
        used_[p] = need;
        return p;
    }

    bool owns(void* p) const { return used_.count(static_cast<char*>(p)) != 0; }

    // Takes a block back and joins it with its free neighbours; slabs that
    // are idle beyond kKeep go to put(base).
    template <class Put>
    void free(void* ptr, Put&& put) {
        auto u = used_.find(static_cast<char*>(ptr));
        if (u == used_.end()) return;
        char* p = u->first;
        size_t size = u->second;
        used_.erase(u);
        auto next = free_.find(p + size);
        if (next != free_.end() && !slabs_.count(next->first)) {   // (slabs may touch)
            const size_t s = next->second;
            drop_free(p + size, s);
            size += s;
        }
        auto prev = free_.lower_bound(p);
        if (prev != free_.begin() && !slabs_.count(p)) {
            --prev;
            char* q = prev->first;
            const size_t s = prev->second;
            if (q + s == p) {
                drop_free(q, s);
                p = q;
                size += s;
            }
        }
        add_free(p, size);
        if (whole_slab(p, size)) idle_ += size;
        if (idle_ > kKeep) trim(put);
    }

    // Gives idle slabs back until at most `keep` bytes of them are left.
    template <class Put>
    void trim(Put&& put, size_t keep = 0) {
        for (auto s = slabs_.begin(); s != slabs_.end() && idle_ > keep;) {
            auto f = free_.find(s->first);
            if (f != free_.end() && f->second == s->second) {
                char* base = s->first;
                idle_ -= s->second;
                drop_free(base, s->second);
                s = slabs_.erase(s);
                put(base);
            } else {
                ++s;
            }
        }
    }

    size_t used_blocks() const { return used_.size(); }
    size_t idle_bytes() const { return idle_; }

private:
    bool whole_slab(char* p, size_t size) const {
        auto s = slabs_.find(p);
        return s != slabs_.end() && s->second == size;
    }
    void add_free(char* p, size_t size) {
        free_[p] = size;
        by_size_.insert({size, p});
    }
    void drop_free(char* p, size_t size) {
        free_.erase(p);
        by_size_.erase({size, p});
    }
    std::map<char*, size_t> slabs_, free_, used_;
    std::set<std::pair<size_t, char*>> by_size_;   // the free blocks again
    size_t idle_ = 0;                              // bytes of slabs with no used block
};

}  // namespace rb
