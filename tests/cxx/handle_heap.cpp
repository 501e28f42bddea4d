// Random allocations and frees over the slab heap, on host memory that is
// never touched: every block inside one slab, aligned, apart from the others;
// idle slabs kept up to the bound; all given back in the end.  Prints "ok".
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>

#include "handle_heap.cuh"

#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    using Heap = rb::HandleHeap;
    for (unsigned seed = 0; seed < 6; seed++) {
        std::mt19937_64 rng(seed);
        Heap heap;
        // slabs from one address range: seeds 0..2 with no gap between them
        std::uintptr_t top = (std::uintptr_t)1 << 40;
        std::map<char*, size_t> slabs;
        auto get = [&](size_t n) -> void* {
            char* p = reinterpret_cast<char*>(top);
            top += n + (seed < 3 ? 0 : 4096);
            slabs[p] = n;
            return p;
        };
        bool known = true;
        auto put = [&](char* p) { known = known && slabs.erase(p) == 1; };
        std::map<char*, size_t> live;
        std::vector<char*> list;
        for (int step = 0; step < 20000; step++) {
            const bool grow = list.size() < 3 || (rng() % 100 < (step / 2000 % 2 ? 40u : 58u));
            if (grow) {
                const unsigned bits = 3 + rng() % 24;                 // 1 byte to 128 MB
                const size_t bytes = 1 + rng() % ((size_t)1 << bits);
                char* p = static_cast<char*>(heap.alloc(bytes, get, seed == 5 ? 0 : Heap::kSlab));
                CHECK(reinterpret_cast<std::uintptr_t>(p) % Heap::kAlign == 0);
                auto s = slabs.upper_bound(p);
                CHECK(s != slabs.begin());
                --s;
                CHECK(p + bytes <= s->first + s->second);
                auto n = live.lower_bound(p);
                CHECK(n == live.end() || p + bytes <= n->first);
                if (n != live.begin()) {
                    --n;
                    CHECK(n->first + n->second <= p);
                }
                live[p] = bytes;
                list.push_back(p);
                CHECK(heap.owns(p));
            } else {
                const size_t k = rng() % list.size();
                char* p = list[k];
                list[k] = list.back();
                list.pop_back();
                live.erase(p);
                heap.free(p, put);
                CHECK(!heap.owns(p));
            }
            CHECK(known);
            CHECK(heap.used_blocks() == live.size());
            CHECK(heap.idle_bytes() <= Heap::kKeep + ((size_t)128 << 20));
        }
        while (!list.empty()) {
            heap.free(list.back(), put);
            list.pop_back();
        }
        CHECK(heap.idle_bytes() <= Heap::kKeep);
        size_t kept = 0;
        for (auto& s : slabs) kept += s.second;
        CHECK(kept == heap.idle_bytes());
        heap.trim(put);
        CHECK(slabs.empty() && known && heap.idle_bytes() == 0 && heap.used_blocks() == 0);
    }
    printf("ok\n");
    return 0;
}
