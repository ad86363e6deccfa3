// Random use of a BlockPool (wah_pool.h) over a driver that counts what it
// hands out and fails past a limit — test code (tests/test_pool.py).
#include "../libfastlib_b200/csrc/wah_pool.h"
#include <cstdint>
#include <cstdlib>
#include <random>
#include <set>
using wah::BlockPool;
namespace {
size_t held, limit, calls;
std::map<void*, size_t> given;
void* get(size_t b) {
    ++calls;
    if (held + b > limit) return nullptr;
    held += b;
    void* p = aligned_alloc(256, b);
    given[p] = b;
    return p;
}
void put(void* p) { held -= given[p]; given.erase(p); free(p); }
}  // namespace
// Returns 0, or the number of the check that failed.
extern "C" int pool_model(uint32_t seed, int steps) {
    held = calls = 0;
    limit = (size_t)1 << 40;
    std::mt19937 r(seed);
    {
        BlockPool P(get, put, 1 << 16, 2, 1 << 20);
        std::map<char*, size_t> live;  // block -> bytes asked for
        for (int i = 0; i < steps; ++i) {
            if (live.empty() || r() % 5 < 3) {
                const size_t b = 1 + (r() % 8 == 0 ? r() % (4 << 20) : r() % (1u << (8 + r() % 10)));
                char* p = static_cast<char*>(P.take(b));
                if (!p || (uintptr_t)p % 256 || P.size(p) < b) return 1;
                auto n = live.lower_bound(p);  // overlaps no other block
                if (n != live.end() && p + b > n->first) return 2;
                if (n != live.begin() && std::prev(n)->first + std::prev(n)->second > p) return 3;
                bool inside = false;
                for (auto& g : given)
                    inside |= p >= (char*)g.first && p + P.size(p) <= (char*)g.first + g.second;
                if (!inside) return 4;
                p[0] = p[b - 1] = 1;
                live[p] = b;
            } else {
                auto it = live.begin();
                std::advance(it, r() % live.size());
                P.give(it->first);
                live.erase(it);
            }
            if (i % 97 == 0) P.trim();
            for (auto& l : live)
                if (i % 50 == 0 && P.size(l.first) < l.second) return 5;
        }
        for (auto& l : live) P.give(l.first);
        P.trim();
        if (held) return 6;
    }
    {  // the same sizes again ask the driver for nothing
        BlockPool P(get, put, 1 << 16, 2, 1 << 20);
        for (int round = 0; round < 3; ++round) {
            const size_t c0 = calls;
            std::vector<void*> v;
            for (size_t b = 100; b < (8u << 20); b = b * 3 / 2) v.push_back(P.take(b));
            for (void* p : v) P.give(p);
            if (round && calls != c0) return 7;
        }
        // and room made beforehand serves without the driver
        BlockPool Q(get, put, 1 << 16, 2, 1 << 20);
        if (!Q.reserve(16 << 20)) return 8;
        const size_t c0 = calls;
        for (int i = 0; i < 4; ++i)
            if (!Q.take(3 << 20)) return 9;
        if (calls != c0) return 10;
    }
    {  // no memory for a whole slab: the block alone; none for that: null, and the pool goes on
        BlockPool P(get, put, 1 << 16, 2, 1 << 20);
        limit = held + 5000;
        void* p = P.take(4000);
        if (!p || P.take(4000)) return 11;
        P.give(p);
        if (P.take(4096) != p) return 12;
        P.give(p);
        P.give(nullptr);
        P.trim();
        if (held || !P.take(300)) return 13;
    }
    return held ? 14 : 0;
}
