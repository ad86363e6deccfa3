// Blocks of device or pinned host memory for one context.
//
// Asking the driver takes long (device memory 0.4-0.5 ms from 2 MB to 256 MB;
// pinned memory 1 ms for 2 MB, 3.4 ms for 8 MB, 32 ms for 64 MB; either now and
// then tens of ms; less than 1 MB is cheap, the driver shares out 2 MB at a
// time), so blocks are carved out of a few slabs, small ones first, that grow,
// and blocks given back serve later calls.  A block is
// handed on in the order of the context's stream: whoever takes it next runs
// after the work that used it.
#ifndef WAH_POOL_H
#define WAH_POOL_H
#include <stddef.h>
#include <algorithm>
#include <iterator>
#include <list>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace wah {

class BlockPool {
  public:
    // get / put: the driver's calls (get: null when there is no memory);
    // first .. most: bytes of a slab, `grow` times the last one's.  Blocks of
    // more than a quarter of `most` have a slab of their own.
    BlockPool(void* (*get)(size_t), void (*put)(void*), size_t first, size_t grow, size_t most)
        : get_(get), put_(put), next_(first), grow_(grow), most_(most) {}
    ~BlockPool() {
        for (Slab& s : slabs_) put_(s.base);
    }
    BlockPool(const BlockPool&) = delete;
    BlockPool& operator=(const BlockPool&) = delete;

    // Powers of two from 256 bytes to 1 MB, then whole MB.
    static size_t size_class(size_t b) {
        constexpr size_t MB = (size_t)1 << 20;
        if (b > MB) return (b + MB - 1) & ~(MB - 1);
        size_t c = 256;
        while (c < b) c <<= 1;
        return c;
    }

    // A block of at least `bytes`, or null.  A block given back serves sizes of
    // its class; one of several MB that shares a slab, sizes down to its half too.
    void* take(size_t bytes) {
        const size_t c = size_class(bytes), upto = c > ((size_t)1 << 20) && c <= most_ / 4 ? 2 * c : c;
        std::lock_guard<std::mutex> g(mu_);
        for (auto it = free_.lower_bound(c); it != free_.end() && it->first <= upto; ++it) {
            if (it->second.empty()) continue;
            void* p = it->second.back();
            it->second.pop_back();
            ++blocks_[p].slab->out;
            return p;
        }
        for (auto s = slabs_.rbegin(); s != slabs_.rend(); ++s)
            if (s->size - s->used >= c) return carve(*s, c);
        if (c <= most_ / 4) {
            if (add(std::max(next_, c))) {
                next_ = std::min(most_, grow_ * next_);
                return carve(slabs_.back(), c);
            }
        }
        return add(c) ? carve(slabs_.back(), c) : nullptr;
    }
    void give(void* p) {
        if (!p) return;
        std::lock_guard<std::mutex> g(mu_);
        auto it = blocks_.find(p);
        if (it == blocks_.end()) return;
        --it->second.slab->out;
        free_[it->second.bytes].push_back(p);
    }
    size_t size(void* p) {
        std::lock_guard<std::mutex> g(mu_);
        auto it = blocks_.find(p);
        return it == blocks_.end() ? 0 : it->second.bytes;
    }
    // Room for `bytes` of blocks beforehand; false when there is no memory.
    bool reserve(size_t bytes) {
        std::lock_guard<std::mutex> g(mu_);
        return bytes == 0 || add(size_class(bytes));
    }
    // Gives back the slabs none of whose blocks are out.
    void trim() {
        std::lock_guard<std::mutex> g(mu_);
        for (auto s = slabs_.begin(); s != slabs_.end();) {
            if (s->out) { ++s; continue; }
            for (auto& f : free_)
                f.second.erase(std::remove_if(f.second.begin(), f.second.end(),
                                              [&](void* p) { return blocks_[p].slab == &*s; }),
                               f.second.end());
            for (auto b = blocks_.begin(); b != blocks_.end();) b = b->second.slab == &*s ? blocks_.erase(b) : std::next(b);
            put_(s->base);
            s = slabs_.erase(s);
        }
    }

  private:
    struct Slab { char* base; size_t size, used; size_t out; };  // out: blocks in use
    struct Block { size_t bytes; Slab* slab; };
    bool add(size_t bytes) {
        void* p = get_(bytes);
        if (p) slabs_.push_back(Slab{static_cast<char*>(p), bytes, 0, 0});
        return p != nullptr;
    }
    void* carve(Slab& s, size_t c) {
        char* p = s.base + s.used;
        s.used += c;
        ++s.out;
        blocks_[p] = Block{c, &s};
        return p;
    }
    void* (*get_)(size_t);
    void (*put_)(void*);
    size_t next_, grow_, most_;
    std::mutex mu_;
    std::list<Slab> slabs_;  // addresses stay
    std::unordered_map<void*, Block> blocks_;
    std::map<size_t, std::vector<void*>> free_;
};

}  // namespace wah
#endif
