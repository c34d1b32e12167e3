// Scratch blocks that outlive a call, one per key (device, purpose, stream).  A block that has been handed out is never freed: a CUDA graph
// captured earlier may have its address in its nodes.  So a block that must grow is set aside and a larger one takes its place, at
// least half as large again, which keeps the blocks set aside below three times the ones in use; and the old one is set aside only once
// the new one is there, so a growth that fails leaves what was there in service.
#pragma once
#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace atoma {

class WorkspacePool {
  public:
    using Key = std::tuple<int, int, const void *>;

    // alloc(bytes) returns a new block or nullptr; may_grow(), asked only where the block at hand is too small: whether it may be called at all.
    // nullptr: there is no block of that size.
    template <typename MayGrow, typename Alloc>
    void *get(const Key &key, size_t bytes, MayGrow may_grow, Alloc alloc) {
        std::lock_guard<std::mutex> lock(mu_);
        Block &b = blocks_[key];
        if (b.size >= bytes && b.ptr) return b.ptr;
        if (!may_grow()) return nullptr;
        const size_t exact = round_up(std::max<size_t>(bytes, 1)), roomy = std::max(exact, round_up(b.size + b.size / 2));
        size_t size = roomy;
        void *p = alloc(size);
        if (!p && roomy > exact) p = alloc(size = exact);
        if (!p) return nullptr;
        if (b.ptr) set_aside_.push_back(b.ptr);
        b.ptr = p;
        b.size = size;
        return p;
    }

  private:
    struct Block {
        void *ptr = nullptr;
        size_t size = 0;
    };
    static size_t round_up(size_t n) { return (n + (size_t{1} << 20) - 1) & ~((size_t{1} << 20) - 1); }
    std::mutex mu_;
    std::map<Key, Block> blocks_;
    std::vector<void *> set_aside_;
};

}  // namespace atoma
