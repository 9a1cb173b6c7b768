// host_blocks.hpp -- the page-locked blocks msosm_host_alloc has handed out, so
// that a kernel writes a result to host memory itself only where the whole
// result lies in one of them: that a pointer's first byte is page-locked says
// nothing about the bytes after it.
#pragma once

#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>

namespace msosm {

class HostBlocks {
public:
    // a block of the context ctx (context_id()); may throw std::bad_alloc
    void add(const void *p, size_t bytes, unsigned long long ctx)
    {
        const std::lock_guard<std::mutex> lock(m_);
        blocks_[(uintptr_t)p] = {bytes, ctx};
    }
    void remove(const void *p)
    {
        const std::lock_guard<std::mutex> lock(m_);
        blocks_.erase((uintptr_t)p);
    }
    // whether [p, p + bytes) lies in one block of the context ctx
    bool covers(const void *p, size_t bytes, unsigned long long ctx) const
    {
        const std::lock_guard<std::mutex> lock(m_);
        auto it = blocks_.upper_bound((uintptr_t)p);
        if (it == blocks_.begin())
            return false;
        --it;
        const uintptr_t at = (uintptr_t)p - it->first;
        return it->second.ctx == ctx && at <= it->second.bytes && bytes <= it->second.bytes - at;
    }

private:
    struct Block {
        size_t bytes;
        unsigned long long ctx;
    };
    mutable std::mutex m_;
    std::map<uintptr_t, Block> blocks_;
};

HostBlocks &host_blocks();  // sim.cu

}  // namespace msosm
