// pinned.cpp -- the process-wide pool of page-locked host blocks.
#include "pinned.h"

#include <cuda_runtime.h>
#include <stdlib.h>

#include <list>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace fgss {

namespace {

// Page-locked blocks for the pairs and token sets handed to the caller: the
// device-to-host copies of the columns run at the link's rate and write no
// freshly mapped pages (200,000 reads tokenized: 95 ms of copies into malloc'd
// pages, 4 ms into blocks of the pool).  Freeing a result gives its block back to
// the pool that the next call takes it from; the pool keeps at most kFreeBytes of
// free blocks, releasing those given back longest ago first, and hands out at most
// kLiveBytes at a time.  It is guarded by a mutex and never destroyed: blocks may
// be given back at exit.
struct PinnedPool {
    std::mutex mu;
    std::list<std::pair<void*, size_t>> free_blocks;  // oldest first
    std::map<void*, size_t> sizes;                    // every block of the pool, handed out or free
    size_t free_bytes = 0, all_bytes = 0;
};
constexpr size_t kFreeBytes = size_t(1) << 30, kLiveBytes = size_t(16) << 30;

PinnedPool& pinned_pool() {
    static PinnedPool* pool = new PinnedPool;
    return *pool;
}

}  // namespace

// The smallest free block of at most twice the size, else a new one.
void* pinned_take(size_t bytes) {
    PinnedPool& P = pinned_pool();
    {
        std::lock_guard<std::mutex> lk(P.mu);
        auto best = P.free_blocks.end();
        for (auto it = P.free_blocks.begin(); it != P.free_blocks.end(); ++it)
            if (it->second >= bytes && it->second <= 2 * bytes + (size_t(1) << 20) &&
                (best == P.free_blocks.end() || it->second < best->second))
                best = it;
        if (best != P.free_blocks.end()) {
            void* b = best->first;
            P.free_bytes -= best->second;
            P.free_blocks.erase(best);
            return b;
        }
        if (P.all_bytes - P.free_bytes + bytes > kLiveBytes) return nullptr;
    }
    void* b = nullptr;
    if (cudaHostAlloc(&b, bytes, cudaHostAllocPortable) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(P.mu);
    P.sizes[b] = bytes;
    P.all_bytes += bytes;
    return b;
}

bool pinned_give(void* b) {
    PinnedPool& P = pinned_pool();
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.sizes.find(b);
    if (it == P.sizes.end()) return false;
    P.free_blocks.emplace_back(b, it->second);
    P.free_bytes += it->second;
    while (P.free_bytes > kFreeBytes) {
        const auto old = P.free_blocks.front();
        P.free_blocks.pop_front();
        P.free_bytes -= old.second;
        P.all_bytes -= old.second;
        P.sizes.erase(old.first);
        if (cudaFreeHost(old.first) != cudaSuccess) (void)cudaGetLastError();
    }
    return true;
}

bool pinned_holds(const void* p, size_t bytes) {
    PinnedPool& P = pinned_pool();
    std::lock_guard<std::mutex> lk(P.mu);
    auto it = P.sizes.upper_bound(const_cast<void*>(p));
    if (it == P.sizes.begin()) return false;
    --it;
    const char* b = static_cast<const char*>(it->first);
    return static_cast<const char*>(p) + bytes <= b + it->second;
}

void alloc_host_sets(fgss_sets* s, uint64_t n, uint64_t T, bool loc) {
    const size_t nc = ((n + 1) * 4 + 255) & ~size_t(255), tc = ((T + 1) * 4 + 255) & ~size_t(255);
    if (char* b = static_cast<char*>(pinned_take(3 * nc + (loc ? 2 : 1) * tc))) {
        s->id = reinterpret_cast<uint32_t*>(b);
        s->pos = reinterpret_cast<uint32_t*>(b + nc);
        s->len = reinterpret_cast<uint32_t*>(b + 2 * nc);
        s->tokens = reinterpret_cast<uint32_t*>(b + 3 * nc);
        s->loc = loc ? reinterpret_cast<uint32_t*>(b + 3 * nc + tc) : nullptr;
        return;
    }
    s->id = static_cast<uint32_t*>(malloc(nc));
    s->pos = static_cast<uint32_t*>(malloc(nc));
    s->len = static_cast<uint32_t*>(malloc(nc));
    s->tokens = static_cast<uint32_t*>(malloc(tc));
    s->loc = loc ? static_cast<uint32_t*>(malloc(tc)) : nullptr;
    if (!s->id || !s->pos || !s->len || !s->tokens || (loc && !s->loc))
        fail(FGSS_ERR_NOMEM, "host allocation for token sets");
}

}  // namespace fgss
