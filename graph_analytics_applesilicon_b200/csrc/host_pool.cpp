// host_pool.cpp -- the process's pool of pinned host memory.
//
// Handles need small pinned buffers (control words, packed depths, copy rings).
// Page-locking one costs about a millisecond whatever its size, and 14 ms for 4
// MiB, more than most calls take.  Blocks are powers of two, so up to twice what
// was asked for: up to kSmall they are cut from slabs, larger ones are page-locked
// one by one and kept for the next request up to kKeep bytes.  When the last block
// comes back (the last handle is gone) everything is given back to the system.
// Blocks are page-locked for every context (portable) and belong to one owner at a
// time; the owner returns a block only after the copies into it are done.
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace gb {
namespace {

constexpr size_t kMin = 256, kSmall = 512u << 10, kSlab = 2u << 20, kKeep = 64u << 20;

struct Pool {
    std::mutex mu;
    std::map<size_t, std::vector<void*>> free;  // by block size
    std::vector<void*> slabs;
    size_t slabUsed = kSlab;  // of the newest slab
    size_t kept = 0;          // bytes of free blocks larger than kSmall
    size_t live = 0;          // blocks with an owner
};

Pool& pool() {
    static Pool* p = new Pool;  // never destroyed: handles may outlive static destruction
    return *p;
}

void* pageLock(size_t bytes) {
    void* p = nullptr;
    GB_CUDA(cudaHostAlloc(&p, bytes, cudaHostAllocPortable));
    return p;
}

size_t classOf(size_t bytes) {
    size_t c = kMin;
    while (c < bytes) c *= 2;
    return c;
}

void giveBack(Pool& p) {
    for (auto& f : p.free)
        if (f.first > kSmall)
            for (void* b : f.second) cudaFreeHost(b);
    for (void* s : p.slabs) cudaFreeHost(s);
    p.free.clear();
    p.slabs.clear();
    p.slabUsed = kSlab;
    p.kept = 0;
}

}  // namespace

void* pinnedAcquire(size_t bytes, size_t* got) {
    const size_t c = classOf(bytes);
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    void* b = nullptr;
    auto it = p.free.find(c);
    if (it != p.free.end() && !it->second.empty()) {
        b = it->second.back();
        it->second.pop_back();
        if (c > kSmall) p.kept -= c;
    } else if (c > kSmall) {
        b = pageLock(c);
    } else {
        if (p.slabUsed + c > kSlab) {
            p.slabs.push_back(pageLock(kSlab));
            p.slabUsed = 0;
        }
        b = static_cast<char*>(p.slabs.back()) + p.slabUsed;
        p.slabUsed += c;
    }
    ++p.live;
    *got = c;
    return b;
}

void pinnedRelease(void* b, size_t c) {
    Pool& p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    if (c > kSmall && p.kept + c > kKeep) {
        cudaFreeHost(b);
    } else {
        p.free[c].push_back(b);
        if (c > kSmall) p.kept += c;
    }
    if (--p.live == 0) giveBack(p);
}

}  // namespace gb
