// The pool behind scratch.h.  Host code only.
#include "scratch.h"

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

namespace wqc {

namespace {

struct Block {
    void* p;
    size_t cap;
};
struct Pool {
    std::vector<Block> idle;  // oldest first
    size_t bytes = 0;
    int states = 0;
};
struct Pools {
    std::mutex mu;
    std::map<int, Pool> of;  // by device
};
// Never destroyed: states may outlive static destructors.
Pools& pools() {
    static Pools* all = new Pools;
    return *all;
}

// Blocks are freed outside the lock: cudaFree waits for the device.
void free_blocks(const std::vector<Block>& blocks) {
    for (const Block& b : blocks) cudaFree(b.p);
}

}  // namespace

void* scratch_take(int device, size_t bytes, size_t* cap) {
    Pools& all = pools();
    std::lock_guard<std::mutex> hold(all.mu);
    Pool& pool = all.of[device];
    auto best = pool.idle.end();
    for (auto it = pool.idle.begin(); it != pool.idle.end(); ++it)
        if (it->cap >= bytes && (best == pool.idle.end() || it->cap < best->cap)) best = it;
    if (best == pool.idle.end()) return nullptr;
    const Block b = *best;
    pool.idle.erase(best);
    pool.bytes -= b.cap;
    *cap = b.cap;
    return b.p;
}

void scratch_give(int device, void* p, size_t cap) {
    std::vector<Block> out;
    {
        Pools& all = pools();
        std::lock_guard<std::mutex> hold(all.mu);
        Pool& pool = all.of[device];
        if (cap > kScratchKeep || pool.states == 0) {
            out.push_back({p, cap});
        } else {
            while (pool.bytes + cap > kScratchKeep) {
                out.push_back(pool.idle.front());
                pool.bytes -= pool.idle.front().cap;
                pool.idle.erase(pool.idle.begin());
            }
            pool.idle.push_back({p, cap});
            pool.bytes += cap;
        }
    }
    free_blocks(out);
}

bool scratch_release(int device) {
    std::vector<Block> out;
    {
        Pools& all = pools();
        std::lock_guard<std::mutex> hold(all.mu);
        Pool& pool = all.of[device];
        out.swap(pool.idle);
        pool.bytes = 0;
    }
    free_blocks(out);
    return !out.empty();
}

void scratch_states(int device, int change) {
    bool last = false;
    {
        Pools& all = pools();
        std::lock_guard<std::mutex> hold(all.mu);
        Pool& pool = all.of[device];
        pool.states += change;
        last = pool.states == 0;
    }
    if (last) scratch_release(device);
}

cudaError_t device_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || !scratch_release(device)) return e;
    cudaGetLastError();
    return cudaMalloc(p, bytes);
}

cudaError_t device_room(uint64_t need, size_t* free_bytes) {
    size_t total = 0;
    int device = 0;
    cudaError_t e = cudaMemGetInfo(free_bytes, &total);
    if (e == cudaSuccess && need > *free_bytes && (e = cudaGetDevice(&device)) == cudaSuccess && scratch_release(device))
        e = cudaMemGetInfo(free_bytes, &total);
    return e;
}

}  // namespace wqc
