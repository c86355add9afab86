// ws_pool.cu -- the memory workspaces are made of.
//
// A program that makes a workspace per problem (lstsq does, each call) spends
// more on the driver than on a small solve: 0.35 ms a cudaMalloc, 0.3 ms a
// cudaFree, 1.1 to 2.8 ms for 4 KB of pinned memory and 0.4 ms to free it,
// 4 to 8 ms of a 200000 x 500 call of 20.  So blocks that workspaces give
// back are kept for later ones: at most kKeepBytes of device memory and
// kKeepHost pinned blocks a process; the device memory is released when an
// allocation fails.
//
// A workspace's memory is used on its own stream, and by the blocking copy of
// a solve's residual history, which is over when it returns.  Its owner waits
// for that stream before a block comes back (release_memory, lsqr.cuh), so
// the next one to be given it finds it idle; not by a wait for the device,
// which another thread's stream capture forbids.  One lock guards the lists; no block is in
// two hands.
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "lsqr.cuh"

namespace tomos_b200 {

namespace {

constexpr size_t kKeepBytes = (size_t)64 << 20;
constexpr size_t kKeepBlocks = 32;
constexpr size_t kKeepHost = 8;
constexpr size_t kHostBlock = 4096;

struct Block {
    void* p;
    size_t bytes;
    int device;
};

struct Pool {
    std::mutex mu;
    std::vector<Block> kept;
    size_t kept_bytes = 0;
    std::unordered_map<void*, Block> live;
    std::vector<void*> host;
};

Pool& pool() {
    static Pool* p = new Pool();  // outlives every workspace; the process's end returns the memory
    return *p;
}

}  // namespace

cudaError_t pool_malloc(void** out, size_t bytes) {
    *out = nullptr;
    Pool& P = pool();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (bytes == 0) bytes = 1;
    std::lock_guard<std::mutex> lk(P.mu);
    size_t best = P.kept.size();
    for (size_t i = 0; i < P.kept.size(); ++i) {  // the smallest that fits without wasting half of itself
        const Block& b = P.kept[i];
        if (b.device != dev || b.bytes < bytes || b.bytes / 2 > bytes) continue;
        if (best == P.kept.size() || b.bytes < P.kept[best].bytes) best = i;
    }
    Block b{nullptr, bytes, dev};
    if (best < P.kept.size()) {
        b = P.kept[best];
        P.kept[best] = P.kept.back();
        P.kept.pop_back();
        P.kept_bytes -= b.bytes;
    } else {
        e = cudaMalloc(&b.p, bytes);
        if (e == cudaErrorMemoryAllocation && !P.kept.empty()) {
            cudaGetLastError();
            for (const Block& k : P.kept) cudaFree(k.p);
            P.kept.clear();
            P.kept_bytes = 0;
            e = cudaMalloc(&b.p, bytes);
        }
        if (e != cudaSuccess) return e;
    }
    P.live[b.p] = b;
    *out = b.p;
    return cudaSuccess;
}

void pool_free(void* p) {
    if (!p) return;
    Pool& P = pool();
    Block b{nullptr, 0, 0};
    {
        std::lock_guard<std::mutex> lk(P.mu);
        auto it = P.live.find(p);
        if (it != P.live.end()) {
            b = it->second;
            P.live.erase(it);
        }
    }
    if (b.p && b.bytes <= kKeepBytes / 2) {
        std::lock_guard<std::mutex> lk(P.mu);
        if (P.kept.size() < kKeepBlocks && P.kept_bytes + b.bytes <= kKeepBytes) {
            P.kept.push_back(b);
            P.kept_bytes += b.bytes;
            return;
        }
    }
    cudaFree(p);
}

cudaError_t pool_malloc_host(void** out, size_t bytes) {
    *out = nullptr;
    if (bytes > kHostBlock) return cudaErrorInvalidValue;
    Pool& P = pool();
    {
        std::lock_guard<std::mutex> lk(P.mu);
        if (!P.host.empty()) {
            *out = P.host.back();
            P.host.pop_back();
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(out, kHostBlock, cudaHostAllocPortable);
}

void pool_free_host(void* p) {
    if (!p) return;
    Pool& P = pool();
    {
        std::lock_guard<std::mutex> lk(P.mu);
        if (P.host.size() < kKeepHost) {
            P.host.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

}  // namespace tomos_b200
