// devmem.cpp -- device and small pinned allocations of the library.
//
// A matrix load makes some twenty device allocations and the serving loop
// loads a matrix per solve.  cudaMalloc maps memory and cudaFree unmaps it
// after waiting for the device: 60 us for a small pair, 0.46 ms for one of
// 512 MB, and a pinned page costs 0.27 ms to allocate and free (GB300).  So
// device blocks come from one memory pool per device (1.9 us for a pair of
// any size) and handles' pinned result words from shared pinned pages.
//
// Bounds: memory that no handle or service uses stays in a pool up to 1/64 of
// the device's (4.4 GB here; what exceeds it goes back to the device at the
// next synchronisation), all but 1/1024 (0.28 GB) goes back when the last block
// is freed, and an allocation that fails empties the pool and tries again.
// (A program that makes, uses and drops one small handle after another maps
// its memory once: without the 1/1024 and one pinned page kept, 0.45 ms of the
// 0.7 to 0.8 ms of each.)  The pool's
// stream only orders allocations: a block is ready on every stream when
// dev_alloc returns, and dev_free, unlike cudaFree, waits for nothing -- its
// callers have synchronised the work that used the block.  A handle cannot
// know all the work that uses its blocks (a graph captured from its stream may
// be replayed on any other), so it frees them inside a DevIdle scope, which
// waits for the device first, as cudaFree did.  All of these may be called
// from any thread.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "internal.h"

namespace pwmgpu {

namespace {

struct Pool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    long long live = 0;  // blocks in use
    size_t keep = 0;     // bytes kept when none is
    void* anchor = nullptr;  // see wait_device
};

std::mutex g_mu;
// never destroyed: blocks may be freed while the process exits
std::map<int, Pool>& pools() {
    static auto* p = new std::map<int, Pool>();
    return *p;
}

// Blocks freed where the device could not be waited for: {device, block}.
std::vector<std::pair<int, void*>>& kept() {
    static auto* p = new std::vector<std::pair<int, void*>>();
    return *p;
}
thread_local int t_keep = 0;  // > 0: this thread's frees go to kept()

// The pool of device `dev` (the current one), made on first use; null with
// *e set when it cannot be made.  Call with g_mu held.
Pool* pool_of(int dev, cudaError_t* e) {
    Pool& p = pools()[dev];
    if (p.pool) return &p;
    size_t total = 0, free_now = 0;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    *e = cudaMemGetInfo(&free_now, &total);
    cudaStream_t st = nullptr;
    if (*e == cudaSuccess) *e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    cudaMemPool_t pool = nullptr;
    if (*e == cudaSuccess) *e = cudaMemPoolCreate(&pool, &props);
    unsigned long long keep = total / 64;
    if (*e == cudaSuccess) *e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (*e != cudaSuccess) {
        if (pool) cudaMemPoolDestroy(pool);
        if (st) cudaStreamDestroy(st);
        return nullptr;
    }
    p.pool = pool;
    p.stream = st;
    p.keep = total / 1024;
    return &p;
}

}  // namespace

cudaError_t dev_alloc(void** out, size_t bytes) {
    *out = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    Pool p;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        Pool* q = pool_of(dev, &e);
        if (!q) return e;
        ++q->live;
        p = *q;
    }
    for (int attempt = 0; attempt < 2; ++attempt) {
        e = cudaMallocFromPoolAsync(out, bytes ? bytes : 1, p.pool, p.stream);
        if (e != cudaErrorMemoryAllocation) break;
        (void)cudaGetLastError();
        (void)cudaStreamSynchronize(p.stream);  // (frees still under way hold their blocks)
        cudaMemPoolTrimTo(p.pool, 0);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(p.stream);
    if (e != cudaSuccess) {
        *out = nullptr;
        std::lock_guard<std::mutex> lk(g_mu);
        --pools()[dev].live;
    }
    return e;
}

void dev_free(void* p) {
    if (!p) return;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (t_keep > 0) {
        try {
            kept().emplace_back(a.device, p);
        } catch (const std::bad_alloc&) {  // the block stays allocated
        }
        return;
    }
    Pool& q = pools()[a.device];
    cudaFreeAsync(p, q.stream);
    if (--q.live == 0) {
        cudaStreamSynchronize(q.stream);
        cudaMemPoolTrimTo(q.pool, q.keep);
    }
}

namespace {

// Waits for the device's work by freeing a small block, as cudaFree does.  Not
// by cudaDeviceSynchronize: that is refused, and the capture spoilt, while any
// stream is being captured, where cudaFree works beside a relaxed capture.
// Another block of the same size stays allocated, so that the memory they lie
// in stays mapped: 2 us, 55 without it.
cudaError_t wait_device(int device) {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        Pool& q = pools()[device];
        if (!q.anchor && cudaMalloc(&q.anchor, 256) != cudaSuccess) {
            (void)cudaGetLastError();
            q.anchor = nullptr;
        }
    }
    void* p = nullptr;
    const cudaError_t e = cudaMalloc(&p, 256);
    if (e == cudaSuccess) return cudaFree(p);
    if (e != cudaErrorMemoryAllocation) return e;
    (void)cudaGetLastError();
    return cudaDeviceSynchronize();
}

}  // namespace

DevIdle::DevIdle(int device) {
    int cur = device;
    (void)cudaGetDevice(&cur);
    if (cur != device) (void)cudaSetDevice(device);
    refused_ = wait_device(device) != cudaSuccess;
    if (cur != device) (void)cudaSetDevice(cur);
    if (refused_) {
        (void)cudaGetLastError();
        ++t_keep;
        return;
    }
    std::vector<std::pair<int, void*>> back;  // what earlier scopes could not wait for
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (kept().empty()) return;
        back.swap(kept());
    }
    for (auto& b : back) {
        if (b.first == device && t_keep == 0) {
            dev_free(b.second);
            continue;
        }
        std::lock_guard<std::mutex> lk(g_mu);
        try {
            kept().push_back(b);
        } catch (const std::bad_alloc&) {
        }
    }
}

DevIdle::~DevIdle() {
    if (refused_) --t_keep;
}

size_t dev_idle_bytes() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lk(g_mu);
    const Pool& q = pools()[dev];
    unsigned long long held = 0, used = 0;
    if (!q.pool || cudaMemPoolGetAttribute(q.pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
        cudaMemPoolGetAttribute(q.pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return held > used ? (size_t)(held - used) : 0;
}

// ---- small pinned blocks ---------------------------------------------------
namespace {

constexpr size_t kPinnedPage = 64 * kPinnedBlock;
struct Pinned {
    std::vector<void*> pages, free;
    size_t used = 0;
};
Pinned& pinned() {
    static auto* p = new Pinned();
    return *p;
}

}  // namespace

cudaError_t pinned_alloc(void** out) {
    *out = nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    Pinned& P = pinned();
    if (P.free.empty()) {
        void* page = nullptr;
        // portable: a block may serve a handle on any device
        const cudaError_t e = cudaHostAlloc(&page, kPinnedPage, cudaHostAllocPortable);
        if (e != cudaSuccess) return e;
        P.pages.push_back(page);
        for (size_t o = kPinnedPage; o > 0; o -= kPinnedBlock)
            P.free.push_back(static_cast<unsigned char*>(page) + (o - kPinnedBlock));
    }
    *out = P.free.back();
    P.free.pop_back();
    ++P.used;
    return cudaSuccess;
}

void pinned_free(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_mu);
    Pinned& P = pinned();
    P.free.push_back(p);
    if (--P.used == 0 && P.pages.size() > 1) {
        for (void* page : P.pages) cudaFreeHost(page);
        P.pages.clear();
        P.free.clear();
    }
}

}  // namespace pwmgpu
