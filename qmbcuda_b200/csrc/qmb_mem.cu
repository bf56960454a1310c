// qmb_mem.cu -- device memory of the library's buffers (DevBuf).
//
// A sector, a matrix and a solve each take and free ten to thirty buffers, and
// cudaMalloc and cudaFree cost 0.1 to 0.3 ms each for the larger ones: at 28
// sites they were 9 of the 13 ms of building a sector and its matrix (its
// kernels take 2.5 ms).  Freed buffers of up to kMaxBlock bytes are therefore
// kept, at most kMaxTotal bytes a device, and handed out again.
//
// Rules.  A buffer comes here only idle: no work on any stream may still use
// it.  DevBuf::mark_idle() says so, and is called after the wait that ends a
// solve or a build, or on a handle's buffers once the first of them went through
// cudaFree, which waits for the device; every other buffer is freed as before.
// A buffer taken from here can thus be used on any stream at once.  Every access
// holds one lock.  The oldest buffers are freed when the total passes the bound
// and all of them when an allocation fails (which is then tried again);
// dev_mem_info() counts them as free memory.  A buffer is larger than the request
// by at most an eighth.  A device reset by the application leaves dangling
// addresses: the context's identifier is compared on every access and buffers of
// an earlier context are forgotten.
#include <cuda.h>

#include <iterator>
#include <list>
#include <map>
#include <mutex>

#include "qmb_common.cuh"

namespace qmb {
namespace {

constexpr size_t kMaxBlock = (size_t)128 << 20;
constexpr size_t kMaxTotal = (size_t)512 << 20;
constexpr int kMaxDevices = 64;

struct Kept {
    void* p;
    size_t bytes;
};
using KeptList = std::list<Kept>;
struct DeviceCache {
    KeptList kept;                                      // oldest first
    std::multimap<size_t, KeptList::iterator> by_size;  // newest last among equals
    size_t total = 0;
    unsigned long long ctx = 0;
};

std::mutex g_mu;
// never destroyed: handles may be released while the process exits
DeviceCache* caches() {
    static DeviceCache* c = new DeviceCache[kMaxDevices];
    return c;
}

// Identifier of the current context, unique in the process (0: unknown).
unsigned long long context_id() {
    using Fn = CUresult (*)(CUcontext, unsigned long long*);
    static Fn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Fn>(f);
    }();
    unsigned long long id = 0;
    if (!fn || fn(nullptr, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// The current device's cache, or null where nothing may be kept.
DeviceCache* current(int dev) {
    if (dev < 0 || dev >= kMaxDevices) return nullptr;
    const unsigned long long id = context_id();
    if (id == 0) return nullptr;
    DeviceCache& c = caches()[dev];
    if (c.ctx != id) {
        c.kept.clear();
        c.by_size.clear();
        c.total = 0;
        c.ctx = id;
    }
    return &c;
}

void* take(DeviceCache& c, std::multimap<size_t, KeptList::iterator>::iterator at) {
    void* p = at->second->p;
    c.total -= at->first;
    c.kept.erase(at->second);
    c.by_size.erase(at);
    return p;
}

void drop(DeviceCache& c, size_t keep) {
    while (c.total > keep && !c.kept.empty()) {
        auto range = c.by_size.equal_range(c.kept.front().bytes);
        for (auto it = range.first; it != range.second; ++it)
            if (it->second == c.kept.begin()) {
                cudaFree(take(c, it));
                break;
            }
    }
}

size_t rounded(size_t bytes) {
    const size_t unit = bytes >= ((size_t)1 << 20) ? (size_t)2 << 20 : 512;
    return (bytes + unit - 1) / unit * unit;
}

}  // namespace

void* dev_alloc(size_t bytes, size_t* got, int* dev_out) {
    int dev = -1;
    QMB_CUDA_TRY(cudaGetDevice(&dev));
    *dev_out = dev;
    const size_t want = rounded(bytes);
    *got = want;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (DeviceCache* c = want <= kMaxBlock ? current(dev) : nullptr) {
            auto it = c->by_size.lower_bound(want);
            if (it != c->by_size.end() && it->first <= want + want / 8) {
                *got = it->first;
                return take(*c, it);
            }
        }
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, want);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        dev_trim();
        e = cudaMalloc(&p, want);
    }
    if (e != cudaSuccess)
        throw Error{e == cudaErrorMemoryAllocation ? QMB_ERR_NOMEM : QMB_ERR_CUDA,
                    std::string("cudaMalloc of ") + std::to_string(want) + " bytes: " + cudaGetErrorString(e)};
    return p;
}

void dev_free(void* p, size_t bytes, int dev, bool idle) {
    if (!p) return;
    int cur = -1;
    if (idle && bytes <= kMaxBlock && cudaGetDevice(&cur) == cudaSuccess && cur == dev) {
        std::lock_guard<std::mutex> lock(g_mu);
        if (DeviceCache* c = current(dev)) {
            c->kept.push_back(Kept{p, bytes});
            c->by_size.emplace(bytes, std::prev(c->kept.end()));
            c->total += bytes;
            drop(*c, kMaxTotal);
            return;
        }
    }
    cudaFree(p);
}

void dev_trim() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    std::lock_guard<std::mutex> lock(g_mu);
    if (DeviceCache* c = current(dev)) drop(*c, 0);
}

bool dev_mem_info(size_t* free_bytes, size_t* total) {
    if (cudaMemGetInfo(free_bytes, total) != cudaSuccess) {
        (void)cudaGetLastError();
        *free_bytes = *total = 0;
        return false;
    }
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return true;
    std::lock_guard<std::mutex> lock(g_mu);
    if (DeviceCache* c = current(dev)) *free_bytes += c->total;
    return true;
}

}  // namespace qmb
