// qmb_mem.cu -- device memory of the library's buffers (DevBuf).
//
// A sector, a matrix and a solve each take and free ten to thirty buffers, and
// cudaMalloc and cudaFree cost 0.1 to 0.3 ms each for the larger ones: at 28
// sites they were 9 of the 13 ms of building a sector and its matrix (its
// kernels take 2.5 ms).  Freed buffers of up to kMaxBlock bytes are therefore
// kept, at most kMaxTotal bytes a context, and handed out again.
//
// Rules.  A buffer comes here only idle: no work on any stream may still use
// it.  DevBuf::mark_idle() says so, and is called after the wait that ends a
// solve or a build, or on a handle's buffers once the first of them went through
// cudaFree, which waits for the device, and was not refused
// (mark_idle_after_wait); every other buffer is freed.
// A buffer taken from here can thus be used on any stream at once.  Every access
// holds one lock.  The oldest buffers are freed when the total passes the bound
// and all of them when an allocation fails (which is then tried again);
// dev_mem_info() counts them as free memory, and qmb_trim() gives them back.  Requests
// are rounded up to 512 bytes, from 1 MB on to 2 MB; a buffer is larger than the rounded
// request by at most an eighth.
//
// A buffer belongs to the context in which it was allocated (DevBuf keeps its
// identifier, unique in the process) and is kept and handed out in that context
// alone.  One released while another context is current is freed, or forgotten
// when its own context is gone: after a device reset its address may belong to a
// live buffer of the new context.
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

struct Kept {
    void* p;
    size_t bytes;
};
using KeptList = std::list<Kept>;
struct Cache {
    KeptList kept;                                      // oldest first
    std::multimap<size_t, KeptList::iterator> by_size;  // newest last among equals
    size_t total = 0;
};

std::mutex g_mu;
// by context; never destroyed: handles may be released while the process exits
std::map<unsigned long long, Cache>& caches() {
    static auto* c = new std::map<unsigned long long, Cache>;
    return *c;
}

// A driver function by name, or null.
template <class Fn>
Fn driver_fn(const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        f = nullptr;
    }
    return reinterpret_cast<Fn>(f);
}

// Identifier of a context (null: the current one), 0 when unknown.
unsigned long long context_id(CUcontext c = nullptr) {
    static const auto fn = driver_fn<CUresult (*)(CUcontext, unsigned long long*)>("cuCtxGetId");
    unsigned long long id = 0;
    if (!fn || fn(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Identifier of the context that the memory at p belongs to now, 0 for none.
unsigned long long owner_id(void* p) {
    static const auto fn =
        driver_fn<CUresult (*)(void*, CUpointer_attribute, CUdeviceptr)>("cuPointerGetAttribute");
    CUcontext c = nullptr;
    if (!fn || fn(&c, CU_POINTER_ATTRIBUTE_CONTEXT, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS || !c) return 0;
    return context_id(c);
}

void* take(Cache& c, std::multimap<size_t, KeptList::iterator>::iterator at) {
    void* p = at->second->p;
    c.total -= at->first;
    c.kept.erase(at->second);
    c.by_size.erase(at);
    return p;
}

void drop(Cache& c, size_t keep) {
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

void* dev_alloc(size_t bytes, size_t* got, DevPlace* at) {
    QMB_CUDA_TRY(cudaGetDevice(&at->dev));
    at->ctx = context_id();
    const size_t want = rounded(bytes);
    *got = want;
    if (want <= kMaxBlock && at->ctx) {
        std::lock_guard<std::mutex> lock(g_mu);
        Cache& c = caches()[at->ctx];
        auto it = c.by_size.lower_bound(want);
        if (it != c.by_size.end() && it->first <= want + want / 8) {
            *got = it->first;
            return take(c, it);
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
    if (!at->ctx) at->ctx = context_id();  // (the first allocation of a process makes the context)
    return p;
}

bool dev_free(void* p, size_t bytes, const DevPlace& at, bool idle) {
    if (!p) return false;
    const unsigned long long id = at.ctx ? context_id() : 0;
    if (at.ctx && id != at.ctx) {
        if (owner_id(p) == at.ctx) cudaFree(p);
        return false;
    }
    if (idle && bytes <= kMaxBlock && id) {
        std::lock_guard<std::mutex> lock(g_mu);
        Cache& c = caches()[id];
        c.kept.push_back(Kept{p, bytes});
        c.by_size.emplace(bytes, std::prev(c.kept.end()));
        c.total += bytes;
        drop(c, kMaxTotal);
        return false;
    }
    if (cudaFree(p) == cudaSuccess) return true;
    (void)cudaGetLastError();
    return false;
}

void dev_trim() {
    const unsigned long long id = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = caches().find(id);
    if (it != caches().end()) drop(it->second, 0);
}

bool dev_mem_info(size_t* free_bytes, size_t* total) {
    if (cudaMemGetInfo(free_bytes, total) != cudaSuccess) {
        (void)cudaGetLastError();
        *free_bytes = *total = 0;
        return false;
    }
    const unsigned long long id = context_id();
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = caches().find(id);
    if (it != caches().end()) *free_bytes += it->second.total;
    return true;
}

}  // namespace qmb
