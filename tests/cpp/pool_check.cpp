// The pool of device buffers (qmb_mem.cu) over a stand-in for the CUDA calls that
// it makes: contexts that are reset or changed, frees
// that are refused.  Host code only.  Prints one
// line "<case> ok" or "<case> FAILED <condition>" per case.
#include <cstdio>
#include <map>
#include <set>
#include <vector>

#include "../../qmbcuda_b200/csrc/qmb_mem.cu"

// ------------------------------------------------------------- stand-in
namespace fake {
unsigned long long ctx = 1, last_ctx = 1;       // the current context
std::set<unsigned long long> live_ctx = {1};
std::map<uintptr_t, unsigned long long> owner;  // live allocations
uintptr_t base = 0x10000000;                    // the first address tried
int mallocs = 0, frees = 0, bad_frees = 0;
bool refuse = false;                            // as while a thread captures a graph

// a reset: the context and its memory are gone, the next one starts at the same addresses
void reset() {
    for (auto it = owner.begin(); it != owner.end();) it = it->second == ctx ? owner.erase(it) : std::next(it);
    live_ctx.erase(ctx);
    live_ctx.insert(ctx = ++last_ctx);
}
// another context beside the present ones, made current
unsigned long long make() {
    live_ctx.insert(ctx = ++last_ctx);
    return ctx;
}
unsigned long long owner_of(const void* p) {
    const auto it = owner.find((uintptr_t)p);
    return it == owner.end() ? 0 : it->second;
}
CUresult ctx_get_id(CUcontext c, unsigned long long* id) {
    *id = c ? (unsigned long long)(uintptr_t)c : ctx;
    return live_ctx.count(*id) ? CUDA_SUCCESS : CUDA_ERROR_CONTEXT_IS_DESTROYED;
}
CUresult pointer_attribute(void* out, CUpointer_attribute, CUdeviceptr p) {
    const unsigned long long o = owner_of((const void*)(uintptr_t)p);
    if (!o) return CUDA_ERROR_INVALID_VALUE;
    *static_cast<CUcontext*>(out) = reinterpret_cast<CUcontext>((uintptr_t)o);
    return CUDA_SUCCESS;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) {
    uintptr_t a = fake::base;
    while (fake::owner.count(a)) a += 0x10000000;
    fake::owner[a] = fake::ctx;
    *p = (void*)a;
    ++fake::mallocs;
    (void)bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (fake::refuse) return cudaErrorStreamCaptureUnsupported;
    if (!fake::owner.erase((uintptr_t)p)) {
        ++fake::bad_frees;
        return cudaErrorInvalidValue;
    }
    ++fake::frees;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = *t = (size_t)1 << 30;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long,
                                    enum cudaDriverEntryPointQueryResult* q) {
    const std::string n = name;
    *f = n == "cuCtxGetId" ? (void*)fake::ctx_get_id : n == "cuPointerGetAttribute" ? (void*)fake::pointer_attribute : nullptr;
    *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}

// ---------------------------------------------------------------- cases
using Buf = qmb::DevBuf<unsigned char>;
static const char* g_case = "";
static bool g_ok = true;
#define EXPECT(c)                                    \
    do {                                             \
        if (!(c) && g_ok) {                          \
            std::printf("%s FAILED %s\n", g_case, #c); \
            g_ok = false;                            \
        }                                            \
    } while (0)

static void reuse() {
    Buf a(1000);
    void* p = a.p;
    a.mark_idle();
    a.release();
    Buf b(1000);
    EXPECT(b.p == p);
    Buf c(1000);
    EXPECT(c.p != p);
}

// a buffer made before a reset and released after it: never handed out, and the
// new context's buffer at the same address stays allocated
static void released_after_reset() {
    for (bool idle : {true, false}) {
        Buf old(3000);
        unsigned char* dead = old.p;
        fake::reset();
        Buf live(3000);
        EXPECT(live.p == dead);  // the stand-in gives the same address again
        if (idle) old.mark_idle();
        old.release();
        EXPECT(fake::owner_of(live.p) == fake::ctx);
        Buf next(3000);
        EXPECT(next.p != live.p);
        EXPECT(fake::owner_of(next.p) == fake::ctx);
    }
    EXPECT(fake::bad_frees == 0);
}

// a buffer kept before a reset is forgotten
static void kept_before_reset() {
    Buf a(5000);
    a.mark_idle();
    a.release();
    size_t f0 = 0, t = 0, f1 = 0;
    qmb::dev_mem_info(&f0, &t);
    fake::reset();
    qmb::dev_mem_info(&f1, &t);
    EXPECT(f1 < f0);
    const int m = fake::mallocs;
    Buf b(5000);
    EXPECT(fake::mallocs == m + 1);
    EXPECT(fake::owner_of(b.p) == fake::ctx);
}

// two live contexts: each hands out its own buffers, and nothing is lost when the
// current one changes
static void two_contexts() {
    const unsigned long long c1 = fake::ctx;
    Buf a(7000);
    unsigned char* pa = a.p;
    a.mark_idle();
    a.release();
    const unsigned long long c2 = fake::make();
    {
        Buf b(7000);
        EXPECT(b.p != pa);
        EXPECT(fake::owner_of(b.p) == c2);
    }
    fake::ctx = c1;
    Buf again(7000);
    EXPECT(again.p == pa);
    // released while the other context is current: freed, not kept there
    again.mark_idle();
    fake::ctx = c2;
    again.release();
    EXPECT(fake::owner_of(pa) == 0);
    Buf d(7000);
    EXPECT(fake::owner_of(d.p) == c2);
    EXPECT(fake::bad_frees == 0);
}

// the shape of the library's handles
struct Handle {
    Buf flag{900}, a{9000}, b{90000};
    ~Handle() { qmb::mark_idle_after_wait(flag, a, b); }
};

// a handle's buffers are handed out again only when the device was waited for
static void refused_free() {
    std::set<void*> first;
    {
        Handle h;
        first = {h.a.p, h.b.p};
    }
    {
        Handle h;
        EXPECT(first.count(h.a.p) && first.count(h.b.p));
        fake::refuse = true;
    }
    fake::refuse = false;
    Handle h;
    EXPECT(!first.count(h.a.p) && !first.count(h.b.p));
}

// what is kept goes back to the driver, what is in use stays
static void trim() {
    Buf used(100), a(100), b(1 << 20);
    void *pa = a.p, *pb = b.p;
    qmb::mark_idle(a, b);
    a.release();
    b.release();
    EXPECT(fake::owner_of(pa) && fake::owner_of(pb));
    qmb::dev_trim();
    EXPECT(!fake::owner_of(pa) && !fake::owner_of(pb) && fake::owner_of(used.p));
    size_t f = 0, t = 0;
    qmb::dev_mem_info(&f, &t);
    EXPECT(f == t);
}

int main() {
    const struct {
        const char* name;
        void (*f)();
    } cases[] = {{"reuse", reuse},
                 {"released_after_reset", released_after_reset},
                 {"kept_before_reset", kept_before_reset},
                 {"two_contexts", two_contexts},
                 {"refused_free", refused_free},
                 {"trim", trim}};
    for (const auto& c : cases) {
        g_case = c.name;
        g_ok = true;
        fake::bad_frees = 0;
        c.f();
        if (g_ok) std::printf("%s ok\n", c.name);
    }
    return 0;
}
