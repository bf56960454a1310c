// qmb_common.cuh -- shared device/host helpers of libqmb_b200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <utility>
#include <vector>

#include "qmb_b200.h"

namespace qmb {

// ------------------------------------------------------------------ errors
void set_error(const std::string& msg);
qmb_status fail(qmb_status s, const std::string& msg);

struct Error {
    qmb_status code;
    std::string msg;
};

#define QMB_CUDA_TRY(expr)                                                                   \
    do {                                                                                     \
        cudaError_t _e = (expr);                                                             \
        if (_e != cudaSuccess)                                                               \
            throw ::qmb::Error{_e == cudaErrorMemoryAllocation ? QMB_ERR_NOMEM : QMB_ERR_CUDA, \
                               std::string(#expr) + ": " + cudaGetErrorString(_e)};          \
    } while (0)

#define QMB_REQUIRE(cond, code, msg)                 \
    do {                                             \
        if (!(cond)) throw ::qmb::Error{code, msg};  \
    } while (0)

// Runs f, converting exceptions into a status.
template <class F>
qmb_status guarded(F&& f) {
    try {
        f();
        return QMB_OK;
    } catch (const Error& e) {
        return fail(e.code, e.msg);
    } catch (const std::bad_alloc&) {
        return fail(QMB_ERR_NOMEM, "host allocation failed");
    } catch (const std::exception& e) {
        return fail(QMB_ERR_INVALID, e.what());
    }
}

// ------------------------------------------------------------ device memory
// qmb_mem.cu: device memory, with freed idle buffers kept for reuse.
struct DevPlace {
    int dev = -1;
    unsigned long long ctx = 0;  // identifier of the context (0: unknown)
};
void* dev_alloc(size_t bytes, size_t* got, DevPlace* at);
// True when the memory went through cudaFree without an error, which waits for
// the device first (measured on 256 bytes with work on a non-blocking stream).
bool dev_free(void* p, size_t bytes, const DevPlace& at, bool idle);
void dev_trim();  // frees what is kept in the current context
bool dev_mem_info(size_t* free_bytes, size_t* total);  // cudaMemGetInfo, kept buffers counted as free

template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    explicit DevBuf(size_t count) { alloc(count); }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept { swap(o); }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this != &o) { release(); swap(o); }
        return *this;
    }
    ~DevBuf() { release(); }
    void alloc(size_t count) {
        release();
        if (count == 0) count = 1;
        p = static_cast<T*>(dev_alloc(count * sizeof(T), &bytes_, &at_));
        n = count;
    }
    bool release() {  // as dev_free
        const bool freed = dev_free(p, bytes_, at_, idle_);
        p = nullptr;
        n = 0;
        idle_ = false;
        return freed;
    }
    // No work on any stream uses the buffer any more: release() may keep it.
    void mark_idle() { idle_ = p != nullptr; }
    void swap(DevBuf& o) noexcept {
        std::swap(p, o.p);
        std::swap(n, o.n);
        std::swap(bytes_, o.bytes_);
        std::swap(at_, o.at_);
        std::swap(idle_, o.idle_);
    }
    void zero(cudaStream_t st = 0) { QMB_CUDA_TRY(cudaMemsetAsync(p, 0, n * sizeof(T), st)); }
    void upload(const T* h, size_t count, cudaStream_t st = 0) {
        QMB_CUDA_TRY(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, st));
    }
    void download(T* h, size_t count, cudaStream_t st = 0) const {
        QMB_CUDA_TRY(cudaMemcpyAsync(h, p, count * sizeof(T), cudaMemcpyDeviceToHost, st));
    }

private:
    size_t bytes_ = 0;   // as allocated
    DevPlace at_;
    bool idle_ = false;
};
// mark_idle() on several buffers
template <class... B>
void mark_idle(B&... b) { (b.mark_idle(), ...); }
// A handle's buffers when it goes: the first is freed, which waits for the device,
// and the others are idle then.  A free is refused while a thread captures a graph
// in global mode; nothing was waited for and the others are freed as if no pool
// were there.  (cudaDeviceSynchronize() would break a capture of any mode in
// another thread.)
template <class T, class... B>
bool mark_idle_after_wait(DevBuf<T>& first, B&... rest) {
    if (!first.release()) return false;
    mark_idle(rest...);
    return true;
}

// Waits for the default stream, where builds run.  (A wait for the whole device would
// break a stream capture in another thread, this library's own among them.)
inline void wait_default_stream() { QMB_CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy)); }

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        int n = 0;
        if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
            throw Error{QMB_ERR_NO_DEVICE, "no CUDA device is visible"};
        QMB_REQUIRE(dev >= 0 && dev < n, QMB_ERR_INVALID, "device ordinal out of range");
        cudaGetDevice(&prev);
        QMB_CUDA_TRY(cudaSetDevice(dev));
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

inline void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{QMB_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)};
}

// ---------------------------------------------------------------- binomials
uint64_t host_binom(int n, int k);

// Next string with the same popcount (Gosper's hack); s != 0.
__host__ __device__ __forceinline__ uint64_t next_comb(uint64_t s) {
    uint64_t c = s & (~s + 1);
    uint64_t r = s + c;
#ifdef __CUDA_ARCH__
    return (((r ^ s) >> 2) >> (__ffsll((long long)c) - 1)) | r;  // c is a power of two
#else
    return (((r ^ s) >> 2) / c) | r;
#endif
}

// ----------------------------------------------------------- group elements
// An element maps bit q to bit perm[q], optionally followed by inversion of
// all L bits.  When every site map is a lattice translation of a torus whose
// rows are W consecutive bits, the map is a rotation of the rows plus a
// rotation inside every row; those run as a few word operations.  Otherwise
// each element uses a table of 16 entries per 4-bit chunk.
struct GroupDev {
    int L;
    int G;           // site maps
    int n_ext;       // G or 2G (with inversion)
    int structured;  // 1: rotations, 0: nibble tables
    int W;           // row width in bits (structured)
    int n_chunks;    // ceil(L/4) (tables)
    uint64_t mask;   // low L bits
    uint64_t row_lo_mask[65];  // unused slots zero; see apply_rot
    const uint8_t* rot_row;    // [G] row rotation (bits, multiple of W)
    const uint8_t* rot_in;     // [G] rotation inside rows (bits)
    const uint64_t* tables;    // [G][n_chunks][16]
};

__device__ __forceinline__ uint64_t rotl_bits(uint64_t x, int r, int L, uint64_t mask) {
    if (r == 0) return x;
    return ((x << r) | (x >> (L - r))) & mask;
}

// Rotation by c bits inside each W-bit row of an L-bit word (L multiple of W).
// lo = bits whose in-row position is < W - c (they move up by c), the rest
// wrap to the bottom of their row.
__device__ __forceinline__ uint64_t rot_rows(uint64_t x, int c, int W, uint64_t lo) {
    if (c == 0) return x;
    return ((x & lo) << c) | ((x & ~lo) >> (W - c));
}

}  // namespace qmb
