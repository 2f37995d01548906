// cpdlp_common.cuh -- shared infrastructure of libcoolpdlp_cuda (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <thread>
#include <utility>
#include <vector>
#include <vector>

#include "../../include/coolpdlp_cuda.h"
#include "host_parallel.h"

namespace cpdlp {

// ---------------------------------------------------------------------------
// errors: every internal failure is a cpdlp::Error carrying a CPDLP_ERR_* code;
// the C-ABI layer turns it into a status and cpdlp_last_error().
// ---------------------------------------------------------------------------
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] inline void fail(int code, const std::string& msg) { throw Error(code, msg); }

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
    if (e != cudaSuccess) {
        char buf[512];
        snprintf(buf, sizeof(buf), "%s failed at %s:%d: %s", what, file, line,
                 cudaGetErrorString(e));
        if (e == cudaErrorMemoryAllocation) fail(CPDLP_ERR_OUT_OF_MEMORY, buf);
        fail(CPDLP_ERR_CUDA, buf);
    }
}
#define CK(x) ::cpdlp::cuda_check((x), #x, __FILE__, __LINE__)
#define CK_LAUNCH() ::cpdlp::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__)

// ---------------------------------------------------------------------------
// device buffer (owning, move-only), stream-ordered: allocated with
// cudaMallocAsync on the calling thread's current allocation stream and freed
// with cudaFreeAsync on the same stream, so that creating or dropping buffers
// never waits for kernels running on other streams (a plain cudaFree would
// synchronise the device, stalling every batch in flight).  Buffers must be
// released before the stream they were allocated on is destroyed.
// ---------------------------------------------------------------------------
inline cudaStream_t& alloc_stream() {
    static thread_local cudaStream_t s = nullptr;
    return s;
}
struct AllocScope {
    cudaStream_t prev;
    explicit AllocScope(cudaStream_t s) : prev(alloc_stream()) { alloc_stream() = s; }
    ~AllocScope() { alloc_stream() = prev; }
    AllocScope(const AllocScope&) = delete;
    AllocScope& operator=(const AllocScope&) = delete;
};

template <class T>
struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;
    DBuf() = default;
    explicit DBuf(size_t count) { alloc(count); }
    DBuf(const DBuf&) = delete;
    DBuf& operator=(const DBuf&) = delete;
    DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), s(o.s) { o.p = nullptr; o.n = 0; }
    DBuf& operator=(DBuf&& o) noexcept {
        if (this != &o) { release(); p = o.p; n = o.n; s = o.s; o.p = nullptr; o.n = 0; }
        return *this;
    }
    ~DBuf() { release(); }
    void alloc(size_t count) {
        release();
        n = count;
        s = alloc_stream();
        if (count) CK(cudaMallocAsync((void**)&p, sizeof(T) * count, s));
    }
    void release() {
        if (p) cudaFreeAsync(p, s);
        p = nullptr;
        n = 0;
    }
    size_t bytes() const { return sizeof(T) * n; }
    T* get() const { return p; }
};

// ---------------------------------------------------------------------------
// scalar semantics shared by host and device (src/utils/linalg.jl:1-53)
// Base.max/min on floats: NaN propagates and -0.0 < +0.0.
// ---------------------------------------------------------------------------
// On the device: FP32 is one instruction (max.NaN orders -0 below +0 too).
// FP64 compares bit patterns as integers, because a comparison on GB300's FP64
// pipe (1.9 lanes a clock and SM) costs as much as an addition and a projection
// onto a box has six: they were 6 of a primal row's 14 FP64 operations.
template <class T>
__host__ __device__ __forceinline__ T jl_max(T x, T y) {
    bool sx = signbit(x), sy = signbit(y);
    if ((y > x) || (sy < sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
}
template <class T>
__host__ __device__ __forceinline__ T jl_min(T x, T y) {
    bool sx = signbit(x), sy = signbit(y);
    if ((y < x) || (sy > sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
}
#ifdef __CUDACC__
// order-preserving integer of a double (-0 just below +0; NaNs outside the infinities)
__device__ __forceinline__ long long f64_key(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}
__device__ __forceinline__ bool f64_is_nan(double x) {
    return (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
#endif
template <>
__host__ __device__ __forceinline__ float jl_max<float>(float x, float y) {
#ifdef __CUDA_ARCH__
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
#else
    bool sx = std::signbit(x), sy = std::signbit(y);
    if ((y > x) || (sy < sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
#endif
}
template <>
__host__ __device__ __forceinline__ float jl_min<float>(float x, float y) {
#ifdef __CUDA_ARCH__
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
#else
    bool sx = std::signbit(x), sy = std::signbit(y);
    if ((y < x) || (sy > sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
#endif
}
template <>
__host__ __device__ __forceinline__ double jl_max<double>(double x, double y) {
#ifdef __CUDA_ARCH__
    const double r = f64_key(y) > f64_key(x) ? y : x;
    return f64_is_nan(x) ? x : f64_is_nan(y) ? y : r;
#else
    bool sx = std::signbit(x), sy = std::signbit(y);
    if ((y > x) || (sy < sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
#endif
}
template <>
__host__ __device__ __forceinline__ double jl_min<double>(double x, double y) {
#ifdef __CUDA_ARCH__
    const double r = f64_key(y) < f64_key(x) ? y : x;
    return f64_is_nan(x) ? x : f64_is_nan(y) ? y : r;
#else
    bool sx = std::signbit(x), sy = std::signbit(y);
    if ((y < x) || (sy > sx)) return (x != x) ? x : y;
    return (y != y) ? y : x;
#endif
}
template <class T>
__host__ __device__ __forceinline__ T proj_box(T x, T l, T u) { return jl_min(u, jl_max(l, x)); }
template <class T>
__host__ __device__ __forceinline__ T pos_part(T a) { return jl_max(a, T(0)); }
template <class T>
__host__ __device__ __forceinline__ T neg_part(T a) { return -jl_min(a, T(0)); }
template <class T>
__host__ __device__ __forceinline__ T safeprod_left(T l, T r) { return isinf(l) ? r : l * r; }
template <class T>
__host__ __device__ __forceinline__ T proj_multiplier(T lam, T l, T u) {
    bool lmin = (l == -INFINITY), umax = (u == INFINITY);
    if (lmin) return umax ? T(0) : -neg_part(lam);
    return umax ? pos_part(lam) : lam;
}
template <class T>
__host__ __device__ __forceinline__ T combine(T l, T u) {
    T ls = isfinite(l) ? fabs(l) : T(0);
    T us = isfinite(u) ? fabs(u) : T(0);
    return jl_max(jl_max(T(0), ls), us);
}

// Exact IEEE products/sums without contraction into FMA, so that sequential
// sums match the Float64 reference operation by operation.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

// a*b + c: rounded twice in FP32 (as the reference's sequence of operations),
// once in FP64, where the number of operations is what steps cost
__device__ __forceinline__ float mul_add(float a, float b, float c) { return add_rn(mul_rn(a, b), c); }
__device__ __forceinline__ double mul_add(double a, double b, double c) { return __fma_rn(a, b, c); }
// 2x - y: doubling is exact, so one fused operation rounds like the product
// and the difference do
__device__ __forceinline__ double extrapolate(double x, double y) { return __fma_rn(2.0, x, -y); }
__device__ __forceinline__ float extrapolate(float x, float y) { return __fmaf_rn(2.0f, x, -y); }

// Scalar loads as volatile PTX: volatile asm statements keep their relative
// order, so loads meant to be in flight together (prefetches) are issued
// before the code that consumes them instead of being sunk to their use.
// ld_stream: read once per pass (evict-first); ld_keep: read-only data that
// other kernels of the same step re-read (normal L2 policy).
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_stream(const double* p) {
    double v;
    asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_keep(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_keep(const double* p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ld_keep(const int* p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// ---------------------------------------------------------------------------
// Programmatic dependent launch of the step kernels in their graphs: a kernel
// starts while the one before it drains, loads what no kernel of the chain
// writes (matrix, bounds, costs), and waits for the one before it to complete
// before it touches anything else.  A kernel lets the next one start only after
// its own wait, so at most two kernels of a chain overlap.  Both instructions
// do nothing in a launch without the attribute.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// set while a step graph is captured
inline bool& chain_launches() {
    static thread_local bool on = false;
    return on;
}
// Whether a step kernel of `threads` threads over `value_bytes` values (0: narrow
// storage) starts early.  FP32 kernels of more than 200,000 threads do not: the
// early blocks' entries displace what the running kernel gathers (a step of
// 1,000,000 nonzeros 14.0 us without, 16.6 us with; the 24M power-law LP 214
// and 218 us).  All others gain: FP32 200,000 nonzeros 7.6 -> 5.9 us, FP64 25,000
// 8.4 -> 6.6, 1,000,000 20.7 -> 18.8, 2,000,000 41.2 -> 38.0 us, the 256 x 256 flow
// LP (narrow, 12.5M nonzeros) 300 steps with checks 21.2 -> 20.3 ms.
inline bool chain_this(int64_t threads, int value_bytes) {
    return chain_launches() && (value_bytes != 4 || threads <= 200000);
}
template <class... P, class... A>
void launch_chained(void (*kern)(P...), unsigned grid, unsigned block, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CK(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

// ---------------------------------------------------------------------------
// handle
// ---------------------------------------------------------------------------
struct Handle {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string last_error;
    int num_sms = 0;
    // error history of the last cpdlp_solve on this handle (every phase of a
    // mixed-precision solve, passes counted from the start of the solve)
    std::vector<int64_t> solve_hist_passes;
    std::vector<cpdlp_kkt_errors> solve_hist_err;
    // reusable small host-pinned area for reductions read back each check
    double* pinned = nullptr;
    size_t pinned_bytes = 0;
    double* pinned_area(size_t bytes) {
        if (bytes > pinned_bytes) {
            if (pinned) cudaFreeHost(pinned);
            pinned = nullptr;
            pinned_bytes = 0;
            CK(cudaMallocHost((void**)&pinned, bytes));
            pinned_bytes = bytes;
        }
        return pinned;
    }
    // Reusable blocks of mapped, page-locked host memory that kernels write
    // results into while they run.  Blocks are returned to the pool instead of
    // freed, because freeing page-locked memory waits for the whole device.
    struct HostBlock {
        void* p;
        size_t bytes;
        bool used;
    };
    std::vector<HostBlock> host_blocks;
    void* host_get(size_t bytes) {
        int best = -1;
        for (size_t i = 0; i < host_blocks.size(); i++) {
            const HostBlock& b = host_blocks[i];
            if (!b.used && b.bytes >= bytes && (best < 0 || b.bytes < host_blocks[best].bytes))
                best = (int)i;
        }
        if (best >= 0) {
            host_blocks[best].used = true;
            return host_blocks[best].p;
        }
        void* p = nullptr;
        const size_t sz = std::max<size_t>(bytes, 1 << 16);
        CK(cudaHostAlloc(&p, sz, cudaHostAllocMapped | cudaHostAllocPortable));
        host_blocks.push_back(HostBlock{p, sz, true});
        return p;
    }
    void host_put(void* p) {
        for (HostBlock& b : host_blocks)
            if (b.p == p) b.used = false;
    }
    void host_release_all() {
        for (HostBlock& b : host_blocks) cudaFreeHost(b.p);
        host_blocks.clear();
    }
};

inline unsigned grid_for(int64_t items, int threads, int64_t cap = 1 << 30) {
    int64_t g = (items + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

// wall clock (seconds)
double now_seconds();

}  // namespace cpdlp
