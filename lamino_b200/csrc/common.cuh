// Shared helpers for the lamino_b200 CUDA library (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <cufft.h>

#include <cstdint>
#include <stdexcept>
#include <string>

namespace lamino {

// Status codes of the C ABI (mirrored in include/lamino.h).
enum Status : int {
    OK = 0,
    ERR_ARG = 1,
    ERR_OOM = 2,
    ERR_CUDA = 3,
    ERR_CUFFT = 4,
    ERR_TIMEOUT = 5,
    ERR_NONFINITE = 6,
    ERR_STATE = 7,
};

struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};

inline void check_cuda(cudaError_t e, const char *what) {
    if (e != cudaSuccess) {
        int code = (e == cudaErrorMemoryAllocation) ? ERR_OOM : ERR_CUDA;
        throw Error(code, std::string(what) + ": " + cudaGetErrorString(e));
    }
}
inline void check_cufft(cufftResult r, const char *what) {
    if (r != CUFFT_SUCCESS) {
        int code = (r == CUFFT_ALLOC_FAILED) ? ERR_OOM : ERR_CUFFT;
        throw Error(code, std::string(what) + ": cufft error " + std::to_string((int)r));
    }
}
#define LAMINO_CUDA(x) ::lamino::check_cuda((x), #x)
#define LAMINO_CUFFT(x) ::lamino::check_cufft((x), #x)
#define LAMINO_LAUNCH(what) ::lamino::check_cuda(cudaGetLastError(), what)

inline unsigned grid_for(int64_t n, int block, int64_t cap = 148LL * 64) {
    int64_t g = (n + block - 1) / block;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (unsigned)g;
}

// Launches that overlap the end of the kernel before them in the stream
// (programmatic dependent launch): launch_after() lets the kernel's CTAs start once
// every CTA of the one before has called allow_next(); the kernel reads and writes
// nothing of earlier kernels before wait_previous(), which returns when they have
// completed and their writes are visible.  A kernel of either kind may come before
// or after.  wait_previous() waits for the one kernel before; that it stands for all earlier
// ones as well takes a wait in at least one CTA of every kernel launched this way (others
// may return without one, as the empty work items of k_rows_spread do).  Data of the kernel before is read by plain loads (no __restrict__ const,
// no __ldg): the read-only path assumes that nothing writes it while the kernel
// runs, and here the kernel runs before the writes are done.  What is gained is the launch latency between short kernels.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
void launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    LAMINO_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

// Raise a kernel's dynamic shared-memory limit to at least `bytes` (never
// lowers it; safe from several host threads).
void raise_smem_limit(const void *kernel, int bytes);

// Allocation stream of the calling host thread.  When it is set (a server
// worker sets its own stream), DevBuf memory comes from the device's
// stream-ordered pool on that stream and goes back with cudaFreeAsync, so a
// request that starts or finishes never stalls the requests running beside it
// (cudaFree waits for the whole device); small table uploads then go through
// upload()/zero_bytes(), which order them on the same stream.
inline cudaStream_t &alloc_stream() {
    static thread_local cudaStream_t s = nullptr;
    return s;
}
// Pool of the calling thread's stream-ordered allocations (null: the device's
// default pool).
inline cudaMemPool_t &alloc_pool() {
    static thread_local cudaMemPool_t p = nullptr;
    return p;
}
// This library's own pool on the current device, for the buffers of one driver
// call (nothing that outlives the call may be allocated from it): it keeps up to
// kCallPoolKeep bytes between calls, which are given back to the device when an
// allocation of this library fails.  Null if the device has no pools.
constexpr uint64_t kCallPoolKeep = 4ull << 30;
cudaMemPool_t call_pool();
void trim_call_pool();
struct AllocStreamScope {
    cudaStream_t prev;
    cudaMemPool_t prev_pool;
    explicit AllocStreamScope(cudaStream_t s, cudaMemPool_t pool = nullptr) : prev(alloc_stream()), prev_pool(alloc_pool()) {
        alloc_stream() = s;
        alloc_pool() = pool;
    }
    ~AllocStreamScope() {
        alloc_stream() = prev;
        alloc_pool() = prev_pool;
    }
    AllocStreamScope(const AllocStreamScope &) = delete;
    AllocStreamScope &operator=(const AllocStreamScope &) = delete;
};

template <typename T>
void upload(T *dst, const T *src, size_t count) {
    cudaStream_t s = alloc_stream();
    if (s) {
        LAMINO_CUDA(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyHostToDevice, s));
        LAMINO_CUDA(cudaStreamSynchronize(s));  // the host source may go out of scope
    } else {
        LAMINO_CUDA(cudaMemcpy(dst, src, count * sizeof(T), cudaMemcpyHostToDevice));
    }
}
inline void zero_bytes(void *p, size_t bytes) {
    cudaStream_t s = alloc_stream();
    if (s) LAMINO_CUDA(cudaMemsetAsync(p, 0, bytes, s));
    else LAMINO_CUDA(cudaMemset(p, 0, bytes));
}

// Owning device buffer (no copy, movable).
template <typename T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t as = nullptr;  // stream-ordered allocation on this stream, if set
    DevBuf() = default;
    explicit DevBuf(size_t count) { alloc(count); }
    void alloc(size_t count) {
        release();
        if (!count) return;
        as = alloc_stream();
        cudaError_t e = get(count * sizeof(T));
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            trim_call_pool();
            e = get(count * sizeof(T));
        }
        if (e != cudaSuccess) {
            p = nullptr;
            cudaGetLastError();
        }
        LAMINO_CUDA(e);
        n = count;
    }
    cudaError_t get(size_t bytes) {
        if (as && alloc_pool()) return cudaMallocFromPoolAsync((void **)&p, bytes, alloc_pool(), as);
        if (as) return cudaMallocAsync((void **)&p, bytes, as);
        return cudaMalloc((void **)&p, bytes);
    }
    void release() {
        if (p) {
            if (as) cudaFreeAsync(p, as);
            else cudaFree(p);
        }
        p = nullptr;
        n = 0;
        as = nullptr;
    }
    ~DevBuf() { release(); }
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept : p(o.p), n(o.n), as(o.as) { o.p = nullptr; o.n = 0; o.as = nullptr; }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            p = o.p; n = o.n; as = o.as;
            o.p = nullptr; o.n = 0; o.as = nullptr;
        }
        return *this;
    }
    size_t bytes() const { return n * sizeof(T); }
};

// cuFFT plan holder; the work area is a DevBuf (stream-ordered under a worker).
struct FftPlan {
    cufftHandle h = 0;
    bool valid = false;
    DevBuf<char> work;
    FftPlan() = default;
    ~FftPlan() { reset(); }
    FftPlan(const FftPlan &) = delete;
    FftPlan &operator=(const FftPlan &) = delete;
    void reset() {
        if (valid) cufftDestroy(h);
        valid = false;
        work.release();
    }
    // contiguous batched transform of rank 1-3 (cufftPlanMany with default layouts);
    // stride > 0: 1-D transforms of elements `stride` apart, one after another
    void make(int rank, int *n, cufftType type, int batch, int stride = 0) {
        reset();
        LAMINO_CUFFT(cufftCreate(&h));
        valid = true;
        LAMINO_CUFFT(cufftSetAutoAllocation(h, 0));
        size_t ws = 0;
        int *embed = stride ? n : nullptr;
        LAMINO_CUFFT(cufftMakePlanMany(h, rank, n, embed, stride ? stride : 1, stride ? 1 : 0, embed, stride ? stride : 1,
                                       stride ? 1 : 0, type, batch, &ws));
        work.alloc(ws > 0 ? ws : 16);
        LAMINO_CUFFT(cufftSetWorkArea(h, work.p));
    }
};

struct Dims3 {
    int64_t n1, n2, n3;  // n3 fastest
    int64_t size() const { return n1 * n2 * n3; }
};

}  // namespace lamino
