// ppf_common.cuh -- shared device helpers of libppf (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <mutex>
#include <utility>

namespace ppf {

template <typename T>
struct __align__(2 * sizeof(T)) cx {
    T x, y;
};

template <typename T> __device__ __forceinline__ cx<T> mk(T a, T b) { cx<T> r; r.x = a; r.y = b; return r; }
template <typename T> __device__ __forceinline__ cx<T> operator+(cx<T> a, cx<T> b) { return mk(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ cx<T> operator-(cx<T> a, cx<T> b) { return mk(a.x - b.x, a.y - b.y); }
template <typename T> __device__ __forceinline__ cx<T> operator*(cx<T> a, T s) { return mk(a.x * s, a.y * s); }
template <typename T> __device__ __forceinline__ cx<T> cmul(cx<T> a, cx<T> b)
{
    return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T> __device__ __forceinline__ cx<T> conj(cx<T> a) { return mk(a.x, -a.y); }
// multiply by -i (forward) or +i (inverse)
template <typename T, bool INV> __device__ __forceinline__ cx<T> mul_mi(cx<T> a)
{
    return INV ? mk(-a.y, a.x) : mk(a.y, -a.x);
}

template <typename T> __device__ __forceinline__ cx<T> ldg(const cx<T>* p) { return *p; }
template <> __device__ __forceinline__ cx<double> ldg(const cx<double>* p)
{
    double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return mk(v.x, v.y);
}
template <> __device__ __forceinline__ cx<float> ldg(const cx<float>* p)
{
    float2 v = __ldg(reinterpret_cast<const float2*>(p));
    return mk(v.x, v.y);
}

// Complex elements per 128-byte bank row of shared memory, the width of the
// tiles' line-index swizzle (sidx_ct)
template <typename T> struct SwizzleG { static constexpr int value = 128 / (int)sizeof(cx<T>); };

// Asynchronous global -> shared copies (cp.async): one element per call,
// completion tracked per thread by commit groups.
__device__ __forceinline__ void cp_async_elem(float* dst, const float* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_elem(cx<float>* dst, const cx<float>* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_f64(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_elem(cx<double>* dst, const cx<double>* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
// 16 bytes, both addresses 16-byte aligned
__device__ __forceinline__ void cp_async_16(void* dst, const void* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// wait until at most N of this thread's most recent groups are pending
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Bulk prefetch of `bytes` (a multiple of 16) at a 16-byte aligned global
// address into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}

// Programmatic dependent launch: a solve's kernels on one stream are launched
// with this allowed, so that the next kernel's blocks are resident and past
// their launch latency when the previous kernel ends.  Every such kernel
// begins with pdl_enter(): it waits for the whole previous kernel (and so,
// each having waited for its own, for all before it) before it touches
// memory, then lets the next kernel's blocks in.  Without the launch
// attribute both instructions do nothing.  A solve's first launch waits for
// its predecessor as usual, and its last kernel only waits (pdl_wait): what
// runs before and after a solve sees ordinary stream order.  What a kernel of
// the solve wrote (spectra, flags, scalars, partial sums) changes while the
// next one is already resident, so it is read by ordinary loads through
// pointers without const __restrict__, which would allow the read-only path
// and loads moved above the wait; the caller's arrays, twiddles, eigenvalues
// and the iterate of a sweep (ld_pair_al) keep it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_enter()
{
    pdl_wait();
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// the stream of a launch, and whether the launch may overlap the end of the
// previous kernel on it (which must then be followed by nothing but kernels
// that begin with pdl_enter)
struct LStream {
    cudaStream_t s;
    bool pdl;
    LStream(cudaStream_t st = nullptr, bool p = false) : s(st), pdl(p) {}
    operator cudaStream_t() const { return s; }
};

template <typename... P, typename... A>
inline cudaError_t launch_on(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, const LStream& st, A&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st.s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = st.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// SMs of the current device
inline cudaError_t device_sms(int* sms)
{
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) : e;
}

// Opt a kernel into `bytes` of dynamic shared memory.  The limit belongs to
// the function, not to a launch, so every host thread shares it: set to each
// call's size, it could be lowered by a smaller call on another thread between
// this call's setting and its launch, which is then refused.  It is therefore
// only ever set to one value and left alone where the 48 KB default (which
// covers static arrays too) is enough: to the most a block of the kernel can
// have on the device.
inline cudaError_t set_smem_most(const void* fn, size_t bytes)
{
    struct Size { size_t free, most; };   // without the limit set, and at most
    static std::map<std::pair<const void*, int>, Size> sizes;
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    Size s{ 0, 0 };
    {
        std::lock_guard<std::mutex> lk(mu);
        const auto it = sizes.find({ fn, dev });
        if (it != sizes.end()) s = it->second;
    }
    if (s.most == 0) {
        int def = 0, optin = 0;
        cudaFuncAttributes at{};
        e = cudaDeviceGetAttribute(&def, cudaDevAttrMaxSharedMemoryPerBlock, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, fn);
        if (e != cudaSuccess) return e;
        s = Size{ (size_t)def - at.sharedSizeBytes, (size_t)optin - at.sharedSizeBytes };
        std::lock_guard<std::mutex> lk(mu);
        sizes[{ fn, dev }] = s;
    }
    if (bytes <= s.free) return cudaSuccess;
    if (bytes > s.most) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.most);
}
template <typename K>
cudaError_t set_smem(K kern, size_t bytes)
{
    return set_smem_most(reinterpret_cast<const void*>(kern), bytes);
}
// Per-axis FFT schedule: complex length n = prod(radix[0..npass)).
struct FftSched {
    int n;
    int npass;
    int radix[12];
    int w;    // lines per tile of the run-time engine (0: default width)
    int rt;   // 1: run-time engine even where a compile-time shape exists
    // fast_div multipliers of the run-time engine: n, n/2 + 1, and the
    // product of the radices before each pass
    unsigned mg_n, mg_np, mg_ns[12];
};

// e / d of small non-negative integers (e d < 2^32) by one multiplication,
// m = div_magic(d)
inline unsigned div_magic(unsigned d) { return d < 2 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }
__device__ __forceinline__ int fast_div(int e, unsigned m) { return m ? (int)__umulhi((unsigned)e, m) : e; }

}  // namespace ppf
