// Stand-in for the CUDA runtime and for the device side of CUDA C++, so that the library's own
// sources (kernels and host code) run on the CPU without a GPU: tests/simt_host.py compiles them with
// this header in cuda_runtime.h's place.
//
// Kernels: a block's threads are fibers of one host thread.  A thread runs until it meets a warp
// collective or a block barrier; warps, and lanes, take their turns in ascending or descending order
// (simt_order), so that code which is right only for some order of what happens in between is found out.
// A block whose threads do not all arrive at the same barrier, or a warp whose lanes do not all arrive
// at the same collective, is recorded (simt_fault).  Blocks run one after another.
// Streams: work is queued and runs, in stream order, only when something waits for it, as late as the
// CUDA runtime may run it; copies from pageable memory are taken when they are issued.
#pragma once
#define __CUDACC__ 1
#define __CUDA_ARCH__ 1000
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <functional>
#include <type_traits>

#define __global__
#define __device__
#define __host__
#define __shared__ static
#define __forceinline__ inline
#define __restrict__ __restrict
#define __launch_bounds__(...)
#define __grid_constant__
#define __align__(n) __attribute__((aligned(n)))

typedef struct CUstream_st* cudaStream_t;
typedef struct CUevent_st* cudaEvent_t;

namespace simt {
struct Dim {
    unsigned x, y, z;
};
struct Thread {
    Dim tid;
};
extern Thread* self;
extern Dim block_idx, grid_dim, block_dim;
void barrier(int line);
int barrier_count(int line, int p);  // how many threads bring p
void named_barrier(int id, int count);
const uint64_t* exchange(int line, uint64_t v);  // the 32 lanes' values
void* dynamic_shared();
long long ticks();  // 4096 per block barrier
bool dropped();  // the running kernel's status words get lost (simt_drop_status)
struct Config {
    unsigned grid, block;
    size_t smem;
    cudaStream_t stream;
};
inline Config config(unsigned long long g, unsigned long long b, size_t m, cudaStream_t s) {
    return Config{(unsigned)g, (unsigned)b, m, s};
}
void queue(const char* name, Config c, std::function<void()> kernel);
template <typename Kernel, typename... Args>
void launch(const char* name, Config c, Kernel k, Args... args) {  // (arguments are taken now)
    queue(name, c, [=]() { k(args...); });
}

template <typename T>
uint64_t to_bits(T v) {
    static_assert(sizeof(T) <= 8, "shuffles of at most 64 bits");
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof(T));
    return b;
}
template <typename T>
T from_bits(uint64_t b) {
    T v;
    std::memcpy(&v, &b, sizeof(T));
    return v;
}
inline unsigned lane() { return self->tid.x & 31u; }
}  // namespace simt

#define threadIdx (simt::self->tid)
#define blockIdx simt::block_idx
#define gridDim simt::grid_dim
#define blockDim simt::block_dim
#define __syncthreads() simt::barrier(__LINE__)
#define __syncthreads_or(p) (simt::barrier_count(__LINE__, (p)) != 0)
#define __syncthreads_count(p) simt::barrier_count(__LINE__, (p))
#define __syncwarp() ((void)simt::exchange(__LINE__, 0))

struct alignas(8) uint2 { unsigned x, y; };
struct alignas(16) uint4 { unsigned x, y, z, w; };
struct alignas(16) int4 { int x, y, z, w; };
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) ulonglong2 { unsigned long long x, y; };
inline uint2 make_uint2(unsigned x, unsigned y) { return {x, y}; }
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }
inline int4 make_int4(int x, int y, int z, int w) { return {x, y, z, w}; }
inline ulonglong2 make_ulonglong2(unsigned long long x, unsigned long long y) { return {x, y}; }

template <typename A, typename B>
constexpr std::common_type_t<A, B> min(A a, B b) {
    using C = std::common_type_t<A, B>;
    return (C)b < (C)a ? (C)b : (C)a;
}
template <typename A, typename B>
constexpr std::common_type_t<A, B> max(A a, B b) {
    using C = std::common_type_t<A, B>;
    return (C)a < (C)b ? (C)b : (C)a;
}
using std::isfinite;

// warp collectives (all 32 lanes)
#define __shfl_sync(m, v, l) simt::from_bits<std::decay_t<decltype(v)>>(simt::exchange(__LINE__, simt::to_bits(v))[(l) & 31])
#define __shfl_xor_sync(m, v, d) \
    simt::from_bits<std::decay_t<decltype(v)>>(simt::exchange(__LINE__, simt::to_bits(v))[(simt::lane() ^ (d)) & 31])
#define __shfl_up_sync(m, v, d) \
    simt::from_bits<std::decay_t<decltype(v)>>(simt::exchange(__LINE__, simt::to_bits(v))[simt::lane() < (unsigned)(d) ? simt::lane() : simt::lane() - (d)])
#define __shfl_down_sync(m, v, d) \
    simt::from_bits<std::decay_t<decltype(v)>>(simt::exchange(__LINE__, simt::to_bits(v))[simt::lane() + (d) > 31u ? simt::lane() : simt::lane() + (d)])
namespace simt {
inline unsigned ballot(int line, bool p) {
    const uint64_t* v = exchange(line, p);
    unsigned m = 0;
    for (int i = 0; i < 32; ++i) m |= (unsigned)(v[i] & 1u) << i;
    return m;
}
inline unsigned reduce_add(int line, unsigned x) {
    const uint64_t* v = exchange(line, x);
    unsigned s = 0;
    for (int i = 0; i < 32; ++i) s += (unsigned)v[i];
    return s;
}
}  // namespace simt
#define __ballot_sync(m, p) simt::ballot(__LINE__, (p))
#define __any_sync(m, p) (simt::ballot(__LINE__, (p)) != 0)
#define __reduce_add_sync(m, v) simt::reduce_add(__LINE__, (v))

// integer and float intrinsics
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __popcll(unsigned long long v) { return __builtin_popcountll(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline unsigned __brev(unsigned v) {
    unsigned r = 0;
    for (int i = 0; i < 32; ++i) r |= ((v >> i) & 1u) << (31 - i);
    return r;
}
inline unsigned __byte_perm(unsigned a, unsigned b, unsigned s) {
    const uint64_t x = ((uint64_t)b << 32) | a;
    unsigned r = 0;
    for (int i = 0; i < 4; ++i) r |= (unsigned)((x >> (8 * ((s >> (4 * i)) & 7u))) & 255u) << (8 * i);
    return r;
}
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned n) {
    return (unsigned)(((((uint64_t)hi << 32) | lo) << (n & 31u)) >> 32);
}
inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned n) {
    return (unsigned)((((uint64_t)hi << 32) | lo) >> (n & 31u));
}
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
inline unsigned __vcmpeq4(unsigned a, unsigned b) {
    unsigned r = 0;
    for (int i = 0; i < 32; i += 8) r |= ((a >> i) & 255u) == ((b >> i) & 255u) ? 255u << i : 0u;
    return r;
}
inline unsigned __float_as_uint(float f) { return simt::from_bits<unsigned>(simt::to_bits(f)); }
inline float __uint_as_float(unsigned u) { return simt::from_bits<float>(u); }
inline float __int_as_float(int u) { return simt::from_bits<float>((unsigned)u); }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __int2float_rn(int v) { return (float)v; }
inline float __ull2float_rn(unsigned long long v) { return (float)v; }
inline int __float2int_rd(float f) { return (int)std::floor(f); }
inline int __float2int_rz(float f) { return (int)f; }

// memory
template <typename T>
T __ldg(const T* p) { return *p; }
template <typename T>
T __ldcg(const T* p) { return *p; }
template <typename T, typename U>
T atomicAdd(T* p, U v) { const T o = *p; *p = (T)(o + (T)v); return o; }
template <typename T, typename U>
T atomicOr(T* p, U v) { const T o = *p; *p = (T)(o | (T)v); return o; }
template <typename T, typename U>
T atomicMin(T* p, U v) { const T o = *p; if ((T)v < o) *p = (T)v; return o; }
template <typename T, typename U>
T atomicMax(T* p, U v) { const T o = *p; if (o < (T)v) *p = (T)v; return o; }
inline void __threadfence() {}
inline void __nanosleep(unsigned) {}

// ---------------------------------------------------------------- runtime ----------------
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToHost, cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, cudaMemcpyDeviceToDevice };
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes {
    cudaMemoryType type;
    int device;
    void *devicePointer, *hostPointer;
};
struct cudaDeviceProp {
    int major, minor, multiProcessorCount;
    char name[256];
};
enum { cudaHostAllocDefault = 0, cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
cudaError_t simt_malloc(void** p, size_t n);
template <typename T>
cudaError_t cudaMalloc(T** p, size_t n) { return simt_malloc(reinterpret_cast<void**>(p), n); }
#define SIMT_API __attribute__((visibility("hidden"))) cudaError_t
SIMT_API cudaFree(void* p);
SIMT_API cudaHostAlloc(void** p, size_t n, unsigned flags);
SIMT_API cudaFreeHost(void* p);
SIMT_API cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st);
SIMT_API cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k);
SIMT_API cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st);
SIMT_API cudaMemset(void* d, int v, size_t n);
SIMT_API cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags);
SIMT_API cudaStreamDestroy(cudaStream_t s);
SIMT_API cudaStreamSynchronize(cudaStream_t s);
SIMT_API cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned flags);
SIMT_API cudaEventCreateWithFlags(cudaEvent_t* e, unsigned flags);
SIMT_API cudaEventCreate(cudaEvent_t* e);
SIMT_API cudaEventDestroy(cudaEvent_t e);
SIMT_API cudaEventRecord(cudaEvent_t e, cudaStream_t s);
SIMT_API cudaEventSynchronize(cudaEvent_t e);
SIMT_API cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b);
SIMT_API cudaGetLastError();
SIMT_API cudaPeekAtLastError();
__attribute__((visibility("hidden"))) const char* cudaGetErrorString(cudaError_t e);
SIMT_API cudaSetDevice(int d);
SIMT_API cudaGetDevice(int* d);
SIMT_API cudaGetDeviceCount(int* n);
SIMT_API cudaGetDeviceProperties(cudaDeviceProp* p, int d);
SIMT_API cudaDeviceReset();
SIMT_API cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p);
#define cudaFuncSetAttribute(...) cudaSuccess
template <typename T>
cudaError_t cudaGetSymbolAddress(void** p, T& sym) { *p = (void*)&sym; return cudaSuccess; }
