// A CUDA runtime for the host, for tests without a GPU: the kernel sources (host_kernels.py rewrites their launches
// and inline PTX) compile with g++ against this header, and a launch runs its blocks here. Every thread of a block
// is a fiber that runs until a barrier, a warp vote or a shuffle and is resumed when the others have arrived. Which
// warp goes first is chosen by emu::order: a missing barrier shows as a wrong result for an order that keeps a warp
// back, a write out of range as a changed guard word behind shared or allocated memory, a barrier that not all reach
// as an abort. One launch after the other; a cluster's blocks run together, other blocks one after the other.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __grid_constant__
#define __shared__ static                     // static shared memory: one block at a time (clusters use none)
#define __align__(n) __attribute__((aligned(n)))

struct dim3 {
    unsigned x, y, z;
    dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {}
};
struct double2 { double x, y; };
inline double2 make_double2(double a, double b) { return {a, b}; }

namespace emu {

struct Fiber {
    void* sp = nullptr;
    char* stack = nullptr;
    int tid = 0, block = 0;
    bool ready = true, done = false;
};
struct Meet { int arrived = 0; std::vector<Fiber*> waiting; };

extern Fiber* cur;
extern std::vector<int> order;                // warps in the order they are resumed (the rest follow, in turn)
extern bool keep;                             // true: a warp runs as far as it can before a later one of the order
int block_threads();
void meet(Meet& m, int n, bool cluster = false);
Meet& barrier(int id);                        // of the current block
Meet& cluster_barrier();
int cluster_size();
void warp_wait();
uint64_t* warp_slots();                       // 32 words of the current warp's next exchange
double* dyn_smem();
double* dyn_smem_of(int rank);
void launch(dim3 grid, dim3 block, size_t smem, const std::function<void()>& body, int cluster = 1);

template <class F>
void launch4(const F& body, dim3 grid, dim3 block, size_t smem, void*) { launch(grid, block, smem, body); }

template <class T>
uint64_t bits(T v) { uint64_t b = 0; std::memcpy(&b, &v, sizeof v); return b; }
template <class T>
T unbits(uint64_t b) { T v; std::memcpy(&v, &b, sizeof v); return v; }

// every lane's value of v, exchanged
template <class T, class F>
auto exchange(T v, F pick) {
    uint64_t* s = warp_slots();
    s[cur->tid & 31] = bits(v);
    warp_wait();
    return pick(s, cur->tid & 31);
}

}  // namespace emu

struct EmuIdx { unsigned x, y, z; };
extern EmuIdx threadIdx, blockIdx, blockDim, gridDim;

inline void __syncthreads() { emu::meet(emu::barrier(0), emu::block_threads()); }
inline void __syncwarp(unsigned = 0) { emu::warp_slots(); emu::warp_wait(); }
inline void __threadfence() {}
inline void __nanosleep(unsigned) {}
template <class T> T __shfl_up_sync(unsigned, T v, int d) {
    return emu::exchange(v, [d](uint64_t* s, int l) { return emu::unbits<T>(s[l >= d ? l - d : l]); });
}
template <class T> T __shfl_down_sync(unsigned, T v, int d) {
    return emu::exchange(v, [d](uint64_t* s, int l) { return emu::unbits<T>(s[l + d < 32 ? l + d : l]); });
}
template <class T> T __shfl_sync(unsigned, T v, int src) {
    return emu::exchange(v, [src](uint64_t* s, int) { return emu::unbits<T>(s[src & 31]); });
}
template <class T> T __shfl_xor_sync(unsigned, T v, int m) {
    return emu::exchange(v, [m](uint64_t* s, int l) { return emu::unbits<T>(s[l ^ m]); });
}
template <class T> unsigned __match_any_sync(unsigned, T v) {
    return emu::exchange(v, [](uint64_t* s, int l) {
        unsigned m = 0;
        for (int i = 0; i < 32; ++i) m |= (s[i] == s[l] ? 1u : 0u) << i;
        return m;
    });
}
inline unsigned __ballot_sync(unsigned, int p) {
    return emu::exchange(p != 0, [](uint64_t* s, int) {
        unsigned m = 0;
        for (int i = 0; i < 32; ++i) m |= (s[i] ? 1u : 0u) << i;
        return m;
    });
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
    return emu::exchange(v, [](uint64_t* s, int) {
        unsigned m = 0;
        for (int i = 0; i < 32; ++i) m = std::max(m, (unsigned)s[i]);
        return m;
    });
}
template <class T, class U> T atomicAdd(T* p, U v) { const T o = *p; *p = o + (T)v; return o; }
template <class T, class U> T atomicMax(T* p, U v) { const T o = *p; *p = std::max(o, (T)v); return o; }
template <class T> T atomicCAS(T* p, T c, T v) { const T o = *p; if (o == c) *p = v; return o; }
template <class T> T __ldcg(const T* p) { return *p; }
template <class T> T __ldg(const T* p) { return *p; }
template <class T> void __stcg(T* p, T v) { *p = v; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline long long __double_as_longlong(double v) { return (long long)emu::bits(v); }
inline double __longlong_as_double(long long v) { return emu::unbits<double>((uint64_t)v); }
inline int __double2hiint(double v) { return (int)(emu::bits(v) >> 32); }
inline double __hiloint2double(int h, int l) {
    return emu::unbits<double>(((uint64_t)(unsigned)h << 32) | (unsigned)l);
}
inline long long __double2ll_rn(double v) {
    if (std::isnan(v)) return (long long)0x8000000000000000ull;
    if (v >= 9.2233720368547758e18) return 0x7fffffffffffffffll;
    if (v <= -9.2233720368547758e18) return (long long)0x8000000000000000ull;
    return std::llrint(v);
}
inline float __fdividef(float a, float b) { return a / b; }
inline long long clock64() { return 0; }
using std::fabs;
using std::floor;
using std::fma;
using std::fmax;
using std::max;
using std::min;
using std::rint;
using std::sqrt;

// ---- the runtime calls of the host code: device memory is host memory, streams run at once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorInvalidDevice = 101 };
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost, cudaMemcpyDeviceToDevice };
enum { cudaDevAttrMaxSharedMemoryPerBlockOptin, cudaDevAttrMultiProcessorCount };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize };
enum { cudaLaunchAttributeClusterDimension, cudaLaunchAttributeCooperative };
struct cudaLaunchAttribute { int id; struct { struct { unsigned x, y, z; } clusterDim; int cooperative; } val; };
struct cudaLaunchConfig_t {
    dim3 gridDim, blockDim;
    size_t dynamicSmemBytes;
    cudaStream_t stream;
    cudaLaunchAttribute* attrs;
    unsigned numAttrs;
};
inline const char* cudaGetErrorString(cudaError_t) { return "host CUDA error"; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int* v, int a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448;          // (sm_100: 227 KB per block)
    return cudaSuccess;
}
extern long emu_mallocs, emu_copies;
namespace emu {
constexpr size_t kGuard = 4096;               // bytes on either side of an allocation, and behind shared memory
constexpr unsigned char kGuardByte = 0xfd;    // (0xfdfd...: as a double a large negative number)
inline void check_guard(const unsigned char* p, const char* what) {
    for (size_t i = 0; i < kGuard; ++i)
        if (p[i] != kGuardByte) {
            std::fprintf(stderr, "emu: a write out of range, %s\n", what);
            std::abort();
        }
}
}  // namespace emu
inline cudaError_t cudaMalloc(void** p, size_t n) {
    ++emu_mallocs;
    unsigned char* q = (unsigned char*)std::malloc(n + 2 * emu::kGuard + 64);
    std::memcpy(q, &n, sizeof n);
    std::memset(q + 64, emu::kGuardByte, emu::kGuard);
    std::memset(q + 64 + emu::kGuard, 0, n);
    std::memset(q + 64 + emu::kGuard + n, emu::kGuardByte, emu::kGuard);
    *p = q + 64 + emu::kGuard;
    return cudaSuccess;
}
inline cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    unsigned char* q = (unsigned char*)p - emu::kGuard - 64;
    size_t n;
    std::memcpy(&n, q, sizeof n);
    emu::check_guard(q + 64, "before an allocation");
    emu::check_guard((unsigned char*)p + n, "behind an allocation");
    std::free(q);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy(void* d, const void* s, size_t n, int) { ++emu_copies; std::memmove(d, s, n); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
inline cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
inline cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
inline cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 34; return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
inline cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
template <class T> cudaError_t cudaEventElapsedTime(T* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
template <class T> cudaError_t cudaGetSymbolAddress(void** p, T& symbol) { *p = (void*)symbol; return cudaSuccess; }
typedef int CUresult;
typedef void* CUcontext;
enum { CUDA_SUCCESS = 0, cudaEnableDefault = 0 };
enum cudaDriverEntryPointQueryResult { cudaDriverEntryPointSuccess, cudaDriverEntryPointSymbolNotFound };
inline cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, int, cudaDriverEntryPointQueryResult*) {
    return cudaErrorInvalidValue;
}
template <class F> cudaError_t cudaFuncSetAttribute(F, int, int) { return cudaSuccess; }
template <class F> cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int*, F, int, size_t) { return cudaErrorInvalidValue; }
inline cudaError_t cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorInvalidValue; }
template <class F> cudaError_t cudaOccupancyMaxActiveClusters(int* n, F, const cudaLaunchConfig_t*) { *n = 1; return cudaSuccess; }
template <class K, class... A> cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* c, K k, const A&... a) {
    emu::launch(c->gridDim, c->blockDim, c->dynamicSmemBytes, [&] { k(a...); },
                (int)(c->numAttrs ? c->attrs[0].val.clusterDim.x : 1));
    return cudaSuccess;
}
