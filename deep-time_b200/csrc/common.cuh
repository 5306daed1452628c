// Shared helpers of the deep-time B200 backend: status handling, complex arithmetic on CUDA's
// vector types, and the deterministic block reductions every CG kernel uses.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>

#include <cstdint>
#include <cstdio>
#include <string>
#include <type_traits>

#include "deeptime_gpu.h"

namespace dt {

// The message behind the last non-OK status of this thread (dt_last_error).
void set_error(const char* fmt, ...);
const char* last_error();

#define DT_CUDA(call)                                                                        \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess) {                                                                 \
      ::dt::set_error("%s:%d: %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_));   \
      return e_ == cudaErrorMemoryAllocation ? DT_OOM : DT_DEVICE_ERROR;                     \
    }                                                                                        \
  } while (0)

// DT_CUDA for functions without a status: records the error, which a later DT_CUDA reports.
#define DT_CUDA_VOID(call)                                                                   \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess)                                                                   \
      ::dt::set_error("%s:%d: %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_));   \
  } while (0)

#define DT_TRY(...)               \
  do {                            \
    dt_status s_ = (__VA_ARGS__); \
    if (s_ != DT_OK) return s_;   \
  } while (0)

template <class T>
struct cx;
template <>
struct cx<double> {
  using type = double2;
};
template <>
struct cx<float> {
  using type = float2;
};
template <class T>
using cplx = typename cx<T>::type;

template <class C>
__host__ __device__ __forceinline__ C mk(decltype(C::x) a, decltype(C::x) b) {
  C r;
  r.x = a;
  r.y = b;
  return r;
}
template <class C>
__device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <class C>
__device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <class C>
__device__ __forceinline__ C cmul(C a, C b) { return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <class C>
__device__ __forceinline__ C cconj(C a) { return mk<C>(a.x, -a.y); }
template <class C>
__device__ __forceinline__ C cscale(C a, decltype(C::x) s) { return mk<C>(a.x * s, a.y * s); }
// i * a
template <class C>
__device__ __forceinline__ C cmuli(C a) { return mk<C>(-a.y, a.x); }

// Single precision: both parts in one paired FP32 instruction (sm_100's add / mul / fma on
// float2), each part rounded as the scalar forms above round it (a - b as fma(b, -1, a), exact
// but for the one rounding of the sum; products contracted into one fma, as the compiler
// contracts the scalar forms).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return __ffma2_rn(make_float2(-a.y, a.y), make_float2(b.y, b.x), __fmul2_rn(make_float2(a.x, a.x), b));
}

// Reciprocals with no slow-path call: float, the correctly rounded intrinsic; double, for normal x
// below 2^1022 (divisors of positive definite systems; 0 and infinity give no number, NaN gives NaN):
// of x = m 2^e, m in [1, 2), the hardware's float estimate of 1 / m, scaled by 2^-e in the exponent
// bits and refined by two Newton-Raphson steps r <- r + r (1 - x r) (each squares the relative
// error: 2^-22 -> 2^-44 -> 2^-88, so the last rounding is what is left).
__device__ __forceinline__ double recip(double x) {
  const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) - 1023;
  const double m = __hiloint2double(hi - (e << 20), __double2loint(x));
  double r = (double)__fdividef(1.0f, (float)m);
  r = __hiloint2double(__double2hiint(r) - (e << 20), __double2loint(r));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}
__device__ __forceinline__ float recip(float x) { return __frcp_rn(x); }

// ---- deterministic reductions -------------------------------------------------------------
// A reducing kernel writes one partial per block (fixed grid, fixed in-block order); the last
// block to finish (an atomic ticket) sums the partials in index order. The result therefore does
// not depend on the order blocks ran in.

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// Sum over the block (any multiple of 32 threads up to 1024); the result is valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* scratch32) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int nwarps = (blockDim.x * blockDim.y + 31) >> 5;
  int tid = threadIdx.x + threadIdx.y * blockDim.x;
  lane = tid & 31;
  warp = tid >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch32[warp] = v;
  __syncthreads();
  double r = 0.0;
  if (warp == 0) {
    r = lane < nwarps ? scratch32[lane] : 0.0;
    r = warp_sum(r);
  }
  return r;
}
template <int NV>
struct Acc {
  double v[NV];
};

// The block's NV values (kind: 0 sum, 1 max per component) reduced in one pass; valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_reduce(double* v, const int* kind, double (*scratch)[32]) {
  const int tid = threadIdx.x + threadIdx.y * blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = (blockDim.x * blockDim.y + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const double u = __shfl_down_sync(0xffffffffu, v[q], o);
      v[q] = kind[q] ? fmax(v[q], u) : v[q] + u;
    }
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) scratch[q][warp] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = lane < nwarps ? scratch[q][lane] : kind[q] ? -INFINITY : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const double u = __shfl_down_sync(0xffffffffu, v[q], o);
        v[q] = kind[q] ? fmax(v[q], u) : v[q] + u;
      }
  }
}

// Writes this block's partials and, in the last block to arrive (an atomic ticket, reset for
// reuse), reduces all of them in a fixed order; true there, with the results in thread 0. A tail
// of latencies at the end of every reducing kernel: the components go through the shuffles
// together, the ticket's atomic carries both halves of the order (its release follows this block's
// partials; its acquire, in the same thread, precedes the barrier that lets the last block's threads
// read the others'), and two partials a thread are in flight (four took the vector kernels past 32
// registers, eight blocks an SM). One component after another, a
// __threadfence and one load at a time made an FP64 512 x 256 update 12.2 us (with the L2 flushed)
// where a kernel without a reduction took 8.2; this 11.5.
template <int NV>
__device__ bool reduce_partials(Acc<NV>& a, const int* kind, double* partials, unsigned int* ticket, unsigned int nblocks) {
  __shared__ double scratch[NV][32];
  __shared__ bool is_last;
  const unsigned tid = threadIdx.x + threadIdx.y * blockDim.x, nthreads = blockDim.x * blockDim.y;
  const unsigned bid = blockIdx.x + blockIdx.y * gridDim.x;
  block_reduce<NV>(a.v, kind, scratch);
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) partials[(size_t)q * nblocks + bid] = a.v[q];
    unsigned int t;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(ticket) : "memory");
    is_last = t == nblocks - 1;
    if (is_last) *ticket = 0u;
  }
  __syncthreads();
  if (!is_last) return false;
#pragma unroll
  for (int q = 0; q < NV; ++q) a.v[q] = kind[q] ? -INFINITY : 0.0;
  for (unsigned b = tid; b < nblocks; b += 2 * nthreads) {
    double p[NV][2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int q = 0; q < NV; ++q)
        p[q][u] = b + u * nthreads < nblocks ? __ldcg(partials + (size_t)q * nblocks + b + u * nthreads)
                                             : kind[q] ? -INFINITY : 0.0;
#pragma unroll
    for (int q = 0; q < NV; ++q)
      a.v[q] = kind[q] ? fmax(fmax(a.v[q], p[q][0]), p[q][1]) : a.v[q] + (p[q][0] + p[q][1]);
  }
  block_reduce<NV>(a.v, kind, scratch);
  return true;
}

// Kernel launches of the calling thread (eager ones, and those recorded while capturing a graph
// body); defined in flexure.cu.
// The U-Net's forward pass on a given stream, without synchronising (defined in unet.cu).
dt_status unet_predict_on(dt_unet* u, cudaStream_t st, const float* x, float* y, int B, int H, int W);

void count_launch();
long long launches_now();
void add_launches(long long k);
void begin_capture_count();
long long end_capture_count();

inline unsigned int ceil_div(size_t a, size_t b) { return (unsigned int)((a + b - 1) / b); }

// Test support for the allocation failure path: with DT_FAIL_ALLOC_AT=n in the environment, the
// n-th device allocation of a handle (its counter `made`, from 1) fails as if the device were out
// of memory. Without the variable every allocation goes to cudaMalloc.
inline bool alloc_fault(size_t& made) {
  ++made;
  const char* e = getenv("DT_FAIL_ALLOC_AT");
  return e && e[0] && (size_t)strtoull(e, nullptr, 10) == made;
}
inline bool is_pow2(long v) { return v > 0 && (v & (v - 1)) == 0; }
inline int ilog2(long v) {
  int r = 0;
  while ((1L << r) < v) ++r;
  return r;
}

}  // namespace dt
