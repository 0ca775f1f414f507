/*
 * devcommon.cuh — device helpers shared by the kernels: the reference's cell
 * index clamps, type packing in float4.w, and block reductions.
 */
#ifndef FLIP_DEVCOMMON_CUH
#define FLIP_DEVCOMMON_CUH

#include "flipgpu_impl.h"
#include "refmath.h"
#include "../../include/flip_rng.h"

/* int i = fmax(0, fmin(gn-1, gn*p)) (src/sorter.cpp:35-37): the double
 * clamp of a float product is exact in float. */
__device__ __forceinline__ int cell_clamp(float p, float fn, int n) {
  return (int)fmaxf(0.0f, fminf((float)(n - 1), fn * p));
}

/* int i = fmin(N-1, fmax(0, p*N)) (src/flip3D.cpp:903-905, 944). */
__device__ __forceinline__ int cell_clamp_minmax(float p, float fn, int n) {
  return (int)fminf((float)(n - 1), fmaxf(0.0f, p * fn));
}

/* FLOAT x = max(0, min(cs, cs*p)) with the macros of src/utility.h:16-17
 * (src/corrector.cpp:59-61), truncated by the int parameter: range [0, n]. */
__device__ __forceinline__ int cell_clamp_macro(float p, float fn) {
  float v = fn * p;
  float mn = (fn > v) ? v : fn;
  float mx = (0.0f > mn) ? 0.0f : mn;
  return (int)mx;
}

/* (i, j, k) of linear index c over extents (., e1, e2), k fastest, in 32-bit
 * arithmetic (grids are at most 1024^3 cells or 1025 x 1024^2 faces, so
 * every index fits; 64-bit division costs several times more) */
__device__ __forceinline__ void decode_index(size_t c, int e1, int e2, int &i, int &j, int &k) {
  const unsigned c32 = (unsigned)c, u1 = (unsigned)e1, u2 = (unsigned)e2;
  const unsigned row = c32 / u2;
  k = (int)(c32 - row * u2);
  i = (int)(row / u1);
  j = (int)(row - (unsigned)i * u1);
}

__device__ __forceinline__ size_t cell_id(int n, int i, int j, int k) {
  return ((size_t)i * n + j) * n + k;
}

__device__ __forceinline__ float pack_type(uint8_t t) {
  return __int_as_float((int)t);
}
__device__ __forceinline__ int unpack_type(float w) { return __float_as_int(w); }

/* Deterministic block sum of doubles: fixed shuffle tree, then warp 0. */
template <int BLOCK>
__device__ __forceinline__ double block_sum_double(double v) {
  __shared__ double warp_part[BLOCK / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) warp_part[wid] = v;
  __syncthreads();
  double r = 0.0;
  if (wid == 0) {
    r = (lane < BLOCK / 32) ? warp_part[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  __syncthreads();
  return r; /* valid in thread 0 */
}

template <int BLOCK>
__device__ __forceinline__ uint32_t block_sum_u32(uint32_t v) {
  __shared__ uint32_t warp_part[BLOCK / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) warp_part[wid] = v;
  __syncthreads();
  uint32_t r = 0;
  if (wid == 0) {
    r = (lane < BLOCK / 32) ? warp_part[lane] : 0u;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  __syncthreads();
  return r;
}

/* Double-float accumulator: hi + lo carries about 44+ significant bits with
 * FP32 instructions only (Knuth TwoSum; products split exactly by FMA). Used
 * for dot products, where per-element FP64 is GB300's bottleneck. */
struct FF {
  float hi, lo;
};

__device__ __forceinline__ FF ff_zero() { return FF{0.0f, 0.0f}; }

/* acc += b (b a float) */
__device__ __forceinline__ void ff_add(FF &a, float b) {
  float s, e;
  refmath::two_sum(a.hi, b, s, e);
  a.hi = s;
  a.lo += e;
}

/* acc += x*y with the product kept exact */
__device__ __forceinline__ void ff_add_prod(FF &a, float x, float y) {
  float p = x * y;
  float pe = fmaf(x, y, -p);
  ff_add(a, p);
  a.lo += pe;
}

__device__ __forceinline__ FF ff_merge(FF a, FF b) {
  float s, e;
  refmath::two_sum(a.hi, b.hi, s, e);
  e += a.lo + b.lo;
  float hi = s + e;
  float lo = e - (hi - s);
  return FF{hi, lo};
}

__device__ __forceinline__ FF ff_shfl_down(FF v, int o) {
  return FF{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
}

/* Block sum in a fixed tree; the result is valid in every thread. */
template <int BLOCK> __device__ __forceinline__ FF block_sum_ff(FF v) {
  __shared__ FF warp_part[BLOCK / 32];
  __shared__ FF total;
  for (int o = 16; o > 0; o >>= 1) v = ff_merge(v, ff_shfl_down(v, o));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) warp_part[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    FF t = warp_part[0];
    for (int i = 1; i < BLOCK / 32; i++) t = ff_merge(t, warp_part[i]);
    total = t;
  }
  __syncthreads();
  FF r = total;
  __syncthreads();
  return r;
}

/* A counting grid barrier: bar[0] counts the arrivals of the whole launch
 * (zeroed before it), so the epoch-th barrier is complete when it reaches
 * epoch x gridDim.x. Thread 0 arrives with an acquire-release add after the
 * block's __syncthreads (the last block to arrive reads no more) and polls
 * with acquire loads: two L2 round trips, no reset and no generation word. The
 * wait gives up after limit_ns of %globaltimer (0: at once), sets *expired and
 * returns false in that block (the others give up at their next barrier). */
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr unsigned long long BARRIER_NS = 2000000000ull;

__device__ __forceinline__ bool count_barrier_for(unsigned *bar, unsigned &epoch, int *expired,
                                                  unsigned long long limit_ns) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    epoch++;
    const unsigned target = epoch * gridDim.x;
    unsigned v;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(bar) : "memory");
    v += 1;
    bool good = true;
    unsigned long long t0 = 0;
    unsigned spins = 0;
    const unsigned mask = limit_ns < BARRIER_NS ? 0u : 1023u; /* polls between looks at the time */
    while ((int)(v - target) < 0) {
      if ((++spins & mask) == 0) {
        const unsigned long long t = global_ns();
        if (t0 == 0 && limit_ns != 0) {
          t0 = t;
        } else if (t - t0 > limit_ns) {
          atomicExch(expired, 1);
          good = false;
          break;
        }
      }
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

/* the solvers' barrier: an expired wait is the solve's FLIPGPU_ETIMEOUT */
__device__ __forceinline__ bool count_barrier(unsigned *bar, unsigned &epoch, int *iflags) {
  return count_barrier_for(bar, epoch, iflags + IF_TIMEOUT, BARRIER_NS);
}

__device__ __forceinline__ double ff_to_double(FF v) { return (double)v.hi + (double)v.lo; }

#endif
