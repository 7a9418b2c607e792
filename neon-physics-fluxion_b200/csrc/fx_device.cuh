// fx_device.cuh -- small device helpers shared by the kernels.
#pragma once
#include <cfloat>
#include <cstdint>

namespace fx {

__device__ __forceinline__ int lin_tid() {
  return threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
}
__device__ __forceinline__ int block_threads() {
  return blockDim.x * blockDim.y * blockDim.z;
}

// Rust's `(v / cell) as usize` followed by `.min(n - 1)` (grid.rs:58-62):
// IEEE f32 division, truncation toward zero, NaN and negatives saturate to 0,
// large values (and +inf) clamp to n - 1. `cell` is the f32 cell size.
__device__ __forceinline__ int cell_at(float v, float cell, int n) {
  const float q = __fdiv_rn(v, cell);
  if (!(q >= 1.0f)) return 0;
  if (q >= (float)n) return n - 1;
  const int c = (int)q;
  return c < n - 1 ? c : n - 1;
}

// Deterministic block reductions (fixed shuffle tree, fixed warp order).
// Every thread of the block must call them; the result is valid everywhere.
__device__ __forceinline__ double block_sum_double(double v) {
  __shared__ double ws[32];
  __shared__ double total;
  const int t = lin_tid(), lane = t & 31, w = t >> 5;
  const int nw = (block_threads() + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  if (w == 0) {
    double u = lane < nw ? ws[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u += __shfl_down_sync(0xffffffffu, u, o);
    if (lane == 0) total = u;
  }
  __syncthreads();
  return total;
}

__device__ __forceinline__ float block_max_float(float v) {
  __shared__ float ws[32];
  __shared__ float total;
  const int t = lin_tid(), lane = t & 31, w = t >> 5;
  const int nw = (block_threads() + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) ws[w] = v;
  __syncthreads();
  if (w == 0) {
    float u = lane < nw ? ws[lane] : -FLT_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u = fmaxf(u, __shfl_down_sync(0xffffffffu, u, o));
    if (lane == 0) total = u;
  }
  __syncthreads();
  return total;
}

// Cross-block FP64 sum in a fixed order: each block stores its partial, the
// last block to finish adds all partials (same order every run) into
// *result and re-arms the counter.
__device__ __forceinline__ void last_block_sum(double block_value,
                                               double *partial,
                                               unsigned int *done,
                                               double *result) {
  __shared__ bool last;
  const int t = lin_tid();
  if (t == 0) {
    partial[blockIdx.x] = block_value;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0;
  for (int i = t; i < (int)gridDim.x; i += block_threads())
    a += ((volatile double *)partial)[i];
  a = block_sum_double(a);
  if (t == 0) {
    *result = a;
    *done = 0;
  }
}

// Global adds whose old value is not needed, issued as reductions: the warp
// does not wait for the L2 round trip of an atomic that returns a value.
__device__ __forceinline__ void red_add_global(int *p, int v) {
  asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "r"(v)
               : "memory");
}
__device__ __forceinline__ void red_add_global(unsigned long long *p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
               "l"(v)
               : "memory");
}

// Warp-aggregated atomic adds: lanes naming the same element (idx >= 0) are
// combined and one lane issues the atomic. Every lane of the warp must call
// these (idx < 0 = nothing to add); base is global memory. Sums of integers
// are exact, so the result does not depend on the grouping.
// Lanes are grouped by __match_any_sync, which takes a step per distinct value,
// only where two neighbouring lanes name the same element; otherwise they are
// spread (an early placement: 61 us for the net kernel at 1M gates, whose four
// adds a net took 67 when always matched, ncu cold) and add lane by lane.
// Crowded elements (a contracted placement, a grid's corner) nearly always
// show such a pair, and what is missed costs time only.
__device__ __forceinline__ bool crowded(int i) {
  const int next = __shfl_down_sync(0xffffffffu, i, 1);  // by every lane, before any test
  return __any_sync(0xffffffffu, i >= 0 && i == next && (threadIdx.x & 31u) < 31u);
}

__device__ __forceinline__ void agg_add_u64(unsigned long long *base, long long idx,
                                            unsigned long long v) {
  const unsigned lane = threadIdx.x & 31u;
  const int i = (int)idx;  // indexes fit 31 bits (density bins: G^2 <= 8192^2)
  if (!crowded(i)) {
    if (i >= 0) red_add_global(base + i, v);
    return;
  }
  const unsigned peers = __match_any_sync(0xffffffffu, i);
  unsigned long long sum = 0;
#pragma unroll
  for (int src = 0; src < 32; ++src) {
    const unsigned long long w = __shfl_sync(0xffffffffu, v, src);
    if ((peers >> src) & 1u) sum += w;
  }
  if (i >= 0 && lane == (unsigned)(__ffs(peers) - 1)) red_add_global(base + i, sum);
}

// Adds the same constant `v` from every lane naming idx (>= 0); `few`: into so
// few elements that lanes are likely to meet anyway, and are always matched.
__device__ __forceinline__ void agg_add_const_i32(int *base, long long idx, int v, bool few) {
  const unsigned lane = threadIdx.x & 31u;
  const int i = (int)idx;  // indexes fit 31 bits
  if (!few && !crowded(i)) {
    if (i >= 0) red_add_global(base + i, v);
    return;
  }
  const unsigned peers = __match_any_sync(0xffffffffu, i);
  if (i >= 0 && lane == (unsigned)(__ffs(peers) - 1)) red_add_global(base + i, v * __popc(peers));
}

// The hardware reciprocal square root without the subnormal handling of
// rsqrtf, for arguments that are never subnormal.
__device__ __forceinline__ float rsqrt_approx_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed pairs of f32 (one instruction, each half rounded as the scalar one).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Order-preserving float <-> uint mapping for atomicMin/atomicMax.
__device__ __forceinline__ unsigned int f2ord(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned int u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

}  // namespace fx
