// fx_bh.cuh -- Barnes-Hut root square, Morton keys and exact sums, shared by
// the kernels of fx_bh.cu and fx_bh_sort.cu.
#pragma once
#include <cstdint>

#include "fx_device.cuh"
#include "fx_internal.h"

namespace fx {

// Root square {x_min, y_min, size, deep} from the ordered-int box
// (BarnesHutTree.cpp:24-46, in f32 without contraction); deep keys when a
// level-15 cell is not always accepted.
__device__ __forceinline__ float4 bh_root_of(const unsigned int *bbox, float th2, float md2) {
  float mnx = ord2f(bbox[0]), mny = ord2f(bbox[1]);
  float mxx = ord2f(bbox[2]), mxy = ord2f(bbox[3]);
  mnx = __fsub_rn(mnx, 1.0f);
  mxx = __fadd_rn(mxx, 1.0f);
  mny = __fsub_rn(mny, 1.0f);
  mxy = __fadd_rn(mxy, 1.0f);
  const float size = fmaxf(__fsub_rn(mxx, mnx), __fsub_rn(mxy, mny));
  const float cx = __fmul_rn(__fadd_rn(mnx, mxx), 0.5f);
  const float cy = __fmul_rn(__fadd_rn(mny, mxy), 0.5f);
  const float half = __fmul_rn(size, 0.5f);
  const float s15 = ldexpf(size, -15);
  return make_float4(__fsub_rn(cx, half), __fsub_rn(cy, half), size,
                     __fmul_rn(s15, s15) >= __fmul_rn(th2, md2) ? 1.0f : 0.0f);
}

__device__ __forceinline__ uint32_t quantize15(float p, float o, float size) {
  const float t = __fmul_rn(__fdiv_rn(__fsub_rn(p, o), size), 32768.0f);
  if (!(t > 0.0f)) return 0u;
  const float c = ceilf(t);
  if (c >= 32768.0f) return 32767u;
  return (uint32_t)c - 1u;
}

__device__ __forceinline__ uint32_t spread15(uint32_t v) {
  v &= 0x7fffu;
  v = (v | (v << 8)) & 0x00ff00ffu;
  v = (v | (v << 4)) & 0x0f0f0f0fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}

__device__ __forceinline__ __int128 fixed64(float v) {
  const uint32_t u = __float_as_uint(v);
  const int e = (int)((u >> 23) & 255u);
  if (e == 0 || e == 255) return 0;
  const unsigned long long m = (u & 0x7fffffu) | 0x800000u;  // v = m * 2^(e - 150)
  const int sh = e - 86;                                     // v * 2^64 = m * 2^(e - 86)
  unsigned __int128 r = 0;
  if (sh >= 0) r = (unsigned __int128)m << sh;
  else if (sh > -64) r = m >> (-sh);
  return (u >> 31) ? -(__int128)r : (__int128)r;
}

__device__ __forceinline__ ulonglong2 pack128(__int128 v) {
  return make_ulonglong2((unsigned long long)v, (unsigned long long)((unsigned __int128)v >> 64));
}
__device__ __forceinline__ __int128 unpack128(ulonglong2 p) {
  return (__int128)(((unsigned __int128)p.y << 64) | p.x);
}
__device__ __forceinline__ __int128 shfl_up128(__int128 v, int d) {
  const ulonglong2 p = pack128(v);
  return unpack128(make_ulonglong2(__shfl_up_sync(0xffffffffu, p.x, d),
                                   __shfl_up_sync(0xffffffffu, p.y, d)));
}


// Exact (x, y) sums.
struct FixSums {
  __int128 x, y;
};
__device__ __forceinline__ ulonglong4 pack_sums(FixSums s) {
  const ulonglong2 a = pack128(s.x), c = pack128(s.y);
  return make_ulonglong4(a.x, a.y, c.x, c.y);
}
__device__ __forceinline__ FixSums unpack_sums(ulonglong4 v) {
  return {unpack128(make_ulonglong2(v.x, v.y)), unpack128(make_ulonglong2(v.z, v.w))};
}
__device__ __forceinline__ FixSums warp_sums128(FixSums s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const ulonglong4 p = pack_sums(s);
    const FixSums u = unpack_sums(make_ulonglong4(
        __shfl_xor_sync(0xffffffffu, p.x, o), __shfl_xor_sync(0xffffffffu, p.y, o),
        __shfl_xor_sync(0xffffffffu, p.z, o), __shfl_xor_sync(0xffffffffu, p.w, o)));
    s.x += u.x;
    s.y += u.y;
  }
  return s;
}
// Sum over a block of kThreads, valid in every thread.
template <int kThreads>
__device__ __forceinline__ FixSums block_sums128(FixSums s) {
  __shared__ ulonglong4 ws[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  s = warp_sums128(s);
  __syncthreads();
  if (lane == 0) ws[w] = pack_sums(s);
  __syncthreads();
  FixSums r{0, 0};
#pragma unroll
  for (int q = 0; q < kThreads / 32; ++q) {
    const FixSums v = unpack_sums(ws[q]);
    r.x += v.x;
    r.y += v.y;
  }
  return r;
}

// The lanes of the warp whose `Bits`-bit digit equals the caller's, by one
// ballot per bit. (In the cluster sort; the eight-bit digits of the many-block
// passes are no faster this way than with __match_any_sync.)
template <int Bits>
__device__ __forceinline__ unsigned match_digit(uint32_t d) {
  unsigned m = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < Bits; ++b) {
    const bool p = (d >> b) & 1u;
    const unsigned v = __ballot_sync(0xffffffffu, p);
    m &= p ? v : ~v;
  }
  return m;
}

// Keys, stable sort, sorted positions, root square and the exact sums of every
// 512 consecutive points (tile_sum: ceil(n / 512) of them) in one launch
// (fx_bh_sort.cu), where bh_cluster_fits: up to 32,768 points, and a device
// share with room for the cluster; for positions whose keys need no deep
// levels. Re-arms bbox.
bool bh_cluster_fits(fx_ctx *ctx, int n);
int bh_cluster_sort(fx_ctx *ctx, const float *x, const float *y, int n, unsigned int *bbox,
                    float th2, float md2, uint32_t *keys, int32_t *idx, float2 *spos,
                    ulonglong4 *tile_sum, float *root, cudaStream_t s);

}  // namespace fx
