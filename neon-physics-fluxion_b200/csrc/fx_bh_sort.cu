// fx_bh_sort.cu -- the Barnes-Hut keys and their sort for a small design, in
// one launch by one thread-block cluster.
//
// The stages are those of fx_bh.cu (root square, 30-bit Morton keys, a stable
// LSD radix sort, the sorted positions and their tile sums) with the same
// results. On a few
// thousand points they are bound by latency, not by the work: seven launches
// whose blocks each run a chain of dependent rounds and, in the sort, wait on
// one another through global memory (69 us for 5k points, of 184 us for the
// whole iteration). Here a cluster of eight blocks keeps the pairs in its
// shared memory throughout: a pass ranks each block's pairs, exchanges the
// blocks' digit counts over distributed shared memory, stages the pairs in
// digit order and copies each digit's run to the blocks that own its places
// (runs, because single remote stores took 2.6 cycles each). Three passes of
// ten bits cover the key. The cluster stops at 32,768 points: there a block
// holds 104 KB of shared memory and 512 threads, so that the cluster still
// finds room beside another job's persistent kernels, and the many-block
// kernels have caught up.
#include <cooperative_groups.h>

#include <cstdlib>

#include "fx_bh.cuh"
#include "fx_internal.h"

namespace cg = cooperative_groups;

namespace fx {
namespace {

constexpr int kCl = 8;              // blocks per cluster (the portable maximum)
constexpr int kClThreads = 512, kClWarps = kClThreads / 32;
constexpr int kClDigits = 1024;     // ten-bit digits, two per thread
constexpr int kClPasses = 3;
constexpr int kClMaxItems = 8;      // pairs per thread
constexpr int kClMax = kCl * kClThreads * kClMaxItems;
static_assert(kClMax <= 1 << 16, "counts and places are packed in 16 bits");

// Pairs (key, index) of this block and in digit order; the warps' digit
// counters; per digit the block's count and the base of its run, two digits
// to a word.
template <int kItems>
struct ClSmem {
  uint2 pair[kClThreads * kItems], stage[kClThreads * kItems];
  uint32_t cnt[kClWarps][kClDigits / 2];
  uint32_t hist[kClDigits / 2];
  uint16_t start[kClDigits];  // of the digit's run in stage
  uint16_t base[kClDigits];   // its place in the whole order, less start
  uint2 wtot[kClWarps];
  ulonglong4 wsum[kItems][kClWarps];
};

// kItems pairs per thread; block b owns places [b * per, (b + 1) * per) with
// per = 512 * kItems, warp w of it the 32 * kItems from w * 32 * kItems on.
template <int kItems>
__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kClThreads)
bh_cluster_sort_kernel(const float *__restrict__ px, const float *__restrict__ py, int n,
                       unsigned int *__restrict__ bbox, float th2, float md2,
                       uint32_t *__restrict__ keys, int32_t *__restrict__ idx,
                       float2 *__restrict__ spos, ulonglong4 *__restrict__ tile_sum,
                       float *__restrict__ root) {
  extern __shared__ __align__(16) unsigned char raw[];
  auto &sh = *reinterpret_cast<ClSmem<kItems> *>(raw);
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int per = kClThreads * kItems;
  constexpr int lg = kItems == 1 ? 9 : kItems == 2 ? 10 : kItems == 4 ? 11 : 12;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int rank = (int)cluster.block_rank();
  const int b0 = rank * per, seg = w * (32 * kItems);
  const float4 rt = bh_root_of(bbox, th2, md2);
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int at = seg + r * 32 + lane, i = b0 + at;
    // places past n get the largest key and stay behind every point
    uint32_t k = 0xffffffffu;
    if (i < n)
      k = (spread15(quantize15(px[i], rt.x, rt.z)) << 1) |
          spread15(quantize15(py[i], rt.y, rt.z));
    sh.pair[at] = make_uint2(k, (uint32_t)i);
  }
  const unsigned lt = (1u << lane) - 1u;
  uint16_t *cnt16 = reinterpret_cast<uint16_t *>(&sh.cnt[w][0]);
#pragma unroll 1
  for (int pass = 0; pass < kClPasses; ++pass) {
    const int shift = 10 * pass;
    for (int i = t; i < kClWarps * kClDigits / 8; i += kClThreads)
      reinterpret_cast<uint4 *>(&sh.cnt[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint2 p[kItems];
    uint32_t rk[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) p[r] = sh.pair[seg + r * 32 + lane];
    // stable ranks within the warp's segment
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t d = (p[r].x >> shift) & (kClDigits - 1);
      const unsigned peers = match_digit<10>(d);
      const uint32_t old = cnt16[d];
      __syncwarp();
      if ((peers & lt) == 0u) cnt16[d] = (uint16_t)(old + __popc(peers));
      __syncwarp();
      rk[r] = old + __popc(peers & lt);
    }
    __syncthreads();
    // thread t = digits 2t, 2t + 1: the warps' first ranks, the block's counts
    uint32_t own = 0;
    {
      uint32_t c[kClWarps];
#pragma unroll
      for (int q = 0; q < kClWarps; ++q) c[q] = sh.cnt[q][t];
#pragma unroll
      for (int q = 0; q < kClWarps; ++q) {
        sh.cnt[q][t] = own;
        own += c[q];  // both halves stay below 2^16
      }
      sh.hist[t] = own;
    }
    cluster.sync();  // every block's counts are out, and its pairs in registers
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int q = 0; q < kCl; ++q) {
      const uint32_t c = cluster.map_shared_rank(sh.hist, q)[t];
      before += q < rank ? c : 0u;
      all += c;
    }
    // exclusive scans over the digits: of the block's counts, and of all
    const uint32_t own0 = own & 0xffffu, own1 = own >> 16, all0 = all & 0xffffu, all1 = all >> 16;
    uint2 inc = make_uint2(own0 + own1, all0 + all1);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t ux = __shfl_up_sync(0xffffffffu, inc.x, o);
      const uint32_t uy = __shfl_up_sync(0xffffffffu, inc.y, o);
      if (lane >= o) {
        inc.x += ux;
        inc.y += uy;
      }
    }
    if (lane == 31) sh.wtot[w] = inc;
    __syncthreads();
    uint2 ex = make_uint2(inc.x - own0 - own1, inc.y - all0 - all1);
#pragma unroll
    for (int q = 0; q < kClWarps; ++q) {
      const uint2 v = sh.wtot[q];
      ex.x += q < w ? v.x : 0u;
      ex.y += q < w ? v.y : 0u;
    }
    // places of all padded pairs wrap at 2^16 only in `base`, which is added
    // to a place in the run modulo 2^16
    sh.start[2 * t] = (uint16_t)ex.x;
    sh.start[2 * t + 1] = (uint16_t)(ex.x + own0);
    sh.base[2 * t] = (uint16_t)(ex.y + (before & 0xffffu) - ex.x);
    sh.base[2 * t + 1] = (uint16_t)(ex.y + all0 + (before >> 16) - (ex.x + own0));
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const uint32_t d = (p[r].x >> shift) & (kClDigits - 1);
      sh.stage[sh.start[d] + cnt16[d] + rk[r]] = p[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      const int j = r * kClThreads + t;
      const uint2 q = sh.stage[j];
      const uint32_t pos = (sh.base[(q.x >> shift) & (kClDigits - 1)] + (uint32_t)j) & 0xffffu;
      cluster.map_shared_rank(sh.pair, (int)(pos >> lg))[pos & (per - 1)] = q;
    }
    cluster.sync();  // the pairs have arrived
  }
  float2 pos[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int at = r * kClThreads + t;
    pos[r] = make_float2(0.f, 0.f);
    if (b0 + at < n) {
      const uint2 q = sh.pair[at];
      keys[b0 + at] = q.x;
      idx[b0 + at] = (int32_t)q.y;
      pos[r] = make_float2(px[q.y], py[q.y]);
    }
  }
  // the sums of each 512 places, row r of the block
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int at = r * kClThreads + t;
    if (b0 + at < n) spos[b0 + at] = pos[r];
    const FixSums s = warp_sums128({fixed64(pos[r].x), fixed64(pos[r].y)});
    if (lane == 0) sh.wsum[r][w] = pack_sums(s);
  }
  __syncthreads();
  if (w < kItems) {
    FixSums s{0, 0};
    if (lane < kClWarps) s = unpack_sums(sh.wsum[w][lane]);
    s = warp_sums128(s);
    if (lane == 0 && b0 + w * kClThreads < n)
      tile_sum[rank * kItems + w] = pack_sums(s);
  }
  if (rank == 0 && t == 0) {
    root[0] = rt.x;
    root[1] = rt.y;
    root[2] = rt.z;
    root[3] = rt.w;
    // every block has read the box (before the first cluster barrier)
    bbox[0] = 0xffffffffu;
    bbox[1] = 0xffffffffu;
    bbox[2] = 0u;
    bbox[3] = 0u;
  }
}

// Whether the device has room for one cluster of this size: a process limited
// to a share of the SMs may not.
template <int kItems>
bool cluster_fits() {
  constexpr int smem = (int)sizeof(ClSmem<kItems>);
  if (raise_smem_limit((const void *)bh_cluster_sort_kernel<kItems>, smem) != FX_OK) return false;
  cudaLaunchAttribute dim{};
  dim.id = cudaLaunchAttributeClusterDimension;
  dim.val.clusterDim.x = kCl;
  dim.val.clusterDim.y = dim.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kCl);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &dim;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, bh_cluster_sort_kernel<kItems>, &cfg) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return clusters > 0;
}

int items_for(int n) {
  const int need = (n + kCl * kClThreads - 1) / (kCl * kClThreads);
  return need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : 8;
}

template <int kItems>
int launch_sort(const float *x, const float *y, int n, unsigned int *bbox, float th2, float md2,
                uint32_t *keys, int32_t *idx, float2 *spos, ulonglong4 *tile_sum, float *root,
                cudaStream_t s) {
  constexpr int smem = (int)sizeof(ClSmem<kItems>);
  FX_TRY(raise_smem_limit((const void *)bh_cluster_sort_kernel<kItems>, smem));
  bh_cluster_sort_kernel<kItems><<<kCl, kClThreads, smem, s>>>(x, y, n, bbox, th2, md2, keys,
                                                               idx, spos, tile_sum, root);
  FX_CHECK_LAUNCH();
  return FX_OK;
}

}  // namespace

// Asked once per context and size; never where the environment variable
// FLUXION_BH_CLUSTER is 0 (a test setting).
bool bh_cluster_fits(fx_ctx *ctx, int n) {
  if (n <= 0 || n > kClMax) return false;
  static const bool off = [] {
    const char *e = std::getenv("FLUXION_BH_CLUSTER");
    return e && std::atoi(e) == 0;
  }();
  if (off) return false;
  const int items = items_for(n);
  signed char &fits = ctx->sort_cluster_fits[items == 8 ? 3 : items / 2];
  if (fits < 0)
    fits = items == 1 ? cluster_fits<1>() : items == 2 ? cluster_fits<2>()
           : items == 4 ? cluster_fits<4>() : cluster_fits<8>();
  return fits > 0;
}

int bh_cluster_sort(fx_ctx *ctx, const float *x, const float *y, int n, unsigned int *bbox,
                    float th2, float md2, uint32_t *keys, int32_t *idx, float2 *spos,
                    ulonglong4 *tile_sum, float *root, cudaStream_t s) {
  if (n <= 0) return FX_OK;
  if (n > kClMax) {
    set_error("bh_cluster_sort: %d points exceed %d", n, kClMax);
    return FX_EINVAL;
  }
  const int items = items_for(n);
  const auto f = items == 1 ? launch_sort<1> : items == 2 ? launch_sort<2>
                 : items == 4 ? launch_sort<4> : launch_sort<8>;
  FX_TRY(f(x, y, n, bbox, th2, md2, keys, idx, spos, tile_sum, root, s));
  ctx->launches += 1;
  return FX_OK;
}

}  // namespace fx
