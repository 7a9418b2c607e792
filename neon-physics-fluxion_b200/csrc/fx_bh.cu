// fx_bh.cu -- row B: Barnes-Hut repulsion on the device.
//
// Tree semantics follow the reference quadtree (O/src/cpp/BarnesHutTree.cpp):
//   * root square: bounding box grown by a margin of 1.0, side = the larger
//     extent, centred on the box (BarnesHutTree.cpp:24-46);
//   * quadrant rule: a point on a midline goes west/south (`px <= mx`,
//     BarnesHutTree.cpp:107-123). The quantised key uses ceil(t) - 1, which
//     maps (k, k+1] to cell k, so a point exactly on a boundary falls in the
//     lower cell;
//   * opening rule: a node is replaced by its centre of mass when it is a
//     single point or size / max(d, min_dist) < theta (BarnesHutTree.cpp:
//     151-166); the law is k * q * Q / d^2 along the unit vector
//     (placer.rs:258-272, q = 1).
// Instead of pointer insertion the tree is built from sorted 30-bit Morton
// keys (15 bits per axis): a binary radix tree (Karras 2012) whose nodes are
// mapped back to quadtree cells. A binary node whose prefix length is
// delta, under a parent of prefix length delta_p, holds exactly the points of
// every quad cell of level l with delta_p < 2l <= delta; those cells share
// one centre of mass, so the walk tests only the smallest (level
// floor(delta/2)). Nodes that stand for no quad level (delta_p and delta in
// the same level) are always opened. Points that share all 30 key bits form
// a bucket (a cell of level 15): it is accepted as a whole by the same rule,
// otherwise each of its points interacts directly.
// Deep keys: the distance in the opening rule is clamped to min_dist, so a
// cell smaller than theta * min_dist is accepted by every point. When a
// level-15 cell is not (size^2 >= theta^2 min_dist^2, decided on the device
// from the root square), each point also gets the 24-bit key of its sub-cell
// within its level-15 cell (12 more levels, computed in f64), the points are
// sorted by (key, sub-key, index), and the tree has 27 levels: its buckets
// are then accepted whole by every point, and a crowded cell costs log k per
// point instead of k. The host skips these kernels when the positions lie in
// the die and (die + 2) / 2^15 < theta * min_dist.
//
// Every value is fixed by the sorted keys alone: node mass sums are added in
// tree order (left + right, FP64) by a bottom-up sweep, decisions and forces
// use IEEE f32 operations without contraction (the inverse square root is a
// fixed bit-level estimate plus Newton steps), and each point adds its terms
// in a fixed order. The result is bit-identical run to run and to a sequential
// restatement of the same rules.
#include <algorithm>
#include <climits>
#include <cstdlib>

#include "fx_internal.h"
#include "fx_bh.cuh"
#include "fx_device.cuh"

namespace fx {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048 keys
constexpr int kWalkWarps = 8;
constexpr int kStack = 64;       // walk stack of a 15-level tree (<= 3 * 15 + 4)
constexpr int kStackDeep = 96;   // of a 27-level tree (<= 3 * 27 + 4)
constexpr int kDeepLevels = 12;  // levels below 15 in deep mode
constexpr int kKeyBits = 30, kDeepBits = kKeyBits + 2 * kDeepLevels;

// ---- bounding box and root square ----------------------------------------
__global__ void bh_bbox_kernel(const float *__restrict__ x,
                               const float *__restrict__ y, int n,
                               unsigned int *__restrict__ bbox) {
  float mnx = FLT_MAX, mny = FLT_MAX, mxx = -FLT_MAX, mxy = -FLT_MAX;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    const float px = x[i], py = y[i];
    mnx = fminf(mnx, px);
    mxx = fmaxf(mxx, px);
    mny = fminf(mny, py);
    mxy = fmaxf(mxy, py);
  }
  __shared__ float red[4][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mnx = fminf(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mxx = fmaxf(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mny = fminf(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mxy = fmaxf(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
  }
  if (lane == 0) {
    red[0][w] = mnx;
    red[1][w] = mny;
    red[2][w] = mxx;
    red[3][w] = mxy;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
      mnx = fminf(mnx, red[0][q]);
      mny = fminf(mny, red[1][q]);
      mxx = fmaxf(mxx, red[2][q]);
      mxy = fmaxf(mxy, red[3][q]);
    }
    atomicMin(bbox + 0, f2ord(mnx));
    atomicMin(bbox + 1, f2ord(mny));
    atomicMax(bbox + 2, f2ord(mxx));
    atomicMax(bbox + 3, f2ord(mxy));
  }
}

// Root square of the box, then re-arms the box for the next accumulation.
__global__ void bh_root_kernel(unsigned int *__restrict__ bbox,
                               float *__restrict__ root, float th2, float md2) {
  const float4 r = bh_root_of(bbox, th2, md2);
  root[0] = r.x;
  root[1] = r.y;
  root[2] = r.z;
  root[3] = r.w;
  bbox[0] = 0xffffffffu;
  bbox[1] = 0xffffffffu;
  bbox[2] = 0u;
  bbox[3] = 0u;
}

// Sub-cell (0..4095) of p within its level-15 cell c15, in f64 without
// contraction; a point the f32 quantisation put in c15 but that lies just
// outside it is clamped to the edge sub-cell, so cells nest.
__device__ __forceinline__ uint32_t quantize_sub(float p, float o, float size, uint32_t c15) {
  const double w = __ddiv_rn((double)size, 32768.0);
  const double o15 = __dadd_rn((double)o, __dmul_rn((double)c15, w));
  const double t = __dmul_rn(__ddiv_rn(__dsub_rn((double)p, o15), w), 4096.0);
  if (!(t > 0.0)) return 0u;
  const double c = ceil(t);
  if (c >= 4096.0) return 4095u;
  return (uint32_t)c - 1u;
}

// Keys (and identity indices); with klo, also the 24-bit sub-cell keys and
// the deep sort's inputs.
__global__ void bh_keys_kernel(const float *__restrict__ x,
                               const float *__restrict__ y, int n,
                               const float *__restrict__ root,
                               uint32_t *__restrict__ keys,
                               int32_t *__restrict__ idx, uint32_t *__restrict__ klo,
                               uint32_t *__restrict__ kl0, int32_t *__restrict__ il0) {
  const float ox = root[0], oy = root[1], size = root[2];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    const uint32_t qx = quantize15(x[i], ox, size);
    const uint32_t qy = quantize15(y[i], oy, size);
    keys[i] = (spread15(qx) << 1) | spread15(qy);
    idx[i] = i;
    if (klo) {
      const uint32_t lo = (spread15(quantize_sub(x[i], ox, size, qx)) << 1) |
                          spread15(quantize_sub(y[i], oy, size, qy));
      klo[i] = lo;
      kl0[i] = lo;
      il0[i] = i;
    }
  }
}

// Deep mode only (root[3] set): the primary keys and indices in the order of
// the sub-key sort (gather into buffer 1, then copy back to buffer 0), and
// the sub-keys in the final sorted order.
__global__ void bh_deep_gather_kernel(const float *__restrict__ root, int n,
                                      const uint32_t *__restrict__ keys0,
                                      const int32_t *__restrict__ il1,
                                      uint32_t *__restrict__ keys1,
                                      int32_t *__restrict__ idx1) {
  if (!(root[3] > 0.f)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int g = il1[i];
    keys1[i] = keys0[g];
    idx1[i] = g;
  }
}

__global__ void bh_deep_copy_kernel(const float *__restrict__ root, int n,
                                    const uint32_t *__restrict__ keys1,
                                    const int32_t *__restrict__ idx1,
                                    uint32_t *__restrict__ keys0, int32_t *__restrict__ idx0) {
  if (!(root[3] > 0.f)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    keys0[i] = keys1[i];
    idx0[i] = idx1[i];
  }
}

__global__ void bh_deep_slo_kernel(const float *__restrict__ root, int n,
                                   const uint32_t *__restrict__ klo,
                                   const int32_t *__restrict__ idx0,
                                   uint32_t *__restrict__ slo) {
  if (!(root[3] > 0.f)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    slo[i] = klo[idx0[i]];
}

// ---- stable LSD radix sort (8-bit digits) ------------------------------------
__global__ void __launch_bounds__(kSortThreads)
radix_hist_kernel(const uint32_t *__restrict__ keys, int n, int shift,
                  uint32_t *__restrict__ tile_hist, int T,
                  const float *__restrict__ gate = nullptr) {
  if (gate && !(gate[3] > 0.f)) return;  // a deep-key pass outside deep mode
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int base = blockIdx.x * kSortTile;
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  tile_hist[(size_t)threadIdx.x * T + blockIdx.x] = h[threadIdx.x];
}

// Per-digit exclusive scan of the digit-major tile histogram: block d scans
// the T tile counts of digit d and records the digit's total.
__global__ void __launch_bounds__(256)
radix_scan_kernel(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                  uint32_t *__restrict__ digit_total, int T,
                  const float *__restrict__ gate = nullptr) {
  if (gate && !(gate[3] > 0.f)) return;
  __shared__ uint32_t ws[8];
  const int d = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint32_t *row = in + (size_t)d * T;
  uint32_t *orow = out + (size_t)d * T;
  const int per = (T + 255) / 256;
  const int b = min(T, t * per), e = min(T, b + per);
  uint32_t s = 0;
  for (int i = b; i < e; ++i) s += row[i];
  uint32_t v = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) ws[w] = v;
  __syncthreads();
  uint32_t run = v - s;
  for (int q = 0; q < w; ++q) run += ws[q];
  for (int i = b; i < e; ++i) {
    const uint32_t c = row[i];
    orow[i] = run;
    run += c;
  }
  if (t == 255) digit_total[d] = run;
}

// Stable scatter: within a tile, warp w ranks its 256 keys in order
// (__match_any_sync groups lanes with equal digits), warps are ordered by a
// per-digit prefix over the warp counts, tiles by the per-digit scan and
// digits by the scan of the digit totals.
__global__ void __launch_bounds__(kSortThreads)
radix_scatter_kernel(const uint32_t *__restrict__ kin,
                     const int32_t *__restrict__ iin,
                     uint32_t *__restrict__ kout, int32_t *__restrict__ iout,
                     int n, int shift, const uint32_t *__restrict__ tile_scan,
                     const uint32_t *__restrict__ digit_total, int T,
                     const float *__restrict__ gate = nullptr) {
  if (gate && !(gate[3] > 0.f)) return;
  constexpr int kWarps = kSortThreads / 32;
  __shared__ uint32_t cnt[kWarps][256];
  __shared__ uint32_t doff[256];
  __shared__ uint32_t ws[kWarps];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int i = t; i < kWarps * 256; i += kSortThreads) (&cnt[0][0])[i] = 0;
  {
    const uint32_t s = digit_total[t];
    uint32_t v = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) ws[w] = v;
    __syncthreads();
    uint32_t off = v - s;
    for (int q = 0; q < w; ++q) off += ws[q];
    doff[t] = off;
  }
  __syncthreads();
  const int base = blockIdx.x * kSortTile + w * (32 * kSortItems);
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t k[kSortItems];
  int32_t v[kSortItems];
  uint32_t rank[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * 32 + lane;
    const bool valid = i < n;
    k[r] = valid ? kin[i] : 0u;
    v[r] = valid ? iin[i] : 0;
    const uint32_t dg = valid ? ((k[r] >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    const int leader = __ffs(peers) - 1;
    const uint32_t old = valid ? cnt[w][dg] : 0u;
    __syncwarp();
    if (valid && lane == leader) cnt[w][dg] = old + __popc(peers);
    __syncwarp();
    rank[r] = old + __popc(peers & lt_mask);
  }
  __syncthreads();
  // thread t = digit t: offsets of the warps within the digit, and the
  // digit's start within the tile (exclusive scan over digits)
  __shared__ uint32_t tstart[256];
  __shared__ uint32_t gbase[256];
  {
    uint32_t run = 0;
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) {
      const uint32_t c = cnt[ww][t];
      cnt[ww][t] = run;
      run += c;
    }
    uint32_t x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += u;
    }
    __syncthreads();
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint32_t st = x - run;
    for (int q = 0; q < w; ++q) st += ws[q];
    tstart[t] = st;
    // output index of tile position j of digit t: gbase[t] + j
    gbase[t] = doff[t] + tile_scan[(size_t)t * T + blockIdx.x] - st;
  }
  __syncthreads();
  // stage the tile in sorted order, then write it out: consecutive threads
  // cover consecutive positions of a digit's run, so the stores coalesce
  __shared__ uint32_t sk[kSortTile];
  __shared__ int32_t sv[kSortTile];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * 32 + lane;
    if (i < n) {
      const uint32_t dg = (k[r] >> shift) & 255u;
      const uint32_t j = tstart[dg] + cnt[w][dg] + rank[r];
      sk[j] = k[r];
      sv[j] = v[r];
    }
  }
  __syncthreads();
  const int m = min(kSortTile, n - (int)(blockIdx.x * kSortTile));
  for (int j = t; j < m; j += kSortThreads) {
    const uint32_t key = sk[j];
    const uint32_t pos = gbase[(key >> shift) & 255u] + (uint32_t)j;
    kout[pos] = key;
    iout[pos] = sv[j];
  }
}

// Stable LSD sort of (key, value) pairs on the low 8*passes key bits. The
// pairs start in (k[0], v[0]); the result is in (k[passes & 1], v[passes & 1]).
// Workspace: tile_hist / tile_scan of 256 * radix_sort_tiles(n) words each
// and digit_total of 256 words.
int radix_sort_pairs(uint32_t *k[2], int32_t *v[2], int n, int passes,
                     uint32_t *tile_hist, uint32_t *tile_scan, uint32_t *digit_total,
                     cudaStream_t s) {
  if (n <= 0) return FX_OK;
  const int T = (n + kSortTile - 1) / kSortTile;
  for (int pass = 0; pass < passes; ++pass) {
    const int src = pass & 1, dst = src ^ 1;
    radix_hist_kernel<<<T, kSortThreads, 0, s>>>(k[src], n, 8 * pass, tile_hist, T);
    radix_scan_kernel<<<256, 256, 0, s>>>(tile_hist, tile_scan, digit_total, T);
    radix_scatter_kernel<<<T, kSortThreads, 0, s>>>(k[src], v[src], k[dst], v[dst], n,
                                                    8 * pass, tile_scan, digit_total, T);
  }
  FX_CHECK_LAUNCH();
  return FX_OK;
}

int radix_sort_tiles(int n) { return (n + kSortTile - 1) / kSortTile; }

// ---- one-sweep LSD radix sort (the Barnes-Hut keys) ----------------------------
// The same stable sort in 1 + passes launches instead of 3 per pass: one
// kernel counts every pass's digits at once; then each pass is one kernel in
// which a block takes the next tile (an atomic ticket, so tiles start in
// order), ranks its keys stably as radix_scatter_kernel does, publishes its
// per-digit counts and finds the counts of all earlier tiles by a look-back
// over their published words (decoupled look-back). A block waits only on
// tiles whose blocks have started and publish their own counts before they
// wait, so every wait ends; each is still bounded, and an expired wait sets
// bit 4 of the error word (the host turns it into FX_ETIMEOUT).
constexpr uint32_t kOsAgg = 1u << 30, kOsInc = 2u << 30, kOsVal = (1u << 30) - 1u;
constexpr uint32_t kOsSpin = 1u << 22;
constexpr int kOsWin = 16;  // earlier tiles read per look-back step
// Tiles of 512 threads and 4 or 8 keys each: a block's time is mostly its
// chain of ranking rounds (one per key of a thread) and its look-back, so few
// keys win while the tiles are few, and long tiles once the look-back is the
// longer of the two. Keys and sort at 100k points: 51 us with 4, 61 with 8 (84
// with 256 threads of 16, and root, counts and identity values as launches and
// arrays of their own); at 1M 126 and 119 (136); even at about 500k.
constexpr int kOsThreads = 512;
constexpr int kOsFew = 1 << 19;
static int os_items(int n) { return n <= kOsFew ? 4 : 8; }
static int os_tiles(int n) {
  const int tile = kOsThreads * os_items(n);
  return (n + tile - 1) / tile;
}

// Root square, keys and every pass's digit counts in one pass over the
// positions (hist: 4 x 256 counts, zeroed before). Root and counts as launches
// of their own cost 14 us at 100k points.
constexpr int kKeysPer = 4;  // points per thread

__global__ void __launch_bounds__(256)
bh_keys_hist_kernel(const float *__restrict__ x, const float *__restrict__ y, int n,
                    const unsigned int *__restrict__ bbox, float th2, float md2,
                    float *__restrict__ root, uint32_t *__restrict__ keys,
                    uint32_t *__restrict__ hist) {
  __shared__ uint32_t h[4][256];
  const int t = threadIdx.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q][t] = 0;
  const float4 rt = bh_root_of(bbox, th2, md2);
  if (blockIdx.x == 0 && t == 0) {
    root[0] = rt.x;
    root[1] = rt.y;
    root[2] = rt.z;
    root[3] = rt.w;
  }
  const int b0 = blockIdx.x * (256 * kKeysPer) + t;
  float px[kKeysPer], py[kKeysPer];
#pragma unroll
  for (int r = 0; r < kKeysPer; ++r) {
    const int i = b0 + r * 256;
    px[r] = i < n ? x[i] : 0.f;
    py[r] = i < n ? y[i] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kKeysPer; ++r) {
    const int i = b0 + r * 256;
    if (i >= n) break;
    const uint32_t k = (spread15(quantize15(px[r], rt.x, rt.z)) << 1) |
                       spread15(quantize15(py[r], rt.y, rt.z));
    keys[i] = k;
#pragma unroll
    for (int q = 0; q < 4; ++q) atomicAdd(&h[q][(k >> (8 * q)) & 255u], 1u);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t c = h[q][t];
    if (c) atomicAdd(hist + q * 256 + t, c);
  }
}

__global__ void __launch_bounds__(256)
os_hist_kernel(const uint32_t *__restrict__ keys, int n, int passes,
               uint32_t *__restrict__ hist) {
  __shared__ uint32_t h[4][256];
  for (int i = threadIdx.x; i < 4 * 256; i += 256) (&h[0][0])[i] = 0;
  __syncthreads();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    const uint32_t k = keys[i];
    for (int q = 0; q < passes; ++q) atomicAdd(&h[q][(k >> (8 * q)) & 255u], 1u);
  }
  __syncthreads();
  for (int q = 0; q < passes; ++q) {
    const uint32_t c = h[q][threadIdx.x];
    if (c) atomicAdd(hist + q * 256 + threadIdx.x, c);
  }
}

// iin null: the values are the places (the first pass of an unsorted batch).
template <int kOsItems>
__global__ void __launch_bounds__(kOsThreads)
os_pass_kernel(const uint32_t *__restrict__ kin, const int32_t *__restrict__ iin,
               uint32_t *__restrict__ kout, int32_t *__restrict__ iout, int n, int shift,
               const uint32_t *__restrict__ hist, uint32_t *__restrict__ status,
               unsigned int *__restrict__ ticket, unsigned int *__restrict__ err,
               const float *__restrict__ px, const float *__restrict__ py,
               float2 *__restrict__ spos) {
  constexpr int kWarps = kOsThreads / 32, kOsTile = kOsThreads * kOsItems;
  __shared__ __align__(16) uint16_t cnt[kWarps][256];  // a warp ranks 32 * kOsItems pairs
  __shared__ uint32_t tstart[256], gbase[256], ws[8], ws2[8];
  __shared__ int tile_s;
  __shared__ uint32_t sk[kOsTile];
  __shared__ int32_t sv[kOsTile];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) tile_s = (int)atomicAdd(ticket, 1u);
  for (int i = t; i < kWarps * 32; i += kOsThreads)
    reinterpret_cast<uint4 *>(&cnt[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
  // threads 0 .. 255 own a digit each: its count over all keys
  const uint32_t dcount = t < 256 ? hist[t] : 0u;
  __syncthreads();
  const int tile = tile_s;
  const int base = tile * kOsTile + w * (32 * kOsItems);
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t k[kOsItems];
  int32_t v[kOsItems];
  uint32_t rank[kOsItems];
#pragma unroll
  for (int r = 0; r < kOsItems; ++r) {
    const int i = base + r * 32 + lane;
    k[r] = i < n ? kin[i] : 0u;
    v[r] = i < n ? (iin ? iin[i] : i) : 0;
  }
  // stable ranks within the tile: per warp by __match_any_sync, then warps
  // in order (as radix_scatter_kernel)
#pragma unroll
  for (int r = 0; r < kOsItems; ++r) {
    const bool valid = base + r * 32 + lane < n;
    const uint32_t dg = valid ? ((k[r] >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    const int leader = __ffs(peers) - 1;
    const uint32_t old = valid ? cnt[w][dg] : 0u;
    __syncwarp();
    if (valid && lane == leader) cnt[w][dg] = (uint16_t)(old + __popc(peers));
    __syncwarp();
    rank[r] = old + __popc(peers & lt_mask);
  }
  __syncthreads();
  // digit t: warp offsets, the digit's count in this tile, its start within
  // the tile and (scan of the counts over all keys) within the output
  uint32_t local = 0, inc = 0, dinc = 0;
  if (t < 256) {
    uint32_t c[kWarps];
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) c[ww] = cnt[ww][t];
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) {
      cnt[ww][t] = (uint16_t)local;
      local += c[ww];
    }
    atomicExch(status + (size_t)tile * 256 + t, (tile == 0 ? kOsInc : kOsAgg) | local);
    inc = local;
    dinc = dcount;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      const uint32_t ud = __shfl_up_sync(0xffffffffu, dinc, o);
      if (lane >= o) {
        inc += u;
        dinc += ud;
      }
    }
    if (lane == 31) {
      ws[w] = inc;
      ws2[w] = dinc;
    }
  }
  __syncthreads();
  if (t < 256) {
    uint32_t st = inc - local, dbase = dinc - dcount;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      st += q < w ? ws[q] : 0u;
      dbase += q < w ? ws2[q] : 0u;
    }
    tstart[t] = st;
    gbase[t] = dbase - st;  // completed by the look-back below
  }
  __syncthreads();
  // stage the tile in sorted order (the other warps while the first eight
  // look back)
#pragma unroll
  for (int r = 0; r < kOsItems; ++r) {
    const int i = base + r * 32 + lane;
    if (i < n) {
      const uint32_t dg = (k[r] >> shift) & 255u;
      const uint32_t j = tstart[dg] + cnt[w][dg] + rank[r];
      sk[j] = k[r];
      sv[j] = v[r];
    }
  }
  if (t < 256 && tile > 0) {  // decoupled look-back for digit t
    volatile uint32_t *stv = status;
    // The words of the kOsWin nearest earlier tiles are loaded together
    // (independent loads, one round trip) and added from the nearest on,
    // up to the first inclusive one; a tile that has not published yet is
    // waited for (bounded), then the window restarts from it.
    uint32_t prefix = 0;
    uint32_t spin = 0;
    for (int p = tile - 1; p >= 0;) {
      uint32_t wv[kOsWin];
#pragma unroll
      for (int q = 0; q < kOsWin; ++q)
        wv[q] = p - q >= 0 ? (uint32_t)stv[(size_t)(p - q) * 256 + t] : (uint32_t)(2u << 30);  // before tile 0: inclusive 0
      int q = 0;
      bool done = false;
#pragma unroll
      for (int r = 0; r < kOsWin; ++r) {
        if (done || q < r) continue;  // stopped at an earlier entry
        const uint32_t flag = wv[r] & ~kOsVal;
        if (flag == 0u) break;         // not published yet: q == r
        prefix += wv[r] & kOsVal;
        q = r + 1;
        if (flag == kOsInc) done = true;
      }
      if (done) break;
      p -= q;
      if (q < kOsWin && p >= 0) {  // wait for tile p to publish
        while ((stv[(size_t)p * 256 + t] & ~kOsVal) == 0u && spin < kOsSpin) ++spin;
        if (spin >= kOsSpin) {  // expired: record it and stop
          atomicOr(err, 4u);
          break;
        }
      }
    }
    __threadfence();
    atomicExch(status + (size_t)tile * 256 + t, kOsInc | (prefix + local));
    gbase[t] += prefix;
  }
  __syncthreads();
  const int m = min(kOsTile, n - tile * kOsTile);
#pragma unroll
  for (int r = 0; r < kOsItems; ++r) {
    const int j = r * kOsThreads + t;
    if (j < m) {
      const uint32_t key = sk[j];
      const uint32_t pos = gbase[(key >> shift) & 255u] + (uint32_t)j;
      const int32_t g = sv[j];
      kout[pos] = key;
      iout[pos] = g;
      if (spos) spos[pos] = make_float2(px[g], py[g]);
    }
  }
}

// Stable LSD sort of (key, value) pairs on the low 8*passes (<= 4) key bits,
// in 1 + passes launches. With spos, the last pass also writes
// spos[i] = (px[v], py[v]) for the sorted values v. Pairs start in (k[0], v[0]); the result is in
// (k[passes & 1], v[passes & 1]). Workspace `ws`: os_sort_words(n, passes)
// words, cleared here.
size_t os_sort_words(int n, int passes) {
  return (size_t)passes * 256 + (size_t)passes * os_tiles(n) * 256 + 4;
}

// The passes of a sort whose digit counts are in ws; v[0] holds the values,
// or the places themselves when `places`.
static int os_passes(uint32_t *k[2], int32_t *v[2], int n, int passes, uint32_t *ws,
                     unsigned int *err, cudaStream_t s, const float *px, const float *py,
                     float2 *spos, bool places) {
  const int T = os_tiles(n);
  uint32_t *hist = ws, *status = ws + passes * 256,
           *ticket = status + (size_t)passes * T * 256;
  for (int pass = 0; pass < passes; ++pass) {
    const int src = pass & 1, dst = src ^ 1;
    const bool last = pass == passes - 1;
    (os_items(n) == 4 ? os_pass_kernel<4> : os_pass_kernel<8>)<<<T, kOsThreads, 0, s>>>(
        k[src], places && pass == 0 ? nullptr : v[src], k[dst], v[dst], n, 8 * pass,
        hist + 256 * pass, status + (size_t)pass * T * 256, ticket + pass, err, px, py,
        last ? spos : nullptr);
  }
  FX_CHECK_LAUNCH();
  return FX_OK;
}

int radix_sort_onesweep(uint32_t *k[2], int32_t *v[2], int n, int passes, uint32_t *ws,
                        unsigned int *err, cudaStream_t s, const float *px,
                        const float *py, float2 *spos) {
  if (n <= 0) return FX_OK;
  if (passes > 4 || n >= (int)kOsVal) {
    set_error("radix_sort_onesweep: %d keys / %d passes out of range", n, passes);
    return FX_EINVAL;
  }
  FX_CHECK_CUDA(cudaMemsetAsync(ws, 0, os_sort_words(n, passes) * 4, s));
  os_hist_kernel<<<std::min((n + 2047) / 2048, 2 * 148), 256, 0, s>>>(k[0], n, passes, ws);
  return os_passes(k, v, n, passes, ws, err, s, px, py, spos, false);
}

// ---- exact prefix sums of the sorted positions ---------------------------------
// Every position becomes the 128-bit integer trunc(v * 2^64) (exact for
// |v| >= 2^-41; smaller magnitudes lose their bits below 2^-64, non-finite
// values count as 0). Integer sums do not depend on the order of addition,
// so the prefix is computed tile-parallel and a node's sum, a prefix
// difference, is exact. Its centre of mass is then
//   ((double)hi * 2^64 + (double)lo) * 2^-64 / count
// with hi/lo the upper (signed) and lower (unsigned) 64 bits, each step
// rounded to nearest.
constexpr int kFixThreads = 256, kFixItems = 8, kFixTile = kFixThreads * kFixItems;
constexpr int kFixSmall = 1 << 18;  // points up to which tiles hold 512

// Inclusive scan of one int128 per thread over the block; also returns the
// block total.
__device__ __forceinline__ __int128 block_scan128(__int128 v, __int128 &total) {
  __shared__ ulonglong2 wtot[kFixThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const __int128 u = shfl_up128(v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) wtot[w] = pack128(v);
  __syncthreads();
  __int128 off = 0, tot = 0;
  for (int q = 0; q < kFixThreads / 32; ++q) {
    const __int128 t = unpack128(wtot[q]);
    if (q < w) off += t;
    tot += t;
  }
  __syncthreads();
  total = tot;
  return v + off;
}

// The (x, y) sums of each tile of 256 * kItems sorted points.
template <int kItems>
__global__ void __launch_bounds__(kFixThreads)
fix_tile_kernel(const float2 *__restrict__ spos, int n, ulonglong4 *__restrict__ tile_sum) {
  const int b0 = blockIdx.x * (kFixThreads * kItems) + threadIdx.x;
  FixSums s{0, 0};
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int i = b0 + k * kFixThreads;
    if (i < n) {
      const float2 p = spos[i];
      s.x += fixed64(p.x);
      s.y += fixed64(p.y);
    }
  }
  s = block_sums128<kFixThreads>(s);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = pack_sums(s);
}

// Inclusive prefix of every point (x lo/hi, y lo/hi), tiles of 256 * kItems
// points: a block adds up the sums of all earlier tiles itself (they are few
// and in L2; a scan of them would be another launch), then scans its own. A
// thread's points are consecutive; they and the prefixes pass through shared
// memory, each warp's by itself, so that global accesses coalesce. 23 us with
// the tile sums at 1M points, 8 at 5k (31 and 17 with their scan, each thread
// writing its own run of 32-byte prefixes).
template <int kItems>
__global__ void __launch_bounds__(kFixThreads)
fix_prefix_kernel(const float2 *__restrict__ spos, int n,
                  const ulonglong4 *__restrict__ tile_sum, ulonglong4 *__restrict__ prefix) {
  constexpr int kWarps = kFixThreads / 32, kRun = 32 * kItems;  // points of a warp
  constexpr int kHalf = 2;  // of a thread's points, staged per turn
  __shared__ float2 pts[kWarps][kRun + 32];
  __shared__ ulonglong4 out[kWarps][32 * kHalf + 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int w0 = blockIdx.x * (kFixThreads * kItems) + w * kRun;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int j = k * 32 + lane;
    pts[w][j + j / kItems] = w0 + j < n ? spos[w0 + j] : make_float2(0.f, 0.f);
  }
  FixSums off{0, 0};
  for (int q = t; q < (int)blockIdx.x; q += kFixThreads) {
    const FixSums v = unpack_sums(tile_sum[q]);
    off.x += v.x;
    off.y += v.y;
  }
  off = block_sums128<kFixThreads>(off);
  __syncwarp();
  FixSums p[kItems], s{0, 0};
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const float2 v = pts[w][lane * (kItems + 1) + k];
    s.x += fixed64(v.x);
    s.y += fixed64(v.y);
    p[k] = s;
  }
  FixSums tot;
  off.x += block_scan128(s.x, tot.x) - s.x;
  off.y += block_scan128(s.y, tot.y) - s.y;
#pragma unroll
  for (int h = 0; h < kItems; h += kHalf) {
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kHalf; ++k)
      out[w][lane * (kHalf + 1) + k] = pack_sums({off.x + p[h + k].x, off.y + p[h + k].y});
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kHalf; ++k) {
      const int j = k * 32 + lane;  // the j-th staged prefix: lane j / kHalf's
      const int i = w0 + (j / kHalf) * kItems + h + j % kHalf;
      if (i < n) prefix[i] = out[w][j + j / kHalf];
    }
  }
}

// ((double)hi * 2^64 + (double)lo) * 2^-64, each step rounded to nearest.
__device__ __forceinline__ double fixed_to_double(__int128 v) {
  const long long hi = (long long)(v >> 64);
  const unsigned long long lo = (unsigned long long)v;
  return __dmul_rn(__dadd_rn(__dmul_rn(__ll2double_rn(hi), 18446744073709551616.0),
                             __ull2double_rn(lo)),
                   5.42101086242752217003726400434970855712890625e-20);
}

// ---- radix tree (Karras 2012) and walk records --------------------------------
// One thread per internal node does everything the walk needs of it: its
// range and split, its centre of mass from the prefix sums, and its quad
// children. What it needs of its parent is the larger of the two prefix lengths
// at its range's ends; what it needs of a child is that child's own prefix
// length and, where the child stands for no quad level, its split, which the
// warp mostly has (shuffles; the few large nodes search). One launch instead
// of two with ranges, splits and lengths stored between them: 14 us against
// 15 at 5k points (ncu cold) and a launch less in the chain; about even at 1M
// (67 us against 60). Latency of the searches' loads and divergence bound it
// (14 of 32 lanes active).
constexpr int kBuildThreads = 256;

struct BhKeys {
  const uint32_t *keys, *lo;  // sorted keys; sub-keys (deep mode) or null
  int n;
  __device__ __forceinline__ uint32_t at(int i) const { return __ldg(keys + i); }
  // Common prefix length of the keys a, b at sorted positions i and j: 30-bit
  // key, then (deep mode) the 24-bit sub-key, then the index.
  __device__ __forceinline__ int delta_of(uint32_t a, uint32_t b, int i, int j) const {
    if (a != b) return __clz(a ^ b) - 2;
    if (lo) {
      const uint32_t la = lo[i], lb = lo[j];
      if (la != lb) return kKeyBits + __clz(la ^ lb) - 8;
      return kDeepBits + __clz((uint32_t)(i ^ j));
    }
    return kKeyBits + __clz((uint32_t)(i ^ j));
  }
  __device__ __forceinline__ int delta(int i, int j) const {
    return j < 0 || j >= n ? -1 : delta_of(at(i), at(j), i, j);
  }
  // The largest x in [lo_x, hi_x] with delta(i, i + x d) > thr, which holds at
  // lo_x and stops holding once. Ranges beyond the staged keys take seven
  // probes a step, their loads in flight together (the chain of a binary
  // search in global memory is most of this kernel's time on small designs);
  // the short ranges of almost all nodes are bisected, since there the
  // instructions count (105 us at 1M points with seven probes throughout).
  __device__ __forceinline__ int reach(int i, int d, int lo_x, int hi_x, int thr) const {
    const uint32_t a = at(i);
    while (hi_x - lo_x > 64) {
      const int step = (hi_x - lo_x + 8) >> 3;  // eight parts of [lo_x, hi_x]
      uint32_t b[7];
#pragma unroll
      for (int p = 0; p < 7; ++p) b[p] = __ldg(keys + (i + min(lo_x + (p + 1) * step, hi_x) * d));
      int c = 0;
#pragma unroll
      for (int p = 0; p < 7; ++p) {
        const int x = lo_x + (p + 1) * step;
        if (x <= hi_x && delta_of(a, b[p], i, i + x * d) > thr) c = p + 1;
      }
      lo_x += c * step;
      hi_x = min(hi_x, lo_x + step - 1);
    }
    while (hi_x > lo_x) {
      const int x = (lo_x + hi_x + 1) >> 1;
      if (delta_of(a, at(i + x * d), i, i + x * d) > thr) lo_x = x;
      else hi_x = x - 1;
    }
    return lo_x;
  }
  // Last place of the left child of the node [f, l] with prefix length dn.
  __device__ __forceinline__ int split(int f, int l, int dn) const {
    return f + reach(f, 1, 0, l - f - 1, dn);
  }
};

constexpr int kNone = INT_MIN;

// Walk record of every internal node (two float4):
//   r0 = {cx_hi, cy_hi, cx_lo, cy_lo}  centre of mass as an f32 hi/lo pair
//   r1 = {count (negative: bucket), size^2 (negative: no quad level),
//         first, last (as int bits)}
// and its quad children: a child that stands for no quad level (at most one
// such level separates two quad cells) is replaced by its own two children, so
// every node lists up to four, in key order (leaf s as ~s, kNone: empty).
__global__ void __launch_bounds__(kBuildThreads)
bh_build_kernel(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ slo,
                const float *__restrict__ root, unsigned int *__restrict__ bbox, int n,
                const ulonglong4 *__restrict__ prefix, float4 *__restrict__ node,
                int4 *__restrict__ qchild) {
  const int i = blockIdx.x * kBuildThreads + threadIdx.x;
  if (i == 0) {  // re-armed for the next accumulation (the keys are made)
    bbox[0] = 0xffffffffu;
    bbox[1] = 0xffffffffu;
    bbox[2] = 0u;
    bbox[3] = 0u;
  }
  const bool valid = i < n - 1;
  const bool deep = slo && root[3] > 0.f;
  const int kb = deep ? kDeepBits : kKeyBits;  // prefix length of a bucket
  const BhKeys k{keys, deep ? slo : nullptr, n};
  int f = 0, l = 0, dn = 0, dp = 0, gamma = 0;
  if (valid) {
    // range: extends from i toward the neighbour it shares more with
    const int dr = k.delta(i, i + 1), dl = k.delta(i, i - 1);
    const int d = (dr - dl) >= 0 ? 1 : -1;
    const int dmin = min(dr, dl);
    // grow the range by factors of two, past 64 of eight, then search the last
    const int most = d > 0 ? n - 1 - i : i;  // places on that side
    int in = 1, top = min(2, most);          // holds at in; unknown at top
    while (top > in && k.delta(i, i + top * d) > dmin) {
      const int by = top < 64 ? 2 : 8;
      in = top;
      top = top > most / by ? most : top * by;
    }
    const int j = i + k.reach(i, d, in, top, dmin) * d;
    f = min(i, j);
    l = max(i, j);
    dn = k.delta(i, j);
    // the parent's prefix length: at i's end it is dmin, at the other end it is
    // what the node shares with the next place
    dp = max(dmin, d > 0 ? k.delta(l, l + 1) : k.delta(f, f - 1));
    gamma = k.split(f, l, dn);
  }
  // the children's prefix lengths and splits, from the lanes that have them
  // (small nodes: a child's index is close to its parent's)
  const int base = i & ~31;
  int cdn[2], cgam[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int src = gamma + h - base;
    cdn[h] = __shfl_sync(0xffffffffu, dn, src & 31);
    cgam[h] = __shfl_sync(0xffffffffu, gamma, src & 31);
    if ((unsigned)src >= 32u) cgam[h] = -1;
  }
  if (!valid) return;
  // centre of mass
  const int cnt = l - f + 1;
  const ulonglong4 pl = prefix[l];
  __int128 sx = unpack128(make_ulonglong2(pl.x, pl.y));
  __int128 sy = unpack128(make_ulonglong2(pl.z, pl.w));
  if (f > 0) {
    const ulonglong4 pf = prefix[f - 1];
    sx -= unpack128(make_ulonglong2(pf.x, pf.y));
    sy -= unpack128(make_ulonglong2(pf.z, pf.w));
  }
  int out[4] = {kNone, kNone, kNone, kNone};
  int o = 0;
  const int lv = dn >> 1;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int cf = h ? gamma + 1 : f, cl = h ? l : gamma;
    if (cf == cl) {
      out[o++] = ~cf;
      continue;
    }
    const int ci = gamma + h;
    const int dc = cgam[h] >= 0 ? cdn[h] : k.delta(cf, cl);
    if (dc < kb && (dc >> 1) == lv) {
      const int g = cgam[h] >= 0 ? cgam[h] : k.split(cf, cl, dc);
      out[o++] = g == cf ? ~g : g;
      out[o++] = g + 1 == cl ? ~(g + 1) : g + 1;
    } else {
      out[o++] = ci;
    }
  }
  qchild[i] = make_int4(out[0], out[1], out[2], out[3]);
  const double cx = __ddiv_rn(fixed_to_double(sx), (double)cnt);
  const double cy = __ddiv_rn(fixed_to_double(sy), (double)cnt);
  const float hx = (float)cx, hy = (float)cy;
  node[2 * i] = make_float4(hx, hy, (float)(cx - (double)hx), (float)(cy - (double)hy));
  const float rs = root[2];
  float c, s2;
  if (dn >= kb) {
    const float sz = ldexpf(rs, -(kb >> 1));
    c = -(float)cnt;
    s2 = __fmul_rn(sz, sz);
  } else {
    c = (float)cnt;
    if (dp >= 0 && (dp >> 1) == lv) {
      s2 = -1.0f;
    } else {
      const float sz = ldexpf(rs, -lv);
      s2 = __fmul_rn(sz, sz);
    }
  }
  node[2 * i + 1] = make_float4(c, s2, __int_as_float(f), __int_as_float(l));
}

// ---- warp-cooperative walk ----------------------------------------------------
// Each warp owns 32 consecutive sorted points (spatially close), split into
// groups of kWalkGroup lanes. Each group walks the quadtree with its own
// shared stack of (node, lane mask) entries, each an opened cell; the groups
// of a warp pop in lockstep, so one pass of the loop serves up to 32/kWalkGroup
// cells. Popping a cell evaluates all its children for the lanes in the mask:
// every lane applies the reference opening rule to its own point, so
// interaction lists are exactly per point. A lane adds, per opened cell, the
// terms of its children in order (single points, accepted cells, opened
// buckets point by point), and then descends into the children it opened, in
// order. A group's stack holds the union of its points' opened cells, which
// near the leaves is much smaller than the union over the whole warp.

// 1/sqrt(x) for x >= min_dist^2 > 0: the bit-level estimate of Lomont
// ("Fast inverse square root", 2003; constant 0x5f375a86) refined by three
// Newton steps y <- y * fma(-(x/2) * y, y, 1.5) in IEEE f32. Integer ops,
// correctly rounded products and fused multiply-adds only (each written out
// explicitly, nothing left to contraction), so a sequential restatement with
// fmaf reproduces it bit for bit; the result is within a couple of ulp of the
// exact value.
__device__ __forceinline__ float bh_rsqrt(float x) {
  float y = __int_as_float(0x5f375a86 - (__float_as_int(x) >> 1));
  const float h = __fmul_rn(0.5f, x);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    y = __fmul_rn(y, __fmaf_rn(-__fmul_rn(h, y), y, 1.5f));
  return y;
}

// The law k*Q/d^2 along (dx, dy)/d with d = max(|r|, min_dist), in f32:
// inv = rsqrt(max(r2, md^2)), f = ((kQ * inv) * inv) * inv,
// F = fma(f, r, F); r2 = fma(dx, dx, dy * dy).
template <bool Fast>
__device__ __forceinline__ void bh_term(float dx, float dy, float r2c, float kq,
                                        float &fx, float &fy) {
  const float inv = Fast ? rsqrtf(r2c) : bh_rsqrt(r2c);
  const float f = __fmul_rn(__fmul_rn(__fmul_rn(kq, inv), inv), inv);
  fx = __fmaf_rn(f, dx, fx);
  fy = __fmaf_rn(f, dy, fy);
}

template <bool Fast>
__device__ __forceinline__ void bh_direct(float px, float py, float2 q,
                                          float kq, float md2, float &fx,
                                          float &fy) {
  const float dx = __fsub_rn(px, q.x), dy = __fsub_rn(py, q.y);
  const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
  bh_term<Fast>(dx, dy, fmaxf(r2, md2), kq, fx, fy);
}

// Applies the opening rule of child c (an internal node when `cell`) to the
// lane's point when `in`; adds accepted-cell, single-point and bucket terms
// (Fast: with the hardware rsqrt; Count: counting them in `terms`).
// Called by all 32 lanes together (the ballot); returns the lanes that open
// c as a cell to descend into.
template <bool Fast, bool Count>
__device__ __forceinline__ unsigned bh_eval(int c, bool in, bool cell, int s,
                                            float2 p, float k, float th2,
                                            float md2,
                                            const float4 *__restrict__ node,
                                            const float2 *__restrict__ spos,
                                            float &fx, float &fy, int &terms) {
  bool op = false;
  if (in) {
    if (!cell) {  // single point ~c
      if (~c != s) {
        bh_direct<Fast>(p.x, p.y, spos[~c], k, md2, fx, fy);
        if (Count) ++terms;
      }
    } else {
      const float4 r0 = node[2 * c], r1 = node[2 * c + 1];
      const float dx = __fsub_rn(__fsub_rn(p.x, r0.x), r0.z);
      const float dy = __fsub_rn(__fsub_rn(p.y, r0.y), r0.w);
      const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
      const float r2c = fmaxf(r2, md2);
      // size^2 < 0 (a node standing for no quad level) is always opened
      if (r1.y >= 0.f && r1.y < __fmul_rn(th2, r2c)) {
        bh_term<Fast>(dx, dy, r2c, __fmul_rn(k, fabsf(r1.x)), fx, fy);
        if (Count) ++terms;
      } else if (r1.x > 0.f) {
        op = true;
      } else {  // bucket: point by point
        const int b = __float_as_int(r1.z), e = __float_as_int(r1.w);
        for (int t = b; t <= e; ++t)
          if (t != s) {
            bh_direct<Fast>(p.x, p.y, spos[t], k, md2, fx, fy);
            if (Count) ++terms;
          }
      }
    }
  }
  return __ballot_sync(0xffffffffu, op);
}

constexpr int kWalkGroup = 8;                    // lanes per group
constexpr int kWalkGroups = 32 / kWalkGroup;     // groups per warp

// The walk of the 32 points of one warp (sorted positions base .. base + 31),
// groups of kWalkGroup lanes each with their own stack in st_node / st_mask
// (this warp's [kWalkGroups][Stack + 1] arrays). Fast: FX_BH_FAST, the same
// cells and term order with the hardware rsqrt (a few ulp) instead of the
// reproducible one; Count: also each point's number of terms.
template <int Stack, bool Fast, bool Count>
__device__ __forceinline__ void bh_group_walk(
    int base, int n, const float2 *__restrict__ spos, const int32_t *__restrict__ perm,
    const int4 *__restrict__ qchild, const float4 *__restrict__ node, float k, float th2,
    float md2, float2 *__restrict__ force, unsigned int *__restrict__ err,
    int32_t *__restrict__ term_count, int32_t (*st_node)[Stack + 1],
    unsigned (*st_mask)[Stack + 1]) {
  const int lane = threadIdx.x & 31;
  const int g = lane / kWalkGroup;
  const bool leader = (lane % kWalkGroup) == 0;
  const unsigned gmask = (kWalkGroup == 32 ? 0xffffffffu
                                           : ((1u << kWalkGroup) - 1u) << (g * kWalkGroup));
  const int s = base + lane;
  const bool valid = s < n;
  const float2 p = valid ? spos[s] : make_float2(0.f, 0.f);
  float fx = 0.f, fy = 0.f;
  int sp = 0;  // this group's stack depth (uniform in the group)
  int terms = 0;
  auto eval = [&](int c, bool in, bool cell) -> unsigned {
    return bh_eval<Fast, Count>(c, in, cell, s, p, k, th2, md2, node, spos, fx, fy, terms);
  };
  if (n >= 2) {
    const unsigned open = eval(0, valid, true) & gmask;
    if (open) {
      if (leader) {
        st_node[g][0] = 0;
        st_mask[g][0] = open;
      }
      sp = 1;
    }
  }
  __syncwarp();
  while (__any_sync(0xffffffffu, sp > 0)) {
    const bool has = sp > 0;
    int nd = 0;
    unsigned mask = 0u;
    if (has) {
      --sp;
      nd = st_node[g][sp];
      mask = st_mask[g][sp];
    }
    __syncwarp();
    int4 q = make_int4(kNone, kNone, kNone, kNone);
    if (has) q = qchild[nd];
    const int qc[4] = {q.x, q.y, q.z, q.w};
    const bool in = (mask >> lane) & 1u;
    unsigned om[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int c = qc[h];
      om[h] = eval(c, in && c != kNone, c >= 0) & gmask;
    }
    const int np = (om[0] != 0u) + (om[1] != 0u) + (om[2] != 0u) + (om[3] != 0u);
    if (sp + np > Stack) {
      if (leader) atomicOr(err, 1u);
    } else {
      // push the opened children in reverse so the first one is popped first
#pragma unroll
      for (int h = 3; h >= 0; --h) {
        if (om[h] != 0u) {
          if (leader) {
            st_node[g][sp] = qc[h];
            st_mask[g][sp] = om[h];
          }
          ++sp;
        }
      }
    }
    __syncwarp();
  }
  if (valid) {
    force[perm[s]] = make_float2(fx, fy);
    if (Count) term_count[perm[s]] = terms;
  }
}

template <int Stack, bool Fast = false, bool Count = false>
__global__ void __launch_bounds__(kWalkWarps * 32, 8)
bh_walk_kernel(int n, const float2 *__restrict__ spos,
               const int32_t *__restrict__ perm,
               const int4 *__restrict__ qchild,
               const float4 *__restrict__ node, float k, float th2, float md2,
               float2 *__restrict__ force, unsigned int *__restrict__ err,
               int32_t *__restrict__ term_count = nullptr) {
  // one stack per group; the odd stride puts the groups' tops (often at the
  // same depth) in different banks
  __shared__ int32_t st_node[kWalkWarps][kWalkGroups][Stack + 1];
  __shared__ unsigned st_mask[kWalkWarps][kWalkGroups][Stack + 1];
  const int w = threadIdx.x >> 5;
  const int base = (blockIdx.x * kWalkWarps + w) * 32;
  if (base >= n) return;  // warp-uniform
  bh_group_walk<Stack, Fast, Count>(base, n, spos, perm, qchild, node, k, th2, md2, force,
                                    err, term_count, st_node[w], st_mask[w]);
}

// ---- walk of small designs --------------------------------------------------
// The group walk bit for bit (the same cells in the same order, each point's
// terms added in the same order), with eight points to a warp and four lanes
// to a point, one per child of the popped cell: the four children's loads and
// terms, a chain of four in the group walk, run side by side, and only the
// additions, from shuffles, keep their order. With few points the walk is
// bound by that chain, not by issue: 313 warps of 10k points left half of the
// schedulers idle. A cell's quad children are loaded with its record, so a
// pass is one trip to memory. 10k points 69 us (group walk 174), 100k 247
// (293), 130k 306 (332); at 300k, where issue counts, the group walk's 551
// wins (729), hence the limit. At opening angle 0 every cell is opened and the
// walk goes by all pairs, where issue counts much earlier: uniform points, 20k
// 7.4 ms (group walk 11.6), 30k 14.9 (17.3), 40k 24.7 (23.4), 130k 209 (107). At
// 0.02 the limit above still holds (130k 40, group walk 48).
constexpr int kSmallWarps = 4;
constexpr int kSmallWalkMax = 1 << 17;
constexpr int kSmallWalkPairs = 1 << 15;  // below an angle of 0.001
constexpr float kPairsTheta2 = 1e-6f;

template <int Stack>
__global__ void __launch_bounds__(kSmallWarps * 32)
bh_small_walk_kernel(int n, const float2 *__restrict__ spos, const int32_t *__restrict__ perm,
                     const int4 *__restrict__ qchild, const float4 *__restrict__ node, float k,
                     float th2, float md2, float2 *__restrict__ force,
                     unsigned int *__restrict__ err) {
  // opened cells: their quad children, and the points that opened them
  __shared__ int4 st_kids[kSmallWarps][Stack + 1];
  __shared__ unsigned st_mask[kSmallWarps][Stack + 1];
  const unsigned full = 0xffffffffu, ones = 0x11111111u;  // a bit per point
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int slot = lane & 3, own = lane & ~3;
  const int base = (blockIdx.x * kSmallWarps + w) * 8;
  if (base >= n) return;  // warp-uniform
  const int s = base + (lane >> 2);
  const bool valid = s < n;
  const float2 p = valid ? spos[s] : make_float2(0.f, 0.f);
  float fx = 0.f, fy = 0.f;
  int sp = 0;
  int4 kids = make_int4(kNone, kNone, kNone, kNone);  // of the lane's child
  // the opening rule of lane's child c for its point, and the point's terms of
  // the four children in order; returns which points open which child
  auto eval = [&](int c, bool in) -> unsigned {
    float dx = 0.f, dy = 0.f, f = 0.f;
    bool acc = false, op = false, bucket = false;
    int b = 0, e = -1;
    if (in) {
      float r2c, kq = k;
      if (c < 0) {  // single point ~c
        const float2 q = spos[~c];
        dx = __fsub_rn(p.x, q.x);
        dy = __fsub_rn(p.y, q.y);
        r2c = fmaxf(__fmaf_rn(dx, dx, __fmul_rn(dy, dy)), md2);
        acc = ~c != s;
      } else {
        const float4 r0 = node[2 * c], r1 = node[2 * c + 1];
        kids = qchild[c];  // with the record, not after it: one round trip a cell
        dx = __fsub_rn(__fsub_rn(p.x, r0.x), r0.z);
        dy = __fsub_rn(__fsub_rn(p.y, r0.y), r0.w);
        r2c = fmaxf(__fmaf_rn(dx, dx, __fmul_rn(dy, dy)), md2);
        kq = __fmul_rn(k, fabsf(r1.x));
        // size^2 < 0 (a node standing for no quad level) is always opened
        acc = r1.y >= 0.f && r1.y < __fmul_rn(th2, r2c);
        op = !acc && r1.x > 0.f;
        bucket = !acc && !op;
        b = __float_as_int(r1.z);
        e = __float_as_int(r1.w);
      }
      const float inv = bh_rsqrt(r2c);
      f = __fmul_rn(__fmul_rn(__fmul_rn(kq, inv), inv), inv);
    }
    const unsigned b_acc = __ballot_sync(full, acc), b_bk = __ballot_sync(full, bucket);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float fh = __shfl_sync(full, f, own + h), xh = __shfl_sync(full, dx, own + h),
                  yh = __shfl_sync(full, dy, own + h);
      if ((b_acc >> (own + h)) & 1u) {
        fx = __fmaf_rn(fh, xh, fx);
        fy = __fmaf_rn(fh, yh, fy);
      }
      if (b_bk & (ones << h)) {  // warp-uniform: some point opens child h, a bucket
        const int bh = __shfl_sync(full, b, own + h), eh = __shfl_sync(full, e, own + h);
        if ((b_bk >> (own + h)) & 1u)
          for (int t = bh; t <= eh; ++t)
            if (t != s) bh_direct<false>(p.x, p.y, spos[t], k, md2, fx, fy);
        __syncwarp();
      }
    }
    return __ballot_sync(full, op);
  };
  if (n >= 2) {
    // the root, by the first lane of each point (lane 0's point always exists)
    const unsigned open = eval(0, valid && slot == 0) & ones;
    if (open) {
      if (lane == 0) {
        st_kids[w][0] = kids;
        st_mask[w][0] = open;
      }
      sp = 1;
    }
  }
  __syncwarp();
  while (sp > 0) {
    --sp;
    const int c = reinterpret_cast<const int *>(&st_kids[w][sp])[slot];
    const unsigned mask = st_mask[w][sp];
    __syncwarp();
    const unsigned ob = eval(c, c != kNone && ((mask >> own) & 1u));
    const unsigned om = (ob >> slot) & ones;  // the points that open this lane's child
    // pushed in reverse, so that the first opened child is popped first
    const unsigned opened = __ballot_sync(full, om != 0u) & 0xfu;
    const int np = __popc(opened);
    if (sp + np > Stack) {
      if (lane == 0) atomicOr(err, 1u);
      break;
    }
    // by the first point that opened the child: its lane has the grandchildren
    if (om != 0u && own == __ffs(om) - 1) {
      const int at = sp + __popc(opened >> (slot + 1));
      st_kids[w][at] = kids;
      st_mask[w][at] = om;
    }
    sp += np;
    __syncwarp();
  }
  if (valid && slot == 0) {
    force[perm[s]] = make_float2(fx, fy);
  }
}

// ---- batched walk (FX_BH_FAST) ----------------------------------------------
// The same cells, decisions and terms as the group walk, organised by cell
// instead of by point. Each warp owns 32 consecutive sorted points and a
// stack of opened cells: the quad children of each, and the lanes that opened
// it and so must evaluate them. A pass pops up to eight cells, a child per
// lane (popping single children instead costs a 32-lane scan of four ids per
// push); each lane first settles its entry for all 32 points at once from the
// box around them:
//   * accepted by all (the opening rule holds at the box's nearest point, with
//     a margin for the rounding of the per-point test; or a single point):
//     its term is added without any test, two entries per packed f32x2
//     instruction (entries that only some lanes must evaluate: one at a time,
//     masked);
//   * opened by all (the rule fails at the farthest point): its children are
//     pushed with its mask, and nothing is evaluated;
//   * neither: every lane evaluates it for its own point from broadcast reads,
//     adds the term if it accepts and votes who opens it, with the f32
//     operations of the group walk.
// Opened cells push their quad children with the opening lanes as the mask;
// opened buckets are walked point by point. Per point the interaction list is
// exactly the group walk's; the terms are added in another order.
// Issue-bound (75 % issue-active, ALU pipe 58 %): of the 613 entries of a warp
// at 1M uniform points 125 are accepted by all, 272 by a mask, 159 tested and
// 57 opened by all; testing every entry for every lane took 0.66 ms and
// 604M warp instructions, this 0.52 ms and 426M (300k points: 0.217, 0.174 ms).
// The stack holds kBatchStack cells (of up to four children; in a CPU model
// of this walk the children of uniform, clustered, line and radial sets of
// 20k-1M points peaked at 160-224): a warp whose stack would overflow starts over with
// the group walk, whose stacks are bounded, in the same shared memory.
constexpr int kBatchStack = 200;

// The stacked cells a warp may use (kBatchStack; less when the environment
// variable FLUXION_BH_BATCH_STACK asks for it, a test setting that sends more
// warps down the group-walk path).
static int batch_stack_cap() {
  static const int cap = [] {
    const char *e = std::getenv("FLUXION_BH_BATCH_STACK");
    const int v = e ? std::atoi(e) : kBatchStack;
    return std::min(kBatchStack, std::max(4, v));
  }();
  return cap;
}

// Whether the batched walk's arithmetic stays finite: it adds a point's term to
// itself as k / min_dist^3 times a zero difference, and lanes that take no part
// in an entry as 0 / d^3, with a reciprocal root that is infinite for a
// subnormal square. The group walk leaves both out, at any distance floor.
static bool batch_finite(float k, float md2) {
  const double inv = 1.0 / std::sqrt((double)md2);
  return md2 >= FLT_MIN && std::fabs((double)k) * inv * inv * inv < 0.25 * FLT_MAX;
}

// Two entries side by side, one half of each packed register: -x and -y of
// their centres (head and tail), k * mass, lane mask, size^2. 80 bytes, so
// that the lanes' stores to their halves conflict two ways at most.
struct alignas(16) EntryPair {
  uint64_t xh, yh;
  uint64_t xl, yl;
  uint64_t m, mask;
  uint64_t s2, self;  // self: (counting) the point of a single-point entry
  uint64_t pad[2];
};

struct BatchSmem {
  int4 kids[kBatchStack];      // an opened cell's quad children
  unsigned mask[kBatchStack];  // and the lanes that opened it
  EntryPair rec[16];           // the entries of a pass, two by two
  unsigned open_s[32];         // per entry: the lanes opening it
};
static_assert(kBatchStack * sizeof(int4) >= 2 * kWalkGroups * (kStackDeep + 1) * sizeof(int32_t),
              "the group walk's stacks must fit in a warp's batch stack");

// Blocks of one warp: its shared memory then lies at fixed addresses, which
// saves the instructions that find a warp's part of a block's (0.52 ms at 1M
// points against 0.56 and 0.57 with blocks of two and eight), and small
// designs reach every SM (43 against 47 us at 5k). 64 registers allow the SM
// all of the 32 blocks it can hold.
template <int Stack, bool Count>
__global__ void __launch_bounds__(32)
bh_batch_walk_kernel(int n, const float2 *__restrict__ spos, const int32_t *__restrict__ perm,
                     const int4 *__restrict__ qchild, const float4 *__restrict__ node,
                     float k, float th2, float md2, float2 *__restrict__ force,
                     unsigned int *__restrict__ err, int32_t *__restrict__ term_count,
                     int stack_cap) {
  __shared__ __align__(16) BatchSmem sh;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x;
  const int base = blockIdx.x * 32;
  const int s = base + lane;
  const bool valid = s < n;
  const unsigned lanebit = 1u << lane, lt = lanebit - 1u;
  const float2 p = valid ? spos[s] : make_float2(0.f, 0.f);
  const unsigned vm = __ballot_sync(full, valid);
  // the points' box: centre and half extents, grown by the rounding of both
  // and of the per-point differences; with a non-finite point nothing is
  // settled for all (the comparisons with an infinite extent fail)
  float bcx, bcy, bhx, bhy;
  {
    const float2 q = valid ? p : spos[base];
    float x0 = q.x, x1 = q.x, y0 = q.y, y1 = q.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x0 = fminf(x0, __shfl_xor_sync(full, x0, o));
      x1 = fmaxf(x1, __shfl_xor_sync(full, x1, o));
      y0 = fminf(y0, __shfl_xor_sync(full, y0, o));
      y1 = fmaxf(y1, __shfl_xor_sync(full, y1, o));
    }
    bcx = 0.5f * x0 + 0.5f * x1;
    bcy = 0.5f * y0 + 0.5f * y1;
    const float slack = 1e-6f * (fmaxf(fabsf(x0), fabsf(x1)) + fmaxf(fabsf(y0), fabsf(y1)));
    bhx = 0.5f * (x1 - x0) + slack;
    bhy = 0.5f * (y1 - y0) + slack;
    if (!__all_sync(full, isfinite(q.x) && isfinite(q.y))) bhx = bhy = __int_as_float(0x7f800000);
  }
  const float th2md2 = __fmul_rn(th2, md2);
  const float th2_lo = th2 * 0.999f, th2_hi = th2 * 1.001f;
  const uint64_t px2 = pack2(p.x, p.x), py2 = pack2(p.y, p.y);
  uint64_t fx2 = 0, fy2 = 0;
  float fx = 0.f, fy = 0.f;
  int terms = 0;
  int sp = 0;  // opened cells on the stack (warp-uniform)
  // the first pass evaluates the root alone, as the only child of a cell that
  // every point opened
  if (n >= 2) {
    if (lane == 0) {
      sh.kids[0] = make_int4(0, kNone, kNone, kNone);
      sh.mask[0] = vm;
    }
    sp = 1;
  }
  __syncwarp();
  bool overflow = stack_cap == 0;  // no batched walk at all (batch_finite)
  if (overflow) sp = 0;
  while (sp > 0) {
    // pop up to eight opened cells: lane l takes child l % 4 of cell l / 4
    const int cnt = min(sp, 8);
    sp -= cnt;
    int c = kNone, bf = 0, bl = -1;
    unsigned mask = 0u;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    float kq = 0.f, s2 = 0.f;
    bool bucket = false, all_acc = false, all_open = false;
    if (lane < 4 * cnt) {
      c = reinterpret_cast<const int *>(sh.kids + sp)[lane];
      mask = sh.mask[sp + (lane >> 2)];
    }
    const bool has = c != kNone;
    if (c >= 0) {
      a = node[2 * c];
      const float4 r1 = node[2 * c + 1];
      // size^2 < 0 (a node standing for no quad level): never accepted
      kq = __fmul_rn(k, fabsf(r1.x));
      s2 = r1.y >= 0.f ? r1.y : __int_as_float(0x7f800000);
      bucket = !(r1.x > 0.f);
      bf = __float_as_int(r1.z);
      bl = __float_as_int(r1.w);
      // squared distances from the centre of mass to the box's nearest and
      // farthest points
      const float ax = fabsf(a.x - bcx), ay = fabsf(a.y - bcy);
      const float slack = 1e-6f * (fabsf(a.x) + fabsf(a.y));
      const float nx = fmaxf(ax - bhx - slack, 0.f), ny = fmaxf(ay - bhy - slack, 0.f);
      const float qx = ax + bhx + slack, qy = ay + bhy + slack;
      all_acc = s2 < th2md2 || s2 < th2_lo * (nx * nx + ny * ny);
      all_open = !all_acc && s2 >= th2_hi * fmaxf(qx * qx + qy * qy, md2);
    } else if (has) {  // single point ~c: always accepted
      const float2 q = spos[~c];
      a = make_float4(q.x, q.y, 0.f, 0.f);
      kq = k;
      s2 = -1.f;
      all_acc = true;
    }
    // staged in one run: accepted by all, accepted by the lanes of a mask, to
    // be tested. A pair that straddles two kinds is treated as the later one,
    // which is right for both.
    const bool staged = has && !all_open;
    const unsigned b_all = __ballot_sync(full, all_acc && mask == vm);
    const unsigned b_acc = __ballot_sync(full, all_acc);
    const unsigned b_any = __ballot_sync(full, staged);
    const int n_all = __popc(b_all), n_acc = __popc(b_acc), n_any = __popc(b_any);
    int slot = 0;
    if (staged) {
      const unsigned bit = lanebit;
      slot = (b_all & bit) ? __popc(b_all & lt)
             : (b_acc & bit) ? n_all + __popc((b_acc & ~b_all) & lt)
                             : n_acc + __popc((b_any & ~b_acc) & lt);
      float *r = reinterpret_cast<float *>(&sh.rec[slot >> 1]) + (slot & 1);
      r[0] = -a.x;
      r[2] = -a.y;
      r[4] = -a.z;
      r[6] = -a.w;
      r[8] = kq;
      r[10] = __uint_as_float(mask);
      r[12] = s2;
      if (Count) r[14] = __int_as_float(c < 0 ? ~c : -1);
      if (slot + 1 == n_any && !(slot & 1)) {  // fill the last pair
        r[1] = r[3] = r[5] = r[7] = r[9] = r[11] = r[13] = 0.f;
        if (Count) r[15] = __int_as_float(-1);
      }
    }
    __syncwarp();
    // both entries' differences and squared distances
    auto pair_r = [&](const EntryPair &q, uint64_t &dx, uint64_t &dy) {
      dx = add2(add2(px2, q.xh), q.xl);
      dy = add2(add2(py2, q.yh), q.yl);
      const float2 r2 = unpack2(fma2(dx, dx, mul2(dy, dy)));
      return make_float2(fmaxf(r2.x, md2), fmaxf(r2.y, md2));
    };
    // their terms; m: k * mass, 0 where a lane takes none
    auto pair_add = [&](uint64_t m, float2 r2c, uint64_t dx, uint64_t dy) {
      // r2c >= md2, which batch_finite keeps normal
      const uint64_t inv = pack2(rsqrt_approx_ftz(r2c.x), rsqrt_approx_ftz(r2c.y));
      const uint64_t f = mul2(mul2(mul2(m, inv), inv), inv);
      fx2 = fma2(f, dx, fx2);
      fy2 = fma2(f, dy, fy2);
    };
    int j = 0;
#pragma unroll 2
    for (; j < (n_all >> 1); ++j) {
      const EntryPair &q = sh.rec[j];
      uint64_t dx, dy;
      const float2 r2c = pair_r(q, dx, dy);
      pair_add(q.m, r2c, dx, dy);
      if (Count) terms += ((int)(uint32_t)q.self != s) + ((int)(q.self >> 32) != s);
    }
#pragma unroll 2
    for (; j < (n_acc >> 1); ++j) {
      const EntryPair &q = sh.rec[j];
      uint64_t dx, dy;
      const float2 r2c = pair_r(q, dx, dy);
      const float2 m = unpack2(q.m);
      const bool in0 = ((uint32_t)q.mask & lanebit) != 0u;
      const bool in1 = ((uint32_t)(q.mask >> 32) & lanebit) != 0u;
      pair_add(pack2(in0 ? m.x : 0.f, in1 ? m.y : 0.f), r2c, dx, dy);
      if (Count)
        terms += (in0 && (int)(uint32_t)q.self != s) + (in1 && (int)(q.self >> 32) != s);
    }
#pragma unroll 2
    for (; 2 * j < n_any; ++j) {
      const EntryPair &q = sh.rec[j];
      uint64_t dx, dy;
      const float2 r2c = pair_r(q, dx, dy);
      const float2 m = unpack2(q.m), sq = unpack2(q.s2);
      const bool in0 = ((uint32_t)q.mask & lanebit) != 0u;
      const bool in1 = ((uint32_t)(q.mask >> 32) & lanebit) != 0u;
      const bool acc0 = sq.x < __fmul_rn(th2, r2c.x), acc1 = sq.y < __fmul_rn(th2, r2c.y);
      const unsigned o0 = __ballot_sync(full, in0 && !acc0);
      const unsigned o1 = __ballot_sync(full, in1 && !acc1);
      if (lane == 0) reinterpret_cast<uint64_t *>(sh.open_s)[j] = (uint64_t)o1 << 32 | o0;
      pair_add(pack2(in0 && acc0 ? m.x : 0.f, in1 && acc1 ? m.y : 0.f), r2c, dx, dy);
      if (Count)
        terms += (in0 && acc0 && (int)(uint32_t)q.self != s) +
                 (in1 && acc1 && (int)(q.self >> 32) != s);
    }
    __syncwarp();
    // the lanes that open this lane's cell
    const unsigned myopen = all_open ? mask : (staged && !all_acc) ? sh.open_s[slot] : 0u;
    // opened buckets: their points one by one
    unsigned bk = __ballot_sync(full, bucket && myopen != 0u);
    while (bk) {
      const int b = __ffs(bk) - 1;
      bk &= bk - 1u;
      const unsigned om = __shfl_sync(full, myopen, b);
      const int f = __shfl_sync(full, bf, b), l = __shfl_sync(full, bl, b);
      const bool in = (om & lanebit) != 0u;
      for (int t = f; t <= l; ++t) {
        const float2 q = spos[t];
        if (in && t != s) {
          bh_direct<true>(p.x, p.y, q, k, md2, fx, fy);
          if (Count) ++terms;
        }
      }
    }
    // opened cells: push their quad children with the opening lanes as mask
    const bool op = myopen != 0u && !bucket;
    const unsigned b_op = __ballot_sync(full, op);
    const int total = __popc(b_op);
    if (sp + total > stack_cap) {  // stack_cap <= kBatchStack
      overflow = true;
      break;
    }
    if (op) {
      const int at = sp + __popc(b_op & lt);
      sh.kids[at] = qchild[c];
      sh.mask[at] = myopen;
    }
    sp += total;
    __syncwarp();
  }
  if (overflow) {  // warp-uniform: start over with the bounded group walk
    __syncwarp();
    int32_t *mem = reinterpret_cast<int32_t *>(&sh.kids[0]);
    bh_group_walk<Stack, true, Count>(
        base, n, spos, perm, qchild, node, k, th2, md2, force, err, term_count,
        reinterpret_cast<int32_t(*)[Stack + 1]>(mem),
        reinterpret_cast<unsigned(*)[Stack + 1]>(mem + kWalkGroups * (Stack + 1)));
    return;
  }
  if (valid) {
    const float2 ax = unpack2(fx2), ay = unpack2(fy2);
    force[perm[s]] = make_float2(fx + (ax.x + ax.y), fy + (ay.x + ay.y));
    if (Count) term_count[perm[s]] = terms;
  }
}

static int bh_alloc(fx_design *d) {
  BHWork &b = d->bh;
  const int n = d->n;
  if (b.n == n && b.node.p) return FX_OK;
  const int T = (n + kSortTile - 1) / kSortTile;
  const size_t ni = n > 1 ? (size_t)n - 1 : 1;
  for (int i = 0; i < 2; ++i) {
    FX_TRY(b.keys[i].alloc(n));
    FX_TRY(b.idx[i].alloc(n));
  }
  FX_TRY(b.tile_hist.alloc((size_t)256 * T));
  FX_TRY(b.tile_scan.alloc((size_t)256 * T));
  FX_TRY(b.digit_total.alloc(256));
  FX_TRY(b.spos.alloc(n));
  FX_TRY(b.qchild.alloc(ni));
  FX_TRY(b.tile_fix.alloc(std::max(((size_t)n + kFixTile - 1) / kFixTile,
                                   ((size_t)std::min(n, kFixSmall) + 511) / 512)));
  FX_TRY(b.prefix.alloc(n));
  FX_TRY(b.node.alloc(2 * ni));
  FX_TRY(b.root.alloc(4));
  FX_TRY(b.bbox.alloc(8));
  FX_TRY(b.force.alloc(n));
  FX_TRY(b.os_ws.alloc(os_sort_words(n, 4)));
  b.n = n;
  return FX_OK;
}

static int bh_alloc_deep(fx_design *d) {
  BHWork &b = d->bh;
  const size_t n = (size_t)d->n;
  if (b.slo.p && b.slo.n >= n) return FX_OK;  // the last one
  FX_TRY(b.klo.alloc(n));
  FX_TRY(b.kl[0].alloc(n));
  FX_TRY(b.kl[1].alloc(n));
  FX_TRY(b.il[0].alloc(n));
  FX_TRY(b.il[1].alloc(n));
  FX_TRY(b.slo.alloc(n));
  return FX_OK;
}

// Whether the deep-key kernels can be needed: unless the positions are known
// to lie in the die and a level-15 cell of the largest possible root square,
// (die + 2) / 2^15, is accepted by every point (margins cover f32 rounding).
static bool bh_maybe_deep(const fx_design *d, float th2, float md2) {
  if (!d->pos_in_box) return true;
  const double rb = ((double)std::max(d->chip_w, d->chip_h) + 2.0) * (1.0 + 1e-6);
  const double s15 = rb / 32768.0;
  return s15 * s15 >= (double)th2 * (double)md2 * (1.0 - 1e-6);
}

// All buffers of bh_run on the design's present positions.
int bh_reserve(fx_design *d, float theta, float min_dist) {
  FX_TRY(bh_alloc(d));
  return bh_maybe_deep(d, theta * theta, min_dist * min_dist) ? bh_alloc_deep(d) : FX_OK;
}

// The walk's and the sort's error word (bh.bbox[4]) as a status.
int bh_error(unsigned int err) {
  if (err & 4u) {
    set_error("Barnes-Hut key sort: a bounded look-back wait expired");
    return FX_ETIMEOUT;
  }
  if (err) {
    set_error("Barnes-Hut walk stack overflow");
    return FX_EINVAL;
  }
  return FX_OK;
}

// Bounding box of the given positions into bh.bbox (re-armed first).
int bh_bbox(fx_ctx *ctx, fx_design *d, const float *x, const float *y,
            cudaStream_t s) {
  FX_TRY(bh_alloc(d));
  // {0xffffffff, 0xffffffff, 0, 0, 0}: min/max seeds of the ordered box and
  // a clear error word (memsets: no host buffer to stage)
  FX_CHECK_CUDA(cudaMemsetAsync(d->bh.bbox.p, 0xff, 8, s));
  FX_CHECK_CUDA(cudaMemsetAsync(d->bh.bbox.p + 2, 0, 12, s));
  int nb = (d->n + 255) / 256;
  if (nb > ctx->num_sms * 8) nb = ctx->num_sms * 8;
  bh_bbox_kernel<<<nb, 256, 0, s>>>(x, y, d->n, d->bh.bbox.p);
  FX_CHECK_LAUNCH();
  ctx->launches += 1;
  return FX_OK;
}

// Keys, sort and sorted positions of a design of any size (with the deep-key
// kernels when `deep`), by kernels of many blocks.
static int bh_sort_large(fx_ctx *ctx, fx_design *d, const float *x, const float *y, float th2,
                         float md2, bool deep, cudaStream_t s) {
  BHWork &b = d->bh;
  const int n = d->n, gb = (n + 255) / 256;
  const int T = (n + kSortTile - 1) / kSortTile;
  int launches = 0;
  cudaEvent_t ev;
  uint32_t *kk[2] = {b.keys[0].p, b.keys[1].p};
  int32_t *vv[2] = {b.idx[0].p, b.idx[1].p};
  timer_begin(ctx, FX_STAGE_BH_KEYS, s, &ev);
  if (!deep) {
    if (n >= (int)kOsVal) {
      set_error("Barnes-Hut sort: %d points out of range", n);
      return FX_EINVAL;
    }
    FX_CHECK_CUDA(cudaMemsetAsync(b.os_ws.p, 0, os_sort_words(n, 4) * 4, s));
    bh_keys_hist_kernel<<<(n + 256 * kKeysPer - 1) / (256 * kKeysPer), 256, 0, s>>>(
        x, y, n, b.bbox.p, th2, md2, b.root.p, b.keys[0].p, b.os_ws.p);
    FX_CHECK_LAUNCH();
    timer_end(ctx, FX_STAGE_BH_KEYS, s, ev);
    timer_begin(ctx, FX_STAGE_BH_SORT, s, &ev);
    // result in buffer 0; the last pass also gathers the sorted positions
    FX_TRY(os_passes(kk, vv, n, 4, b.os_ws.p, b.bbox.p + 4, s, x, y, b.spos.p, true));
    timer_end(ctx, FX_STAGE_BH_SORT, s, ev);
    ctx->launches += 5;
    return FX_OK;
  }
  bh_root_kernel<<<1, 1, 0, s>>>(b.bbox.p, b.root.p, th2, md2);
  FX_CHECK_LAUNCH();
  bh_keys_kernel<<<gb, 256, 0, s>>>(x, y, n, b.root.p, b.keys[0].p, b.idx[0].p, b.klo.p,
                                    b.kl[0].p, b.il[0].p);
  FX_CHECK_LAUNCH();
  launches += 2;
  timer_end(ctx, FX_STAGE_BH_KEYS, s, ev);
  timer_begin(ctx, FX_STAGE_BH_SORT, s, &ev);
  const float *gate = b.root.p;
  {
    // stable sort by the 24-bit sub-key (3 passes; no-ops unless root[3]),
    // then the primary keys and indices in that order into buffer 0
    for (int pass = 0; pass < 3; ++pass) {
      const int src = pass & 1, dst = src ^ 1;
      radix_hist_kernel<<<T, kSortThreads, 0, s>>>(b.kl[src].p, n, 8 * pass, b.tile_hist.p, T,
                                                   gate);
      radix_scan_kernel<<<256, 256, 0, s>>>(b.tile_hist.p, b.tile_scan.p, b.digit_total.p, T,
                                            gate);
      radix_scatter_kernel<<<T, kSortThreads, 0, s>>>(
          b.kl[src].p, b.il[src].p, b.kl[dst].p, b.il[dst].p, n, 8 * pass, b.tile_scan.p,
          b.digit_total.p, T, gate);
    }
    bh_deep_gather_kernel<<<gb, 256, 0, s>>>(gate, n, b.keys[0].p, b.il[1].p, b.keys[1].p,
                                             b.idx[1].p);
    bh_deep_copy_kernel<<<gb, 256, 0, s>>>(gate, n, b.keys[1].p, b.idx[1].p, b.keys[0].p,
                                           b.idx[0].p);
    FX_CHECK_LAUNCH();
    launches += 9 + 2;
  }
  // result in buffer 0; the last pass also gathers the sorted positions
  FX_TRY(radix_sort_onesweep(kk, vv, n, 4, b.os_ws.p, b.bbox.p + 4, s, x, y, b.spos.p));
  launches += 5;
  bh_deep_slo_kernel<<<gb, 256, 0, s>>>(gate, n, b.klo.p, b.idx[0].p, b.slo.p);
  ++launches;
  FX_CHECK_LAUNCH();
  timer_end(ctx, FX_STAGE_BH_SORT, s, ev);
  ctx->launches += launches;
  return FX_OK;
}

// Full Barnes-Hut force evaluation on the current positions; bh.bbox must
// hold their bounding box. Result: bh.force (original gate order).
int bh_run(fx_ctx *ctx, fx_design *d, float k, float theta, float min_dist, int walk,
           cudaStream_t s, int32_t *term_count) {
  FX_TRY(bh_alloc(d));
  BHWork &b = d->bh;
  const int n = d->n;
  const float *x = d->x[d->cur].p, *y = d->y[d->cur].p;
  unsigned int *err = b.bbox.p + 4;
  const float th2 = theta * theta, md2 = min_dist * min_dist;
  const bool deep = bh_maybe_deep(d, th2, md2);  // launch the deep-key kernels
  if (deep) FX_TRY(bh_alloc_deep(d));
  cudaEvent_t ev;
  int launches = 0;
  // Small designs: one cluster does keys and sort (fx_bh_sort.cu) up to its
  // capacity, where the device has room for it: 20 us at 5k points and 28 at
  // 10k against 69 and 73 for the seven launches of the many-block kernels.
  const bool one = !deep && bh_cluster_fits(ctx, n);
  if (one) {
    timer_begin(ctx, FX_STAGE_BH_SORT, s, &ev);
    FX_TRY(bh_cluster_sort(ctx, x, y, n, b.bbox.p, th2, md2, b.keys[0].p, b.idx[0].p, b.spos.p,
                           b.tile_fix.p, b.root.p, s));
    timer_end(ctx, FX_STAGE_BH_SORT, s, ev);
  } else {
    FX_TRY(bh_sort_large(ctx, d, x, y, th2, md2, deep, s));
  }
  timer_begin(ctx, FX_STAGE_BH_TREE, s, &ev);
  if (n >= 2) {
    // exact prefix sums, from tile sums (the cluster sort makes its own);
    // small tiles spread a small design over the SMs, but a block adds up all
    // earlier tiles' sums
    if (n <= kFixSmall) {
      const int tiles = (n + 511) / 512;
      if (!one) fix_tile_kernel<2><<<tiles, kFixThreads, 0, s>>>(b.spos.p, n, b.tile_fix.p);
      fix_prefix_kernel<2><<<tiles, kFixThreads, 0, s>>>(b.spos.p, n, b.tile_fix.p, b.prefix.p);
    } else {
      const int tiles = (n + kFixTile - 1) / kFixTile;
      fix_tile_kernel<kFixItems><<<tiles, kFixThreads, 0, s>>>(b.spos.p, n, b.tile_fix.p);
      fix_prefix_kernel<kFixItems><<<tiles, kFixThreads, 0, s>>>(b.spos.p, n, b.tile_fix.p,
                                                                 b.prefix.p);
    }
    launches += one ? 1 : 2;
    bh_build_kernel<<<(n - 1 + kBuildThreads - 1) / kBuildThreads, kBuildThreads, 0, s>>>(
        b.keys[0].p, deep ? b.slo.p : nullptr, b.root.p, b.bbox.p, n, b.prefix.p, b.node.p, b.qchild.p);
    ++launches;
  }
  FX_CHECK_LAUNCH();
  timer_end(ctx, FX_STAGE_BH_TREE, s, ev);
  timer_begin(ctx, FX_STAGE_BH_WALK, s, &ev);
  if (walk == FX_BH_EXACT && n <= (th2 < kPairsTheta2 ? kSmallWalkPairs : kSmallWalkMax)) {
    const int wb = (n + kSmallWarps * 8 - 1) / (kSmallWarps * 8);
    if (deep)
      bh_small_walk_kernel<kStackDeep><<<wb, kSmallWarps * 32, 0, s>>>(
          n, b.spos.p, b.idx[0].p, b.qchild.p, b.node.p, k, th2, md2, b.force.p, err);
    else
      bh_small_walk_kernel<kStack><<<wb, kSmallWarps * 32, 0, s>>>(
          n, b.spos.p, b.idx[0].p, b.qchild.p, b.node.p, k, th2, md2, b.force.p, err);
  } else if (walk == FX_BH_EXACT) {
    const int wb = (n + kWalkWarps * 32 - 1) / (kWalkWarps * 32);
    if (deep)
      bh_walk_kernel<kStackDeep><<<wb, kWalkWarps * 32, 0, s>>>(
          n, b.spos.p, b.idx[0].p, b.qchild.p, b.node.p, k, th2, md2, b.force.p, err);
    else
      bh_walk_kernel<kStack><<<wb, kWalkWarps * 32, 0, s>>>(
          n, b.spos.p, b.idx[0].p, b.qchild.p, b.node.p, k, th2, md2, b.force.p, err);
  } else {
    const int wb = (n + 31) / 32;
    const int cap = batch_finite(k, md2) ? batch_stack_cap() : 0;
#define FX_FAST_WALK(ST, CNT)                                                             \
  bh_batch_walk_kernel<ST, CNT><<<wb, 32, 0, s>>>(                                        \
      n, b.spos.p, b.idx[0].p, b.qchild.p, b.node.p, k, th2, md2, b.force.p, err, term_count, \
      cap)
    if (deep) {
      if (term_count) FX_FAST_WALK(kStackDeep, true);
      else FX_FAST_WALK(kStackDeep, false);
    } else {
      if (term_count) FX_FAST_WALK(kStack, true);
      else FX_FAST_WALK(kStack, false);
    }
#undef FX_FAST_WALK
  }
  FX_CHECK_LAUNCH();
  ++launches;
  timer_end(ctx, FX_STAGE_BH_WALK, s, ev);
  ctx->launches += launches;
  return FX_OK;
}

}  // namespace fx

using namespace fx;

namespace fx {
// The stage call's outputs in the caller's layout: forces as two arrays, keys
// in gate order (perm maps sorted position -> gate).
__global__ void bh_unpack_kernel(int n, const float2 *__restrict__ force,
                                 const uint32_t *__restrict__ skeys,
                                 const int32_t *__restrict__ perm, float *__restrict__ fx,
                                 float *__restrict__ fy, uint32_t *__restrict__ keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 f = force[i];
  fx[i] = f.x;
  fy[i] = f.y;
  keys[perm[i]] = skeys[i];
}
}  // namespace fx

extern "C" int fx_stage_barnes_hut_walk(fx_ctx *ctx, fx_design *d, float k, float theta,
                                        float min_dist, int32_t walk, float *out_fx,
                                        float *out_fy, uint32_t *out_keys, int32_t *out_perm,
                                        float *out_root, int32_t *out_terms) {
  if (!ctx || !d || !(theta >= 0.f) || !(min_dist > 0.f) ||
      (walk != FX_BH_FAST && walk != FX_BH_EXACT) || (out_terms && walk != FX_BH_FAST)) {
    set_error("fx_stage_barnes_hut: invalid arguments");
    return FX_EINVAL;
  }
  FX_CHECK_CUDA(cudaSetDevice(ctx->device));
  AllocScope alloc_scope(ctx->stream);
  cudaStream_t s = ctx->stream;
  const size_t n = (size_t)d->n;
  DevBuf<int32_t> terms;
  if (out_terms) FX_TRY(terms.alloc(n));
  FX_TRY(bh_bbox(ctx, d, d->x[d->cur].p, d->y[d->cur].p, s));
  FX_TRY(bh_run(ctx, d, k, theta, min_dist, walk, s, out_terms ? terms.p : nullptr));
  if (out_terms)
    FX_CHECK_CUDA(cudaMemcpyAsync(out_terms, terms.p, n * 4, cudaMemcpyDeviceToHost, s));
  // straight into the caller's arrays (unpacking on the host took 1.1 of 1.7 ms
  // at 300k points); the scratch is the stage's own force buffer and the sort's
  // second key buffer
  float *ux = reinterpret_cast<float *>(d->fattr.p), *uy = ux + n;
  uint32_t *uk = d->bh.keys[1].p;
  bh_unpack_kernel<<<((int)n + 255) / 256, 256, 0, s>>>((int)n, d->bh.force.p, d->bh.keys[0].p,
                                                        d->bh.idx[0].p, ux, uy, uk);
  FX_CHECK_LAUNCH();
  ctx->launches += 1;
  unsigned int err = 0;
  auto out = [&](void *dst, const void *src) {
    return dst ? cudaMemcpyAsync(dst, src, n * 4, cudaMemcpyDeviceToHost, s) : cudaSuccess;
  };
  FX_CHECK_CUDA(out(out_fx, ux));
  FX_CHECK_CUDA(out(out_fy, uy));
  FX_CHECK_CUDA(out(out_keys, uk));
  FX_CHECK_CUDA(out(out_perm, d->bh.idx[0].p));
  if (out_root)
    FX_CHECK_CUDA(cudaMemcpyAsync(out_root, d->bh.root.p, 12, cudaMemcpyDeviceToHost, s));
  FX_CHECK_CUDA(cudaMemcpyAsync(&err, d->bh.bbox.p + 4, 4, cudaMemcpyDeviceToHost, s));
  FX_CHECK_CUDA(cudaStreamSynchronize(s));
  FX_TRY(bh_error(err));
  return FX_OK;
}

extern "C" int fx_stage_barnes_hut(fx_ctx *ctx, fx_design *d, float k, float theta,
                                   float min_dist, float *out_fx, float *out_fy,
                                   uint32_t *out_keys, int32_t *out_perm, float *out_root) {
  return fx_stage_barnes_hut_walk(ctx, d, k, theta, min_dist, FX_BH_EXACT, out_fx, out_fy,
                                  out_keys, out_perm, out_root, nullptr);
}
