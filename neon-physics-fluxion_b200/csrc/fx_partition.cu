// fx_partition.cu -- (f.2) the hierarchy build: recursive spectral bisection
// (build_hierarchy, H/src/algorithm/partitioner.rs:36-100) on the device,
// plus the region pass of hapr_placement (H/src/algorithm/placer.rs:40-63,
// 111-141).
//
// The shape of the tree depends only on cluster sizes: a cluster of n gates
// is a leaf when n <= max_leaf_size or n <= min_cluster_size (:75), otherwise
// it splits at clamp(n/2, ceil(n*balance), n - ceil(n*balance)) (:197-212)
// into two halves. The host therefore lays out the whole tree up front; the
// device decides which gates go where. All clusters of one depth are
// processed together:
//   * every cluster is a contiguous segment of a gate permutation, left child
//     before right child, so the leaves come out in HierarchyTree::leaves()
//     order (hierarchy.rs:176-190);
//   * the power iteration runs on all clusters of the depth at once, on the
//     induced Laplacians (in-cluster adjacency entries in reference order);
//   * a stable segmented sort by Fiedler value (slice::sort_by with
//     partial_cmp, under which -0.0 == +0.0) reorders each segment, and the
//     split index cuts it into its two children.
// Two arithmetic modes:
//   FX_PART_EXACT  the reference's f32 iteration: v0 = sin(i * 2.71828) from
//                  the host's libm (the reference's f32::sin calls it too),
//                  sums of lv and lv^2 as sequential f32 folds (one warp per
//                  cluster, one lane adding), f32 mean / sqrt / divide:
//                  identical leaves.
//   FX_PART_FP64   f32 SpMV, FP64 chunked reductions (mean, norm, Rayleigh
//                  quotient), per-cluster stop once the Rayleigh quotient
//                  changes by <= tol (relative), at most power_iterations.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "fx_internal.h"

namespace fx {
namespace {

constexpr int kPartChunk = 4096;

// Index of the last entry of the sorted array a[0..C) that is <= x.
__device__ __forceinline__ int last_le(const int32_t *__restrict__ a, int C, int x) {
  int lo = 0, hi = C - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a[mid] <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Cluster of every position and gate at this depth (-1: not split here).
__global__ void part_fill_kernel(int n, const int32_t *__restrict__ perm,
                                 const int32_t *__restrict__ beg,
                                 const int32_t *__restrict__ end, int C,
                                 int32_t *__restrict__ clp, int32_t *__restrict__ clg) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int c = last_le(beg, C, p);
  const int cl = (beg[c] <= p && p < end[c]) ? c : -1;
  clp[p] = cl;
  clg[perm[p]] = cl;
}

// Degrees of the induced Laplacian (partitioner.rs:124-137: +1.0 per
// in-cluster adjacency entry) and the start vector v_i = sin(i * 2.71828).
__global__ void part_init_kernel(int n, const int32_t *__restrict__ perm,
                                 const int32_t *__restrict__ adj_ptr,
                                 const int32_t *__restrict__ adj_idx,
                                 const int32_t *__restrict__ clp,
                                 const int32_t *__restrict__ clg,
                                 const int32_t *__restrict__ beg,
                                 const float *__restrict__ sin_tab,
                                 float *__restrict__ deg, float *__restrict__ v) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int c = clp[p];
  if (c < 0) return;
  const int g = perm[p];
  int cnt = 0;
  for (int e = adj_ptr[g]; e < adj_ptr[g + 1]; ++e) cnt += clg[adj_idx[e]] == c;
  deg[p] = (float)cnt;
  v[p] = sin_tab[p - beg[c]];
}

// The depth's induced Laplacians as one CSR in position order: row p lists
// the positions of p's in-cluster neighbours in adjacency order, so the 30
// products of a depth read only in-cluster entries, row after row, instead
// of every adjacency entry through three gathers. Row lengths are the
// degrees part_init_kernel counted (0 outside the depth's clusters); an
// exclusive scan gives the row starts.
constexpr int kScanItems = 8, kScanTile = 256 * kScanItems;

__global__ void __launch_bounds__(256)
part_scan_tile_kernel(int n, const int32_t *__restrict__ clp, const float *__restrict__ deg,
                      int32_t *__restrict__ rp, int32_t *__restrict__ tsum) {
  __shared__ int32_t wsum[8];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int base = blockIdx.x * kScanTile + t * kScanItems;
  int c[kScanItems];
  int run = 0;
#pragma unroll
  for (int r = 0; r < kScanItems; ++r) {
    const int p = base + r;
    c[r] = p < n && clp[p] >= 0 ? (int)deg[p] : 0;
    run += c[r];
  }
  int x = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  int before = x - run;
  for (int q = 0; q < w; ++q) before += wsum[q];
#pragma unroll
  for (int r = 0; r < kScanItems; ++r) {
    const int p = base + r;
    if (p < n) rp[p] = before;
    before += c[r];
  }
  if (t == 255) tsum[blockIdx.x] = before;  // the tile's total
}

// Exclusive scan of the T tile totals in place (one block); tsum[T] = total.
__global__ void __launch_bounds__(1024)
part_scan_top_kernel(int T, int32_t *__restrict__ tsum) {
  __shared__ int32_t wsum[32];
  __shared__ int32_t carry_s;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) carry_s = 0;
  __syncthreads();
  for (int b0 = 0; b0 < T; b0 += 1024) {
    const int i = b0 + t;
    const int v = i < T ? tsum[i] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += u;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int y = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += u;
      }
      wsum[lane] = y;
    }
    __syncthreads();
    const int carry = carry_s;
    const int excl = carry + (w > 0 ? wsum[w - 1] : 0) + x - v;
    if (i < T) tsum[i] = excl;
    __syncthreads();
    if (t == 1023) carry_s = excl + v;
    __syncthreads();
  }
  if (t == 0) tsum[T] = carry_s;
}

__global__ void part_scan_add_kernel(int n, int T, const int32_t *__restrict__ tsum,
                                     int32_t *__restrict__ rp) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) rp[p] += tsum[p / kScanTile];
  if (p == 0) rp[n] = tsum[T];
}

__global__ void part_csr_kernel(int n, const int32_t *__restrict__ perm,
                                const int32_t *__restrict__ pos_of,
                                const int32_t *__restrict__ adj_ptr,
                                const int32_t *__restrict__ adj_idx,
                                const int32_t *__restrict__ clp,
                                const int32_t *__restrict__ beg,
                                const int32_t *__restrict__ end,
                                const int32_t *__restrict__ rp, int32_t *__restrict__ col) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int c = clp[p];
  if (c < 0) return;
  const int g = perm[p];
  int k = rp[p];
  // a cluster is a segment of positions
  const int b = beg[c], e = end[c];
  for (int q = adj_ptr[g], q1 = adj_ptr[g + 1]; q < q1; ++q) {
    const int t = pos_of[adj_idx[q]];
    if (t >= b && t < e) col[k++] = t;
  }
}

// lv = deg * v - A v in the reference's f32 order per row: deg*v first,
// then minus each in-cluster neighbour in adjacency order
// (partitioner.rs:158-165), over the depth's CSR.
__global__ void part_spmv_csr_kernel(int n, const int32_t *__restrict__ rp,
                                     const int32_t *__restrict__ col,
                                     const int32_t *__restrict__ clp,
                                     const int32_t *__restrict__ active,
                                     const float *__restrict__ deg,
                                     const float *__restrict__ v, float *__restrict__ lv) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int c = clp[p];
  if (c < 0 || !active[c]) return;
  float l = __fmul_rn(deg[p], v[p]);
  const int e1 = rp[p + 1];
  for (int e = rp[p]; e < e1; ++e) l = __fsub_rn(l, v[col[e]]);
  lv[p] = l;
}

}  // namespace

// FX_PART_EXACT reductions: sequential f32 folds in position order
// (Iterator::sum), one warp per cluster. The warp stages tiles of x in
// shared memory with coalesced loads and lane 0 folds each tile in order, so
// the fold is bound by the add latency rather than by global loads. With
// `deflate`: mean = sum(x) / n and x -= mean in place (:167-171); then
// norm = sqrt(sum(x*x)), kept as the divisor only when norm > 1e-10
// (:151-156, :174-180).
constexpr int kSeqTile = 2048;

__global__ void __launch_bounds__(32)
part_seq_kernel(int C, const int32_t *__restrict__ beg, const int32_t *__restrict__ end,
                float *__restrict__ x, int deflate, float *__restrict__ nrm) {
  __shared__ float tile[kSeqTile];
  const int c = blockIdx.x, lane = threadIdx.x;
  if (c >= C) return;
  const int b = beg[c], e = end[c];
  float mean = 0.f;
  if (deflate) {
    float s = 0.f;
    for (int t0 = b; t0 < e; t0 += kSeqTile) {
      const int m = min(kSeqTile, e - t0);
      for (int i = lane; i < m; i += 32) tile[i] = x[t0 + i];
      __syncwarp();
      if (lane == 0) {
#pragma unroll 16
        for (int i = 0; i < m; ++i) s = __fadd_rn(s, tile[i]);
      }
      __syncwarp();
    }
    mean = __fdiv_rn(__shfl_sync(0xffffffffu, s, 0), (float)(e - b));
  }
  float q = 0.f;
  for (int t0 = b; t0 < e; t0 += kSeqTile) {
    const int m = min(kSeqTile, e - t0);
    for (int i = lane; i < m; i += 32) tile[i] = x[t0 + i];
    __syncwarp();
    if (lane == 0) {
      if (deflate) {
#pragma unroll 16
        for (int i = 0; i < m; ++i) {
          const float y = __fsub_rn(tile[i], mean);
          tile[i] = y;
          q = __fadd_rn(q, __fmul_rn(y, y));
        }
      } else {
#pragma unroll 16
        for (int i = 0; i < m; ++i) q = __fadd_rn(q, __fmul_rn(tile[i], tile[i]));
      }
    }
    __syncwarp();
    if (deflate)
      for (int i = lane; i < m; i += 32) x[t0 + i] = tile[i];
    __syncwarp();
  }
  if (lane == 0) {
    const float norm = __fsqrt_rn(q);
    nrm[c] = norm > 1e-10f ? norm : 0.f;
  }
}

namespace {

// v = (x - mean) / norm, or without the division when the norm was too
// small, for the active clusters. x may be v.
__global__ void part_div_kernel(int n, const int32_t *__restrict__ clp,
                                const int32_t *__restrict__ active, const float *x,
                                const float *__restrict__ mean,
                                const float *__restrict__ nrm, float *v) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int c = clp[p];
  if (c < 0 || !active[c]) return;
  float y = x[p];
  if (mean) y = __fsub_rn(y, mean[c]);
  const float r = nrm[c];
  v[p] = r > 0.f ? __fdiv_rn(y, r) : y;
}

// FX_PART_FP64 sums of a cluster: s1 = sum x, s2 = sum x^2, s3 = sum v.x over
// chunks of kPartChunk positions, each chunk by 32 strided sequential sums and
// a shuffle tree, chunks added in order; every kernel below keeps this order.
__device__ __forceinline__ double tree_sum(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  return s;
}

// Mean and norm of a cluster of n positions (|x - mean|^2 = sum(x^2) - n
// mean^2: 1^T L v = 0, so no cancellation); without `deflate` (the start
// vector) the norm only. nrm 0 where it is too small to divide by.
__device__ __forceinline__ void mean_norm(double s1, double s2, double n, int deflate,
                                          float &mean, float &nrm) {
  const double m = deflate ? s1 / n : 0.0;
  const double var = deflate ? fmax(s2 - s1 * m, 0.0) : s2;
  const double norm = sqrt(var);
  mean = (float)m;
  nrm = norm > 1e-10 ? (float)norm : 0.f;
}

__device__ __forceinline__ float normed(float x, float mean, float nrm) {
  const float y = __fsub_rn(x, mean);
  return nrm > 0.f ? __fdiv_rn(y, nrm) : y;
}

// One warp per chunk (<= kPartChunk positions of one cluster) sums x, x^2
// and v.x in FP64; one thread per cluster then adds its chunks in order, so
// the reductions are deterministic.
__global__ void part_chunk_kernel(int K, const int32_t *__restrict__ ck_beg,
                                  const int32_t *__restrict__ ck_end,
                                  const int32_t *__restrict__ ck_cl,
                                  const int32_t *__restrict__ active,
                                  const float *__restrict__ x, const float *__restrict__ v,
                                  double *__restrict__ part) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (k >= K || !active[ck_cl[k]]) return;
  double s1 = 0.0, s2 = 0.0, s3 = 0.0;
  // eight loads in flight per lane, added in order
  const int e = ck_end[k];
  for (int p0 = ck_beg[k] + lane; p0 < e; p0 += 32 * 8) {
    float a8[8], v8[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int p = p0 + 32 * r;
      a8[r] = p < e ? x[p] : 0.f;
      v8[r] = v && p < e ? v[p] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (p0 + 32 * r >= e) break;
      const double a = (double)a8[r];
      s1 += a;
      s2 += a * a;
      if (v) s3 += (double)v8[r] * a;
    }
  }
  s1 = tree_sum(s1);
  s2 = tree_sum(s2);
  s3 = tree_sum(s3);
  if (lane == 0) {
    part[3 * k] = s1;
    part[3 * k + 1] = s2;
    part[3 * k + 2] = s3;
  }
}

// Mean and norm per cluster, the Rayleigh quotient v.Lv of the unit v, and
// the stop test.
__global__ void part_combine_kernel(int C, const int32_t *__restrict__ beg,
                                    const int32_t *__restrict__ end,
                                    const int32_t *__restrict__ cl_ck,
                                    const double *__restrict__ part, int deflate,
                                    double tol, int32_t *__restrict__ active,
                                    float *__restrict__ mean, float *__restrict__ nrm,
                                    double *__restrict__ lambda,
                                    int32_t *__restrict__ iters) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C || !active[c]) return;
  double s1 = 0.0, s2 = 0.0, s3 = 0.0;
  for (int k = cl_ck[c]; k < cl_ck[c + 1]; ++k) {
    s1 += part[3 * k];
    s2 += part[3 * k + 1];
    s3 += part[3 * k + 2];
  }
  mean_norm(s1, s2, (double)(end[c] - beg[c]), deflate, mean[c], nrm[c]);
  if (!deflate) return;
  const double prev = lambda[c];
  lambda[c] = s3;
  iters[c] += 1;
  if (tol > 0.0 && iters[c] > 1 && fabs(s3 - prev) <= tol * fabs(s3))
    active[c] = 2;  // converged: this update is the last
}

// ---- fixed iteration counts on clusters of several chunks --------------------
// Every power iteration of a depth in one cooperative launch. Per iteration:
// a block per chunk sums it (part), all blocks meet, each combines the chunks
// of the clusters its own positions lie in, multiplies (the inputs normalised
// as they are read, v_j = (x_j - mean) / norm: a division per neighbour, but
// no pass of its own over the vector), and all meet again. At 100k gates an
// iteration takes 7 to 10 us (22 with two launches each, whose longest rows,
// 129 neighbours in sequence, set the time): sums 2, meetings 1.5 each, the
// combination 1.3, the product 1.5 to 4. Bound by L2 round trips and a lane's
// 128 dependent FP64 sums. Blocks get even shares of positions and neighbours,
// not of positions: the order by Fiedler value gathers the hubs at the ends
// (9.9 us a product by positions, 4.3 by shares). A hierarchy of 100k gates
// takes 3.6 ms (5.4 before), of 1M 16.9.
constexpr int kPowerThreads = 512;
constexpr int kPowerClusters = 1024;      // clusters the positions of a block may span
constexpr int kPowerTile = kPartChunk / 4;  // chunk sums staged at a time
constexpr int kPowerEdges = 8192;           // neighbours gathered at a time
static_assert(kPowerEdges >= 2 * kPartChunk, "buf holds a chunk in FP64");
constexpr int kPowerPos = 8;  // work of a position, in neighbours
constexpr int kPowerSmem = 2 * kPowerEdges * 4;
constexpr int kMeetSpin = 1 << 22;        // polls before a block gives up (seconds)

// Polls a block may make at a meeting (kMeetSpin; less when the environment
// variable FLUXION_PART_MEET_POLLS asks for it, a test setting that makes the
// wait run out).
int meet_polls() {
  static const int polls = [] {
    const char *e = std::getenv("FLUXION_PART_MEET_POLLS");
    const int v = e ? std::atoi(e) : kMeetSpin;
    return std::min(kMeetSpin, std::max(1, v));
  }();
  return polls;
}

// Every block arrives and waits for the others, which a cooperative launch
// keeps resident; sync[0] counts arrivals (target: those so far and this
// meeting's), sync[1] is set by a block that gave up. True if all went well.
__device__ bool all_meet(unsigned int *sync, unsigned int target, int polls) {
  __syncthreads();
  bool bad = false;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sync) : "memory");
    int spin = 0;
    unsigned int seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(sync) : "memory");
    } while ((int)(seen - target) < 0 && ++spin < polls);
    bad = spin >= polls;
    if (bad) atomicExch(sync + 1, 1u);
  }
  return !__syncthreads_or(bad);
}

struct PowerArgs {
  int n, K, iterations, polls;  // positions, chunks
  const int32_t *ck_beg, *ck_end, *cl_ck, *beg, *end, *rp, *col, *clp;
  const float *deg;
  float *x, *y, *v;  // start vector in x; the last normalised vector goes to v
  double *part;      // [3K]
  unsigned int *sync;
};

__global__ void __launch_bounds__(kPowerThreads)
part_power_kernel(PowerArgs a) {
  extern __shared__ __align__(16) float power_sm[];
  float *buf = power_sm;  // [kPowerEdges]: a chunk, chunk sums or neighbours
  int32_t *col_s = reinterpret_cast<int32_t *>(power_sm + kPowerEdges);  // [kPowerEdges]
  __shared__ float mean_s[kPowerClusters], nrm_s[kPowerClusters];
  __shared__ int ca_s, cb_s;
  __shared__ int range[2];
  double *ps = reinterpret_cast<double *>(buf);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) {
    ca_s = INT_MAX;
    cb_s = -1;
  }
  // the block's positions: an even share of kPowerPos per position and one
  // per neighbour
  if (w < 2) {
    const long long all = (long long)kPowerPos * a.n + a.rp[a.n];
    const long long want = all * (blockIdx.x + w) / gridDim.x;
    int lo = 0, hi = a.n;  // the first p with kPowerPos * p + rp[p] >= want lies in [lo, hi]
    while (lo < hi) {      // 32 places a round, the last one short of hi
      const int step = (hi - lo + 31) / 32, p = min(hi - 1, lo + lane * step);
      const int below = __popc(__ballot_sync(
          0xffffffffu, (long long)kPowerPos * p + a.rp[p] < want));
      // places 0 .. below - 1 are too low
      const int last = below ? min(hi - 1, lo + (below - 1) * step) : lo;
      hi = below < 32 ? min(hi - 1, lo + below * step) : hi;
      lo = below ? last + 1 : lo;
    }
    if (lane == 0) range[w] = lo;
  }
  __syncthreads();
  const int p0 = range[0], p1 = range[1];
  for (int p = p0 + t; p < p1; p += kPowerThreads) {
    const int c = a.clp[p];
    if (c >= 0) {
      atomicMin(&ca_s, c);
      atomicMax(&cb_s, c);
    }
  }
  __syncthreads();
  // A share can hold no cluster: positions of leaves only, or none at all
  // beside a row longer than a share. Its range is then the empty [0, -1].
  const int cb = cb_s, ca = cb >= 0 ? ca_s : 0;
  const int kb = cb >= 0 ? a.cl_ck[ca] : 0, ke = cb >= 0 ? a.cl_ck[cb + 1] : 0;
  // all neighbours at hand in one go, their positions kept in shared memory
  const int r0 = a.rp[p0], edges = a.rp[p1] - r0;
  const bool fits = edges <= kPowerEdges;
  if (fits)
    for (int i = t; i < edges; i += kPowerThreads) col_s[i] = a.col[r0 + i];
  float *x = a.x, *y = a.y;
  unsigned int target = 0;
  for (int it = 0;; ++it) {
    // chunk sums: the chunk in one round of loads, then warp 0 sums x, warp 1 x^2
    for (int k = blockIdx.x; k < a.K; k += gridDim.x) {
      const int b = a.ck_beg[k], m = a.ck_end[k] - b;
      float u[kPartChunk / kPowerThreads];
#pragma unroll
      for (int r = 0; r < kPartChunk / kPowerThreads; ++r) {
        const int i = r * kPowerThreads + t;
        u[r] = i < m ? x[b + i] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < kPartChunk / kPowerThreads; ++r) ps[r * kPowerThreads + t] = (double)u[r];
      __syncthreads();
      if (w < 2) {
        double s = 0.0;
        if (w == 0) {
#pragma unroll 16
          for (int i = lane; i < m; i += 32) s += ps[i];
        } else {
#pragma unroll 16
          for (int i = lane; i < m; i += 32) s += ps[i] * ps[i];
        }
        s = tree_sum(s);
        if (lane == 0) a.part[3 * k + w] = s;
      }
      __syncthreads();
    }
    target += gridDim.x;
    if (!all_meet(a.sync, target, a.polls)) return;
    // mean and norm of the block's clusters, chunks added in order
    double s1[kPowerClusters / kPowerThreads] = {}, s2[kPowerClusters / kPowerThreads] = {};
    for (int k0 = kb; k0 < ke; k0 += kPowerTile) {
      const int k1 = min(ke, k0 + kPowerTile);
      for (int i = t; i < 2 * (k1 - k0); i += kPowerThreads)
        ps[i] = __ldcg(a.part + 3 * (size_t)(k0 + (i >> 1)) + (i & 1));
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kPowerClusters / kPowerThreads; ++r) {
        const int c = ca + r * kPowerThreads + t;
        if (c > cb) continue;
        const int q1 = min(k1, a.cl_ck[c + 1]);
#pragma unroll 4
        for (int q = max(k0, a.cl_ck[c]); q < q1; ++q) {
          s1[r] += ps[2 * (q - k0)];
          s2[r] += ps[2 * (q - k0) + 1];
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kPowerClusters / kPowerThreads; ++r) {
      const int i = r * kPowerThreads + t, c = ca + i;
      if (c <= cb)
        mean_norm(s1[r], s2[r], (double)(a.end[c] - a.beg[c]), it > 0, mean_s[i], nrm_s[i]);
    }
    __syncthreads();
    if (it == a.iterations) break;
    // y = L normed(x), in the order of part_spmv_csr_kernel: neighbours are
    // gathered and normalised edge by edge, then each position subtracts its
    // row; all of the block's at once where they fit, else those of
    // kPowerThreads positions a round, kPowerEdges at a time
    auto gather = [&](const int32_t *col, int t0, int t1, int &ec, int &ec_end) {
      for (int e = t0 + t; e < t1; e += 8 * kPowerThreads) {
        float g[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int f = e + q * kPowerThreads;
          g[q] = f < t1 ? x[col[f - t0]] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int f = e + q * kPowerThreads;
          if (f >= t1) break;
          while (f >= ec_end) ec_end = a.rp[a.end[++ec]];
          buf[f - t0] = normed(g[q], mean_s[ec - ca], nrm_s[ec - ca]);
        }
      }
    };
    auto subtract = [&](float l, const float *row, int m) {
      for (int f = 0; f < m; f += 8) {
        float g[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) g[q] = row[min(f + q, m - 1)];
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (f + q < m) l = __fsub_rn(l, g[q]);
      }
      return l;
    };
    int ec = ca, ec_end = cb >= 0 ? a.rp[a.end[ca]] : 0;  // cluster of the edge at hand
    if (fits) {
      int p = p0 + t, c = -1, e0 = 0, e1 = 0;
      float d = 0.f, xp = 0.f;
      auto load = [&] {
        if (p >= p1) return;
        c = a.clp[p], e0 = a.rp[p], e1 = a.rp[p + 1], d = a.deg[p], xp = x[p];
      };
      load();
      gather(col_s, r0, r0 + edges, ec, ec_end);
      __syncthreads();
      for (; p < p1; p += kPowerThreads, load()) {
        if (c < 0) continue;
        const float l = __fmul_rn(d, normed(xp, mean_s[c - ca], nrm_s[c - ca]));
        y[p] = subtract(l, buf + (e0 - r0), e1 - e0);
      }
    } else {
      for (int b0 = p0; b0 < p1; b0 += kPowerThreads) {
        const int p = b0 + t, b1 = min(p1, b0 + kPowerThreads);
        const int c = p < p1 ? a.clp[p] : -1;
        const int e0 = p < p1 ? a.rp[p] : 0, e1 = p < p1 ? a.rp[p + 1] : 0;
        float l = 0.f;
        if (c >= 0) l = __fmul_rn(a.deg[p], normed(x[p], mean_s[c - ca], nrm_s[c - ca]));
        const int te = a.rp[b1];
        for (int t0 = a.rp[b0]; t0 < te; t0 += kPowerEdges) {
          const int t1 = min(te, t0 + kPowerEdges);
          gather(a.col + t0, t0, t1, ec, ec_end);
          __syncthreads();
          const int f0 = max(e0, t0), f1 = min(e1, t1);
          if (f0 < f1) l = subtract(l, buf + (f0 - t0), f1 - f0);
          __syncthreads();
        }
        if (c >= 0) y[p] = l;
      }
    }
    target += gridDim.x;
    if (!all_meet(a.sync, target, a.polls)) return;
    float *o = x;
    x = y;
    y = o;
  }
  for (int p = p0 + t; p < p1; p += kPowerThreads) {
    const int c = a.clp[p];
    if (c >= 0) a.v[p] = normed(x[p], mean_s[c - ca], nrm_s[c - ca]);
  }
}

// take(map[idx[q]]) for q in [q0, q1) in order, 16 entries' loads in flight:
// the longest rows (129 neighbours at 100k gates) set the time of a block's
// row passes, two L2 round trips a batch (a depth 134 -> 127 us).
template <class F>
__device__ __forceinline__ void each_neighbour(const int32_t *__restrict__ idx, int q0, int q1,
                                               const int32_t *map, F take) {
  for (int q = q0; q < q1; q += 16) {
    int32_t j[16], m[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) j[u] = idx[min(q + u, q1 - 1)];
#pragma unroll
    for (int u = 0; u < 16; ++u) m[u] = map[j[u]];
#pragma unroll
    for (int u = 0; u < 16; ++u)
      if (q + u < q1) take(m[u]);
  }
}

// ---- a whole depth of clusters of one chunk each --------------------------------
// A block per cluster of at most kPartChunk positions does all that the depth
// does to it: the in-cluster CSR, every power iteration with the vectors in
// shared memory, the stable sort by Fiedler value (position breaks ties, so
// a bitonic sort of (key, place) pairs is stable) and the new order. One
// launch of 127 us (a depth of 100k gates, ncu cold; 141 with a warp per sum
// and mean and norm in every thread) instead of 4 * 30 + 25
// launches of 1.2 ms: the lower depths' clusters of some hundred gates left
// each launch waiting on one chain of sums. Bound by that chain (a lane's 128
// dependent FP64 sums) and the barriers of 30 iterations. The sums keep the
// chunked kernels' order, so the orders that come out are the same.
// In its own segment a block overwrites perm and pos_of; other blocks only ask
// whether a gate's place lies in their own segment, which no write changes.
__host__ __device__ inline int pow2_above(int n) {
  int p = 32;
  while (p < n) p <<= 1;
  return p;
}
// In-cluster neighbours per cluster up to which that pays, with a fixed count
// and with the stop rule. One block goes through them in each iteration (0.3 ns
// a neighbour) where the kernels above spread them over the device. Whole calls,
// ms, here against everything above: 2,500 gates of 21 neighbours 0.9 and 1.9,
// of 51 1.7 and 1.1 (stop rule: 1.7 and 1.9), of 446 16 and 2.8 (16 and 6.4);
// 4,096 of 3,509 180 and 16 (180 and 28).
constexpr int64_t kSmallEdges = 1 << 16, kSmallEdgesStop = 1 << 18;

// Rows so long that the one-launch form is the slower: a tile of its neighbours
// holds few rows, each one lane's chain, and there are many tiles. 30,000 gates
// of 6,993 neighbours 246 ms, stepped 90; of 1,172 28 and 29.
constexpr int64_t kDenseEdges = 1 << 24;
constexpr int kDenseRow = 512;
static bool dense_rows(double per_gate, int64_t positions) {
  return per_gate * (double)positions > kDenseEdges && per_gate > kDenseRow;
}
static size_t part_small_smem(int most) {
  return (size_t)pow2_above(most) * 8 + (size_t)most * 8 + ((size_t)most + 1) * 4;
}

__global__ void __launch_bounds__(1024)
part_small_kernel(const int32_t *__restrict__ beg, const int32_t *__restrict__ end, int most,
                  const int32_t *__restrict__ adj_ptr, const int32_t *__restrict__ adj_idx,
                  const float *__restrict__ sin_tab, int iterations, double tol,
                  int32_t *perm, int32_t *pos_of, uint16_t *__restrict__ col,
                  unsigned int *__restrict__ total, unsigned long long *__restrict__ iters) {
  extern __shared__ __align__(16) unsigned char raw[];
  uint64_t *key = reinterpret_cast<uint64_t *>(raw);
  float *v = reinterpret_cast<float *>(key + pow2_above(most));
  float *lv = v + most;
  int32_t *rp = reinterpret_cast<int32_t *>(lv + most);
  __shared__ int32_t wsum[32];
  __shared__ unsigned int base_sh;
  __shared__ double lambda_sh;
  __shared__ float mean_sh, nrm_sh;
  double *ld = reinterpret_cast<double *>(key);  // lv in FP64; the keys come after the iterations
  const int T = blockDim.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int b = beg[blockIdx.x], e = end[blockIdx.x], n = e - b;
  // in-cluster CSR: counts, row starts, columns (local places)
  for (int i = t; i < n; i += T) {
    const int g = perm[b + i], q1 = adj_ptr[g + 1];
    int c = 0;
    each_neighbour(adj_idx, adj_ptr[g], q1, pos_of,
                   [&](int p) { c += (unsigned)(p - b) < (unsigned)n; });
    rp[i + 1] = c;
  }
  __syncthreads();
  const int per = (n + T - 1) / T, i0 = min(n, t * per), i1 = min(n, i0 + per);
  int run = 0;
  for (int i = i0; i < i1; ++i) run += rp[i + 1];
  int inc = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  int at = inc - run;
  for (int q = 0; q < w; ++q) at += wsum[q];
  for (int i = i0; i < i1; ++i) {
    at += rp[i + 1];
    rp[i + 1] = at;
  }
  if (t == 0) rp[0] = 0;
  __syncthreads();
  if (t == 0) base_sh = atomicAdd(total, (unsigned int)rp[n]);
  __syncthreads();
  uint16_t *mine = col + base_sh;
  for (int i = t; i < n; i += T) {
    const int g = perm[b + i], q1 = adj_ptr[g + 1];
    int k = rp[i];
    each_neighbour(adj_idx, adj_ptr[g], q1, pos_of, [&](int p) {
      if ((unsigned)(p - b) < (unsigned)n) mine[k++] = (uint16_t)(p - b);
    });
    lv[i] = sin_tab[i];
    ld[i] = (double)lv[i];
  }
  __syncthreads();
  // warp 0 sums x = lv and x^2 (two chains at once, from FP64 copies) and
  // has mean and norm; warp 1 sums v.x where the stop test asks for it
  auto reduce = [&](int deflate) {
    if (w == 0) {
      double s1 = 0.0, s2 = 0.0;
#pragma unroll 16
      for (int i = lane; i < n; i += 32) {
        const double a = ld[i];
        s1 += a;
        s2 += a * a;
      }
      s1 = tree_sum(s1);
      s2 = tree_sum(s2);
      if (lane == 0) mean_norm(0.0 + s1, 0.0 + s2, (double)n, deflate, mean_sh, nrm_sh);
    } else if (w == 1 && deflate && tol > 0.0) {
      double s = 0.0;
#pragma unroll 8
      for (int i = lane; i < n; i += 32) s += (double)v[i] * ld[i];
      s = tree_sum(s);
      if (lane == 0) lambda_sh = 0.0 + s;
    }
    __syncthreads();
  };
  auto normalise = [&] {
    const float m = mean_sh, r = nrm_sh;
    for (int i = t; i < n; i += T) v[i] = normed(lv[i], m, r);
    __syncthreads();
  };
  reduce(0);
  normalise();
  double lambda = 0.0;
  int it = 0;
  while (it < iterations) {
    for (int i = t; i < n; i += T) {
      const int k1 = rp[i + 1], k0 = rp[i];
      float l = __fmul_rn((float)(k1 - k0), v[i]);
      for (int k = k0; k < k1; k += 8) {
        int j[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) j[q] = k + q < k1 ? mine[k + q] : i;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (k + q < k1) l = __fsub_rn(l, v[j[q]]);
      }
      lv[i] = l;
      ld[i] = (double)l;
    }
    __syncthreads();
    reduce(1);
    ++it;
    const double prev = lambda;
    if (tol > 0.0) lambda = lambda_sh;
    const bool stop = tol > 0.0 && it > 1 && fabs(lambda - prev) <= tol * fabs(lambda);
    normalise();  // a converged cluster takes this update as its last
    if (stop) break;
  }
  if (t == 0 && it > 0) atomicAdd(iters, (unsigned long long)it);
  // stable sort by value (-0.0 as +0.0), then the new order
  const int P = pow2_above(n);
  for (int i = t; i < P; i += T) {
    uint64_t k = ~0ull;
    if (i < n) {
      float f = v[i];
      if (f == 0.f) f = 0.f;
      const uint32_t u = __float_as_uint(f);
      k = (uint64_t)((u & 0x80000000u) ? ~u : (u | 0x80000000u)) << 32 | (uint32_t)i;
    }
    key[i] = k;
  }
  __syncthreads();
  for (int size = 2; size <= P; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int j = t; j < P / 2; j += T) {
        const int lo = 2 * j - (j & (stride - 1)), hi = lo + stride;
        const uint64_t x = key[lo], y = key[hi];
        if ((x > y) == ((lo & size) == 0)) {
          key[lo] = y;
          key[hi] = x;
        }
      }
      __syncthreads();
    }
  int32_t *gate = reinterpret_cast<int32_t *>(lv);
  for (int i = t; i < n; i += T) gate[i] = perm[b + i];
  __syncthreads();
  for (int i = t; i < n; i += T) {
    const int g = gate[(uint32_t)key[i]];
    perm[b + i] = g;
    pos_of[g] = b + i;
  }
}

__global__ void part_retire_kernel(int C, int32_t *__restrict__ active,
                                   int32_t *__restrict__ any) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  if (active[c] == 2) active[c] = 0;
  if (active[c]) atomicOr(any, 1);
}

// Sort input for the A positions of the bisected clusters, packed cluster
// by cluster (slot t of cluster c <-> position beg[c] + t - off[c]): the
// Fiedler value as an order-preserving uint32 (-0.0 read as +0.0, so equal
// values keep their order), the slot as the value.
__global__ void part_keys_kernel(int A, int C, const int32_t *__restrict__ beg,
                                 const int32_t *__restrict__ off,
                                 const float *__restrict__ v, uint32_t *__restrict__ key,
                                 int32_t *__restrict__ slot_pos, int32_t *__restrict__ val) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A) return;
  const int c = last_le(off, C, t);
  const int p = beg[c] + (t - off[c]);
  float f = v[p];
  if (f == 0.f) f = 0.f;
  const uint32_t u = __float_as_uint(f);
  key[t] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  slot_pos[t] = p;
  val[t] = t;
}

// After the value sort: the cluster of each slot's source, as the next key.
__global__ void part_major_kernel(int A, int C, const int32_t *__restrict__ val,
                                  const int32_t *__restrict__ off,
                                  uint32_t *__restrict__ key) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A) return;
  key[t] = (uint32_t)last_le(off, C, val[t]);
}

// Slot t now holds source slot val[t]: that gate moves to slot t's position.
__global__ void part_apply_kernel(int A, const int32_t *__restrict__ val,
                                  const int32_t *__restrict__ slot_pos,
                                  const int32_t *__restrict__ perm_in,
                                  int32_t *__restrict__ perm_out,
                                  int32_t *__restrict__ pos_of) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A) return;
  const int dst = slot_pos[t];
  const int g = perm_in[slot_pos[val[t]]];
  perm_out[dst] = g;
  pos_of[g] = dst;
}

struct PNode {
  int32_t beg, end, depth, left = -1, right = -1;
  float cx = 0.f, cy = 0.f, w = 0.f, h = 0.f;
};

// The tree of sizes (recursive_bisect, partitioner.rs:64-100), nodes in
// pre-order (the reference's next_id order).
int32_t build_shape(std::vector<PNode> &nodes, int32_t beg, int32_t end, int32_t depth,
                    const fx_part_cfg &cfg) {
  const int32_t id = (int32_t)nodes.size();
  PNode nd;
  nd.beg = beg;
  nd.end = end;
  nd.depth = depth;
  nodes.push_back(nd);
  const int32_t n = end - beg;
  if (n <= cfg.max_leaf_size || n <= cfg.min_cluster_size) return id;
  // split_by_fiedler (:197-212): min_size = (n as f32 * balance).ceil() as usize
  const float fm = std::ceil((float)n * cfg.balance_factor);
  const int64_t min_size = fm > 0.f ? (int64_t)fm : 0;
  int64_t split = n / 2;
  split = std::max<int64_t>(split, min_size);
  split = std::min<int64_t>(split, (int64_t)n - min_size);
  if (split <= 0 || split >= n) return id;  // an empty half: the cluster stays a leaf
  const int32_t l = build_shape(nodes, beg, beg + (int32_t)split, depth + 1, cfg);
  const int32_t r = build_shape(nodes, beg + (int32_t)split, end, depth + 1, cfg);
  nodes[id].left = l;
  nodes[id].right = r;
  return id;
}

// place_level_recursive (placer.rs:111-141) for two children: cols =
// ceil(sqrt(2)) = 2 and rows = 1, so each child gets one column of its
// parent, in the reference's f32 operations.
void place_regions(std::vector<PNode> &nodes, int32_t id) {
  const PNode nd = nodes[id];
  if (nd.left < 0) return;
  const int32_t kids[2] = {nd.left, nd.right};
  const size_t cnt = 2;
  const float half_w = nd.w / 2.0f, half_h = nd.h / 2.0f;
  const float ox = nd.cx - half_w, oy = nd.cy - half_h;
  const size_t cols = (size_t)std::ceil(std::sqrt((float)cnt));
  const size_t rows = (cnt + cols - 1) / cols;
  for (size_t i = 0; i < cnt; ++i) {
    const size_t col = i % cols, row = i / cols;
    const float cw = nd.w / (float)cols;
    const float ch = nd.h / (float)rows;
    PNode &c = nodes[kids[i]];
    c.cx = ox + ((float)col + 0.5f) * cw;
    c.cy = oy + ((float)row + 0.5f) * ch;
    c.w = cw;
    c.h = ch;
  }
  place_regions(nodes, nd.left);
  place_regions(nodes, nd.right);
}

template <class T>
int upload(DevBuf<T> &d, const std::vector<T> &h, cudaStream_t s) {
  FX_TRY(d.alloc(h.empty() ? 1 : h.size()));
  if (!h.empty())
    FX_CHECK_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T),
                                  cudaMemcpyHostToDevice, s));
  return FX_OK;
}

}  // namespace
}  // namespace fx

using namespace fx;

extern "C" int fx_part_cfg_default(fx_part_cfg *c) {
  if (!c) return FX_EINVAL;
  // PartitionConfig::default (partitioner.rs:24-32) with the power-iteration
  // count main.rs:80 passes; the FP64 mode's tolerance.
  c->max_leaf_size = 64;
  c->min_cluster_size = 8;
  c->balance_factor = 0.4f;
  c->power_iterations = 30;
  c->mode = FX_PART_EXACT;
  c->reserved0 = 0;
  c->tol = 1e-6;
  return FX_OK;
}

extern "C" int fx_partition(fx_ctx *ctx, fx_design *d, const fx_part_cfg *cfg,
                            int32_t leaf_capacity, int32_t *out_leaf_ptr,
                            int32_t *out_leaf_gate, float *out_region,
                            int32_t *out_leaf_depth, fx_part_stats *out_stats) {
  if (!ctx || !d || !cfg || cfg->max_leaf_size < 1 || cfg->min_cluster_size < 0 ||
      !(cfg->balance_factor >= 0.f && cfg->balance_factor <= 0.5f) ||
      cfg->power_iterations < 0 ||
      (cfg->mode != FX_PART_EXACT && cfg->mode != FX_PART_FP64) || !(cfg->tol >= 0.0) ||
      leaf_capacity < 0) {
    set_error("fx_partition: invalid arguments");
    return FX_EINVAL;
  }
  const int32_t N = d->n;
  std::vector<PNode> nodes;
  if (N > 0) build_shape(nodes, 0, N, 0, *cfg);
  int32_t max_depth = 0, n_leaves = 0, levels = 0, max_active = 0;
  for (const PNode &nd : nodes) {
    if (nd.left < 0) {
      ++n_leaves;
      max_depth = std::max(max_depth, nd.depth);
    } else {
      levels = std::max(levels, nd.depth + 1);
      max_active = std::max(max_active, nd.end - nd.beg);
    }
  }
  if (n_leaves > leaf_capacity && (out_leaf_ptr || out_region || out_leaf_depth)) {
    set_error("fx_partition: the tree has %d leaves, capacity %d", n_leaves, leaf_capacity);
    return FX_EINVAL;
  }
  FX_CHECK_CUDA(cudaSetDevice(ctx->device));
  AllocScope alloc_scope(ctx->stream);
  cudaStream_t s = ctx->stream;
  const bool exact = cfg->mode == FX_PART_EXACT;
  int64_t total_iters = 0;
  DevBuf<int32_t> perm[2], pos_of;
  int cur = 0;
  if (N > 0) {
    std::vector<int32_t> iota((size_t)N);
    for (int32_t i = 0; i < N; ++i) iota[i] = i;
    FX_TRY(upload(perm[0], iota, s));
    FX_TRY(upload(pos_of, iota, s));
    FX_TRY(perm[1].alloc(N));
  }
  if (levels > 0) {
    // the reference's start vector, from the host libm (as f32::sin); the table
    // depends on nothing else, so the context keeps the longest one made
    DevBuf<float> &d_sin = ctx->sin_tab;
    if (d_sin.n < (size_t)max_active) {
      std::vector<float> sin_tab((size_t)max_active);
      for (int32_t i = 0; i < max_active; ++i) sin_tab[i] = std::sin((float)i * 2.71828f);
      if (upload(d_sin, sin_tab, s) != FX_OK || cudaStreamSynchronize(s) != cudaSuccess) {
        d_sin.release();
        set_error("fx_partition: start vector upload failed");
        return FX_ECUDA;
      }
    }
    DevBuf<float> deg, v, lv, mean, nrm;
    DevBuf<int32_t> clp, clg, beg, end, off, act, iters, any, ck_beg, ck_end, ck_cl, cl_ck;
    DevBuf<double> part, lambda;
    DevBuf<uint32_t> keys[2], th, ts, dt;
    DevBuf<int32_t> vals[2], slot_pos;
    DevBuf<float> lv2;
    DevBuf<unsigned int> counters;         // block arrivals, gave up; CSR entries
    DevBuf<unsigned long long> small_its;  // iterations of the one-chunk depths
    FX_TRY(counters.alloc(3));
    FX_TRY(small_its.alloc(1));
    FX_CHECK_CUDA(cudaMemsetAsync(counters.p, 0, 12, s));
    FX_CHECK_CUDA(cudaMemsetAsync(small_its.p, 0, 8, s));
    FX_TRY(clp.alloc(N));
    FX_TRY(clg.alloc(N));
    FX_TRY(deg.alloc(N));
    FX_TRY(v.alloc(N));
    FX_TRY(lv.alloc(N));
    FX_TRY(keys[0].alloc(N));
    FX_TRY(keys[1].alloc(N));
    FX_TRY(vals[0].alloc(N));
    FX_TRY(vals[1].alloc(N));
    FX_TRY(slot_pos.alloc(N));
    FX_TRY(th.alloc((size_t)256 * radix_sort_tiles(N)));
    FX_TRY(ts.alloc((size_t)256 * radix_sort_tiles(N)));
    FX_TRY(dt.alloc(256));
    FX_TRY(any.alloc(1));
    const int nb = (N + 255) / 256;
    // the depth's in-cluster CSR: row starts, tile totals, neighbour positions
    const int st = (N + kScanTile - 1) / kScanTile;
    DevBuf<int32_t> rp, tsum, col;
    FX_TRY(rp.alloc((size_t)N + 1));
    FX_TRY(tsum.alloc((size_t)st + 1));
    FX_TRY(col.alloc(std::max<size_t>(d->adj_idx.n, 1)));
    // in-cluster neighbours a gate: the design's mean (a depth's is mostly
    // lower), or the last depth's own where that was asked for
    double per_gate = (double)d->a / (double)N;
    for (int32_t depth = 0; depth < levels; ++depth) {
      // the clusters bisected at this depth, in position order (pre-order
      // lists them left to right within a depth)
      std::vector<int32_t> hb, he, hoff;
      int32_t A = 0;
      for (const PNode &nd : nodes)
        if (nd.depth == depth && nd.left >= 0) {
          hb.push_back(nd.beg);
          he.push_back(nd.end);
          hoff.push_back(A);
          A += nd.end - nd.beg;
        }
      const int C = (int)hb.size();
      if (C == 0) continue;
      FX_TRY(upload(beg, hb, s));
      FX_TRY(upload(end, he, s));
      int32_t most = 0;
      for (int c = 0; c < C; ++c) most = std::max(most, he[c] - hb[c]);
      const int64_t small_edges = cfg->tol > 0.0 ? kSmallEdgesStop : kSmallEdges;
      // of a cluster: by the mean, and at most all its pairs
      auto cluster_edges = [&](double gates) { return std::min(gates, per_gate) * gates; };
      if (!exact && most <= kPartChunk && cluster_edges(most) <= (double)small_edges) {
        // one block per cluster; two to four positions a thread
        const size_t smem = part_small_smem(most);
        const int threads = std::min(1024, std::max(96, (most / 2 + 31) / 32 * 32));
        FX_TRY(raise_smem_limit((const void *)part_small_kernel, (int)smem));
        FX_CHECK_CUDA(cudaMemsetAsync(counters.p + 2, 0, 4, s));
        part_small_kernel<<<C, threads, smem, s>>>(
            beg.p, end.p, most, d->adj_ptr.p, d->adj_idx.p, d_sin.p, cfg->power_iterations,
            cfg->tol, perm[cur].p, pos_of.p, reinterpret_cast<uint16_t *>(col.p),
            counters.p + 2, small_its.p);
        FX_CHECK_LAUNCH();
        ctx->launches += 1;
        FX_CHECK_CUDA(cudaStreamSynchronize(s));  // beg and end are reused
        continue;
      }
      FX_TRY(upload(off, hoff, s));
      FX_TRY(upload(act, std::vector<int32_t>((size_t)C, 1), s));
      FX_TRY(mean.alloc(C));
      FX_TRY(nrm.alloc(C));
      FX_TRY(lambda.alloc(C));
      FX_TRY(iters.alloc(C));
      FX_CHECK_CUDA(cudaMemsetAsync(lambda.p, 0, (size_t)C * 8, s));
      FX_CHECK_CUDA(cudaMemsetAsync(iters.p, 0, (size_t)C * 4, s));
      int K = 0;
      if (!exact) {
        std::vector<int32_t> hcb, hce, hcc, hclck((size_t)C + 1, 0);
        for (int c = 0; c < C; ++c) {
          for (int32_t p = hb[c]; p < he[c]; p += kPartChunk) {
            hcb.push_back(p);
            hce.push_back(std::min(p + kPartChunk, he[c]));
            hcc.push_back(c);
          }
          hclck[(size_t)c + 1] = (int32_t)hcb.size();
        }
        K = (int)hcb.size();
        FX_TRY(upload(ck_beg, hcb, s));
        FX_TRY(upload(ck_end, hce, s));
        FX_TRY(upload(ck_cl, hcc, s));
        FX_TRY(upload(cl_ck, hclck, s));
        FX_TRY(part.alloc((size_t)3 * K));
      }
      const int cb = (C + 63) / 64, kb = (K * 32 + 255) / 256;
      part_fill_kernel<<<nb, 256, 0, s>>>(N, perm[cur].p, beg.p, end.p, C, clp.p, clg.p);
      part_init_kernel<<<nb, 256, 0, s>>>(N, perm[cur].p, d->adj_ptr.p, d->adj_idx.p, clp.p,
                                          clg.p, beg.p, d_sin.p, deg.p, v.p);
      part_scan_tile_kernel<<<st, 256, 0, s>>>(N, clp.p, deg.p, rp.p, tsum.p);
      part_scan_top_kernel<<<1, 1024, 0, s>>>(st, tsum.p);
      part_scan_add_kernel<<<nb, 256, 0, s>>>(N, st, tsum.p, rp.p);
      part_csr_kernel<<<nb, 256, 0, s>>>(N, perm[cur].p, pos_of.p, d->adj_ptr.p, d->adj_idx.p,
                                         clp.p, beg.p, end.p, rp.p, col.p);
      ctx->launches += 4;
      // a fixed count in one launch, where a block's positions span few enough
      // clusters (clusters of a depth differ by one position, so up to 1e8 gates)
      int least = N, per_sm = 0;
      for (int c = 0; c < C; ++c) least = std::min(least, he[c] - hb[c]);
      FX_TRY(raise_smem_limit((const void *)part_power_kernel, kPowerSmem));
      FX_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, part_power_kernel,
                                                                  kPowerThreads, kPowerSmem));
      // blocks an SM so that a block's share fits its shared memory, if it can
      const int64_t work = (int64_t)kPowerPos * N + d->a;
      const int64_t share = (int64_t)ctx->num_sms * (kPowerEdges - kPowerEdges / 8);
      const int grid = ctx->num_sms * (int)std::min<int64_t>(per_sm, (work + share - 1) / share);
      // positions of a block: its share, all positions without neighbours
      const int64_t per = grid > 0 ? ((int64_t)N + d->a / kPowerPos) / grid + 2 : N;
      bool fixed = !exact && cfg->tol <= 0.0 && grid > 0 && per / least + 2 <= kPowerClusters &&
                   !dense_rows(per_gate, A);
      if (fixed) {
        FX_TRY(lv2.alloc(N));
        // the start vector is in v: x = v, and v gets the last one
        FX_CHECK_CUDA(cudaMemcpyAsync(lv2.p, v.p, (size_t)N * 4, cudaMemcpyDeviceToDevice, s));
        FX_CHECK_CUDA(cudaMemsetAsync(counters.p, 0, 4, s));
        PowerArgs pa{N,        K,        cfg->power_iterations, meet_polls(), ck_beg.p,
                     ck_end.p, cl_ck.p,  beg.p,                 end.p,        rp.p,
                     col.p,    clp.p,    deg.p,                 lv2.p,        lv.p,
                     v.p,      part.p,   counters.p};
        void *args[] = {&pa};
        const cudaError_t e = cudaLaunchCooperativeKernel((const void *)part_power_kernel, dim3(grid),
                                                          dim3(kPowerThreads), args, kPowerSmem, s);
        if (e == cudaErrorCooperativeLaunchTooLarge) {  // a share of the device: step by step
          cudaGetLastError();
          fixed = false;
        } else {
          FX_CHECK_CUDA(e);
          ctx->launches += 1;
          total_iters += (int64_t)cfg->power_iterations * C;
        }
      }
      // normalise the start vector (:151-156)
      if (fixed) {
      } else if (exact) {
        part_seq_kernel<<<C, 32, 0, s>>>(C, beg.p, end.p, v.p, 0, nrm.p);
      } else {
        part_chunk_kernel<<<kb, 256, 0, s>>>(K, ck_beg.p, ck_end.p, ck_cl.p, act.p, v.p,
                                             nullptr, part.p);
        part_combine_kernel<<<cb, 64, 0, s>>>(C, beg.p, end.p, cl_ck.p, part.p, 0, 0.0, act.p,
                                              mean.p, nrm.p, lambda.p, iters.p);
      }
      if (!fixed) {
        part_div_kernel<<<nb, 256, 0, s>>>(N, clp.p, act.p, v.p, nullptr, nrm.p, v.p);
        FX_CHECK_LAUNCH();
        ctx->launches += exact ? 4 : 5;
      }
      int it = 0;
      while (!fixed && it < cfg->power_iterations) {
        part_spmv_csr_kernel<<<nb, 256, 0, s>>>(N, rp.p, col.p, clp.p, act.p, deg.p, v.p,
                                                lv.p);
        ++it;
        if (exact) {
          // deflate and norm in place in lv, then v = lv / norm (v = lv, :182)
          part_seq_kernel<<<C, 32, 0, s>>>(C, beg.p, end.p, lv.p, 1, nrm.p);
          part_div_kernel<<<nb, 256, 0, s>>>(N, clp.p, act.p, lv.p, nullptr, nrm.p, v.p);
          FX_CHECK_LAUNCH();
          ctx->launches += 3;
          continue;
        }
        part_chunk_kernel<<<kb, 256, 0, s>>>(K, ck_beg.p, ck_end.p, ck_cl.p, act.p, lv.p, v.p,
                                             part.p);
        part_combine_kernel<<<cb, 64, 0, s>>>(C, beg.p, end.p, cl_ck.p, part.p, 1, cfg->tol,
                                              act.p, mean.p, nrm.p, lambda.p, iters.p);
        part_div_kernel<<<nb, 256, 0, s>>>(N, clp.p, act.p, lv.p, mean.p, nrm.p, v.p);
        FX_CHECK_LAUNCH();
        ctx->launches += 4;
        if (cfg->tol <= 0.0) continue;  // fixed iteration count: nothing converges early
        FX_CHECK_CUDA(cudaMemsetAsync(any.p, 0, 4, s));
        part_retire_kernel<<<cb, 64, 0, s>>>(C, act.p, any.p);
        FX_CHECK_LAUNCH();
        ctx->launches += 1;
        if ((it & 7) == 0) {  // every 8 iterations: all converged?
          int32_t h_any = 0;
          FX_CHECK_CUDA(cudaMemcpyAsync(&h_any, any.p, 4, cudaMemcpyDeviceToHost, s));
          FX_CHECK_CUDA(cudaStreamSynchronize(s));
          if (!h_any) break;
        }
      }
      if (exact) {
        total_iters += (int64_t)it * C;
      } else if (!fixed) {
        std::vector<int32_t> hit((size_t)C);
        FX_CHECK_CUDA(cudaMemcpyAsync(hit.data(), iters.p, (size_t)C * 4,
                                      cudaMemcpyDeviceToHost, s));
        FX_CHECK_CUDA(cudaStreamSynchronize(s));
        for (int32_t x : hit) total_iters += x;
      }
      // stable segmented sort: by value (4 passes), then stably by cluster
      const int ab = (A + 255) / 256;
      part_keys_kernel<<<ab, 256, 0, s>>>(A, C, beg.p, off.p, v.p, keys[0].p, slot_pos.p,
                                          vals[0].p);
      FX_CHECK_LAUNCH();
      uint32_t *kk[2] = {keys[0].p, keys[1].p};
      int32_t *vv[2] = {vals[0].p, vals[1].p};
      FX_TRY(radix_sort_pairs(kk, vv, A, 4, th.p, ts.p, dt.p, s));  // result in buffer 0
      int rb = 0;
      if (C > 1) {
        part_major_kernel<<<ab, 256, 0, s>>>(A, C, vals[0].p, off.p, keys[0].p);
        FX_CHECK_LAUNCH();
        const int passes = C <= 256 ? 1 : (C <= 65536 ? 2 : 3);
        FX_TRY(radix_sort_pairs(kk, vv, A, passes, th.p, ts.p, dt.p, s));
        rb = passes & 1;
      }
      FX_CHECK_CUDA(cudaMemcpyAsync(perm[cur ^ 1].p, perm[cur].p, (size_t)N * 4,
                                    cudaMemcpyDeviceToDevice, s));
      part_apply_kernel<<<ab, 256, 0, s>>>(A, vals[rb].p, slot_pos.p, perm[cur].p,
                                           perm[cur ^ 1].p, pos_of.p);
      FX_CHECK_LAUNCH();
      ctx->launches += 3;
      cur ^= 1;
      int32_t had = 0;
      // the exact count where the next depth's choice may hang on it
      const bool ask =
          !exact && ((most <= 2 * kPartChunk && cluster_edges(0.5 * most) > (double)small_edges) ||
                     dense_rows(per_gate, A));
      if (ask)
        FX_CHECK_CUDA(cudaMemcpyAsync(&had, rp.p + N, 4, cudaMemcpyDeviceToHost, s));
      FX_CHECK_CUDA(cudaStreamSynchronize(s));
      if (ask) per_gate = (double)had / (double)A;
    }
    unsigned long long si = 0;
    unsigned int gave_up = 0;
    FX_CHECK_CUDA(cudaMemcpyAsync(&si, small_its.p, 8, cudaMemcpyDeviceToHost, s));
    FX_CHECK_CUDA(cudaMemcpyAsync(&gave_up, counters.p + 1, 4, cudaMemcpyDeviceToHost, s));
    FX_CHECK_CUDA(cudaStreamSynchronize(s));
    if (gave_up) {
      set_error("fx_partition: a bounded wait of a block for the others expired");
      return FX_ETIMEOUT;
    }
    total_iters += (int64_t)si;
  }
  // outputs: leaves in position order, with their regions
  if (!nodes.empty()) {
    nodes[0].cx = d->chip_w / 2.0f;
    nodes[0].cy = d->chip_h / 2.0f;
    nodes[0].w = d->chip_w;
    nodes[0].h = d->chip_h;
    place_regions(nodes, 0);
  }
  if (out_leaf_gate && N > 0)
    FX_CHECK_CUDA(cudaMemcpyAsync(out_leaf_gate, perm[cur].p, (size_t)N * 4,
                                  cudaMemcpyDeviceToHost, s));
  FX_CHECK_CUDA(cudaStreamSynchronize(s));
  int32_t l = 0;
  for (const PNode &nd : nodes) {
    if (nd.left >= 0) continue;
    if (out_leaf_ptr) out_leaf_ptr[l] = nd.beg;
    if (out_region) {
      out_region[4 * l + 0] = nd.cx;
      out_region[4 * l + 1] = nd.cy;
      out_region[4 * l + 2] = nd.w;
      out_region[4 * l + 3] = nd.h;
    }
    if (out_leaf_depth) out_leaf_depth[l] = nd.depth;
    ++l;
  }
  if (out_leaf_ptr) out_leaf_ptr[n_leaves] = N;
  if (out_stats) {
    out_stats->n_leaves = n_leaves;
    out_stats->n_nodes = (int32_t)nodes.size();
    out_stats->max_depth = max_depth;
    out_stats->levels = levels;
    out_stats->power_iterations = total_iters;
  }
  return FX_OK;
}
