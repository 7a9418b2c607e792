// fx_refine.cu -- the congestion refinement loop (refine_placement,
// H/src/algorithm/refiner.rs:34-126) on the device.
//
// Each iteration: congestion counts (rows D+F kernels), the total overflow as
// the reference's f32 running sum over cells in row-major order (the stop and
// stall rules compare this exact value), then every gate whose
// cell is hot (overflow > threshold, gates_in_hot_cells, congestion.rs:77-93)
// moves toward the first least-congested cell within radius 3
// (move_gate_from_hot_cell, refiner.rs:92-126; Iterator::min_by keeps the
// first minimum in (dr, dc) order). A move reads only the gate's own position
// and the grid frozen at the start of the iteration, so all gates move in
// parallel with the reference's sequential result.
#include <climits>
#include <cmath>
#include <cstring>

#include "fx_internal.h"
#include "fx_device.cuh"

namespace fx {

__device__ __forceinline__ float rclampf(float v, float lo, float hi) {
  if (v < lo) v = lo;
  if (v > hi) v = hi;
  return v;
}

// grid.rs:86-91 total_overflow: the reference's f32 running sum over the
// cells in row-major order, bit for bit, by a whole block. Every term is
// >= 0, so the sum only grows. While it stays in one binade [2^e, 2^(e+1)) it
// is an integer S of units u = 2^(e-23), S < 2^24, and adding a term adds
// floor(a / u) or one more: which of the two depends on the term alone, except
// at a tie, where it makes the new S even and so depends on the parity of S
// too. A run of terms therefore maps each starting parity to one increment,
// and such maps compose: each thread composes its cells, a scan
// composes the threads (plain sums in a warp without ties), and only the first term that takes S to 2^24 (where u
// doubles) is added as the f32 addition it is. Then the rest of the chunk is
// scanned again in the new unit: one scan per chunk of 4096 cells and one per
// doubling of the sum.
// One lane folding the cells in order is bound by the latency of its additions
// (65536 dependent ones: 459 us at 256 x 256, ncu); this takes 33 us.
// Also keeps the loop's state (stop and stall rules, refiner.rs:45-72), so
// the host may queue an iteration before it has read the previous one's total.
struct RefineState {
  float total, most;  // of the last count before the stop
  float prev;
  int stall, iters, stop;
  unsigned int moves;
};

constexpr int kTotalThreads = 512, kTotalItems = 8, kTotalWarps = kTotalThreads / 32;
constexpr int kTotalChunk = kTotalThreads * kTotalItems;
constexpr int kTotalHead = 512;      // cells one lane folds first: the sum doubles often there
constexpr int kTotalFull = 1 << 24;  // units where the binade ends
// A term of kTotalWhole units or more counts as kTotalSat: it is added by itself.
constexpr int kTotalSat = 1 << 25;
// Below this both additions of total_term are whole to the unit: the larger
// one, to 1.5 * 2^23 + 1, stays below 2^24, where the spacing becomes 2.
constexpr float kTotalWhole = 4194303.0f;

// Increment of the sum for a term of t = a / u units (exact), as {from even
// S, from odd S}: t rounded once to an integer, ties to the parity that makes
// S plus it even, by one f32 addition to 1.5 * 2^23 or to the odd number after
// it (no conversions, which run at an eighth of the addition rate).
__device__ __forceinline__ int2 total_term(float t) {
  if (!(t < kTotalWhole)) return make_int2(kTotalSat, kTotalSat);
  return make_int2(__float_as_int(__fadd_rn(t, 12582912.0f)) - 0x4b400000,
                   __float_as_int(__fadd_rn(t, 12582913.0f)) - 0x4b400001);
}

// First a, then b. Saturated maps stay above kTotalFull and their sums fit:
// at most 32 of them are composed between two total_clip.
__device__ __forceinline__ int2 total_then(int2 a, int2 b) {
  return make_int2(a.x + ((a.x & 1) ? b.y : b.x), a.y + ((a.y & 1) ? b.x : b.y));
}
__device__ __forceinline__ int2 total_clip(int2 a) {
  return make_int2(min(a.x, kTotalSat), min(a.y, kTotalSat));
}

// Inclusive composition over the first kN lanes of the warp.
template <int kN>
__device__ __forceinline__ int2 total_scan(int2 v, int lane) {
#pragma unroll
  for (int o = 1; o < kN; o <<= 1) {
    const int2 before = make_int2(__shfl_up_sync(0xffffffffu, v.x, o),
                                  __shfl_up_sync(0xffffffffu, v.y, o));
    if (lane >= o) v = total_then(before, v);
  }
  return v;
}

__global__ void __launch_bounds__(kTotalThreads)
refine_total_kernel(const uint32_t *__restrict__ counts, int cells, float cap, float threshold,
                    int decide, RefineState *__restrict__ st, RefineState *__restrict__ host) {
  __shared__ int2 wsum[kTotalWarps];
  __shared__ float s_sh;
  __shared__ int cross_sh;
  __shared__ float wmax[kTotalWarps];
  __shared__ float head[kTotalHead];
  if (decide && st->stop) {  // the loop has ended: its totals stand
    if (threadIdx.x == 0) *host = *st;
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  float mx = 0.0f;
  float s = 0.0f;  // the running sum, the same in every thread
  // raw counts of a chunk (the next one's are in flight while one is summed)
  auto load = [&](int base, uint32_t *c) {
    const int i0 = base + tid * kTotalItems;
    if (i0 + kTotalItems <= cells) {
#pragma unroll
      for (int r = 0; r < kTotalItems; r += 4) {
        const uint4 p = *reinterpret_cast<const uint4 *>(counts + i0 + r);
        c[r] = p.x;
        c[r + 1] = p.y;
        c[r + 2] = p.z;
        c[r + 3] = p.w;
      }
    } else {
#pragma unroll
      for (int r = 0; r < kTotalItems; ++r) c[r] = i0 + r < cells ? counts[i0 + r] : 0u;
    }
  };
  uint32_t nxt[kTotalItems];
  load(0, nxt);
  for (int base = 0; base < cells; base += kTotalChunk) {
    float a[kTotalItems];
#pragma unroll
    for (int r = 0; r < kTotalItems; ++r) {
      const float f = (float)nxt[r];
      const float ov = fmaxf(__fsub_rn(__fadd_rn(f, f), cap), 0.0f);
      a[r] = base + tid * kTotalItems + r < cells ? ov : 0.0f;  // adding 0 changes nothing
      mx = fmaxf(mx, a[r]);
    }
    if (base + kTotalChunk < cells) load(base + kTotalChunk, nxt);
    if (base == 0) {
#pragma unroll
      for (int r = 0; r < kTotalItems; ++r) {
        const int i = tid * kTotalItems + r;
        if (i < kTotalHead) {
          head[i] = a[r];
          a[r] = 0.0f;
        }
      }
      __syncthreads();
      if (tid == 0) {
#pragma unroll 16
        for (int i = 0; i < kTotalHead; ++i) s = __fadd_rn(s, head[i]);
        s_sh = s;
      }
      __syncthreads();
      s = s_sh;
    }
    for (;;) {
      // unit of the sum's binade; below 2^-90 (and at 0) every positive term
      // is added by itself
      const int e = (int)(__float_as_uint(s) >> 23) - 127;
      const bool small = e < -90;
      // 2^(23-e), its exponent kept in range: a sum beyond 2^126 would need
      // cells past 2^26 of counts past 2^32
      const float inv_u = __int_as_float((127 + (small ? 0 : 23 - e)) << 23);
      const int S0 = small ? 0 : (int)((__float_as_uint(s) & 0x7fffffu) | 0x800000u);
      auto units = [&](float v) {
        return small ? (v > 0.0f ? (float)kTotalSat : 0.0f) : __fmul_rn(v, inv_u);
      };
      int2 t[kTotalItems];
      int sum = 0;
      bool tie = false;
#pragma unroll
      for (int r = 0; r < kTotalItems; ++r) {
        t[r] = total_term(units(a[r]));
        sum += t[r].x;
        tie |= t[r].x != t[r].y;
      }
      // the chunk's map: the warps' totals (plain sums unless a term ties),
      // composed in order. No scan yet: most chunks stay in their binade.
      const bool warp_tie = __any_sync(0xffffffffu, tie);
      int2 d = make_int2(sum, sum);
      if (warp_tie) {
        d = t[0];
#pragma unroll
        for (int r = 1; r < kTotalItems; ++r) d = total_then(d, t[r]);
      }
      d = total_clip(d);
      int2 inc = d;  // of the warp, valid in its last lane
      if (!warp_tie) {
        const int all = __reduce_add_sync(0xffffffffu, d.x);
        inc = make_int2(all, all);
      } else {
        inc = total_scan<32>(d, lane);
      }
      inc = total_clip(inc);
      if (lane == 31) wsum[w] = inc;
      if (tid == 0) cross_sh = INT_MAX;
      __syncthreads();
      int2 wi = lane < kTotalWarps ? wsum[lane] : make_int2(0, 0);
      const int odd = S0 & 1;
      int all;
      const bool block_tie = __any_sync(0xffffffffu, wi.x != wi.y);
      if (!block_tie) {
        all = __reduce_add_sync(0xffffffffu, wi.x);
      } else {
        const int2 c = total_scan<kTotalWarps>(wi, lane);
        all = __shfl_sync(0xffffffffu, odd ? c.y : c.x, kTotalWarps - 1);
      }
      if (S0 + all < kTotalFull) {  // the chunk ends in this binade
        if (!small) s = __fmul_rn((float)(S0 + all), __int_as_float((127 + e - 23) << 23));
        __syncthreads();  // wsum and cross_sh are free again
        break;
      }
      inc = total_scan<32>(d, lane);
      wi = total_scan<kTotalWarps>(wi, lane);
      // the first term that takes S to 2^24, by the thread that holds it
      const int2 wex = make_int2(__shfl_sync(0xffffffffu, wi.x, max(w - 1, 0)),
                                 __shfl_sync(0xffffffffu, wi.y, max(w - 1, 0)));
      int2 ex = make_int2(__shfl_up_sync(0xffffffffu, inc.x, 1),
                          __shfl_up_sync(0xffffffffu, inc.y, 1));
      if (lane == 0) ex = make_int2(0, 0);
      if (w > 0) ex = total_then(wex, ex);
      int S = S0 + (odd ? ex.y : ex.x);
      if (S < kTotalFull) {
        bool found = false;
#pragma unroll
        for (int r = 0; r < kTotalItems; ++r) {
          if (found) continue;
          const int Sn = S + ((S & 1) ? t[r].y : t[r].x);
          if (Sn >= kTotalFull) {
            found = true;
            const float sv = small ? s : __fmul_rn((float)S, __int_as_float((127 + e - 23) << 23));
            s_sh = __fadd_rn(sv, a[r]);
            cross_sh = tid * kTotalItems + r;
          } else {
            S = Sn;
          }
        }
      }
      __syncthreads();
      const int cross = cross_sh;
      s = s_sh;
#pragma unroll
      for (int r = 0; r < kTotalItems; ++r)
        if (tid * kTotalItems + r <= cross) a[r] = 0.0f;  // added already
      __syncthreads();
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) wmax[w] = mx;
  __syncthreads();
  if (tid != 0) return;
  for (int q = 0; q < kTotalWarps; ++q) mx = fmaxf(mx, wmax[q]);
  RefineState n = *st;
  n.total = s;
  n.most = mx;
  if (decide) {
    if (s <= threshold) {
      n.stop = 1;
    } else {
      if (fabsf(__fsub_rn(n.prev, s)) < __fmul_rn(0.01f, fmaxf(n.prev, 1.0f))) {
        if (++n.stall >= 10) n.stop = 1;
      } else {
        n.stall = 0;
      }
      if (!n.stop) {
        n.prev = s;
        ++n.iters;
      }
    }
  }
  *st = n;
  *host = n;
}

__global__ void refine_move_kernel(float *__restrict__ x, float *__restrict__ y, int n,
                                   const uint32_t *__restrict__ counts, int cols,
                                   int rows, float cw, float ch, float cap,
                                   float threshold, float max_move, float chip_w,
                                   float chip_h, RefineState *__restrict__ st) {
  if (st->stop) return;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const float gx = x[g], gy = y[g];
  const int col = cell_at(gx, cw, cols), row = cell_at(gy, ch, rows);
  const float c0 = (float)counts[(size_t)row * cols + col];
  const float ov = fmaxf(__fsub_rn(__fadd_rn(c0, c0), cap), 0.0f);
  if (!(ov > threshold)) return;
  bool found = false;
  int bc = 0, br = 0;
  float best = 0.0f;
  for (int dr = -3; dr <= 3; ++dr)
    for (int dc = -3; dc <= 3; ++dc) {
      if (dr == 0 && dc == 0) continue;
      const int nc = col + dc, nr = row + dr;
      if (nc < 0 || nc >= cols || nr < 0 || nr >= rows) continue;
      const float c = (float)counts[(size_t)nr * cols + nc];
      const float tot = __fadd_rn(c, c);
      if (!found || tot < best) {
        found = true;
        best = tot;
        bc = nc;
        br = nr;
      }
    }
  if (!found) return;
  const float tx = __fmul_rn(__fadd_rn((float)bc, 0.5f), cw);
  const float ty = __fmul_rn(__fadd_rn((float)br, 0.5f), ch);
  const float dx = rclampf(__fsub_rn(tx, gx), -max_move, max_move);
  const float dy = rclampf(__fsub_rn(ty, gy), -max_move, max_move);
  x[g] = rclampf(__fadd_rn(gx, dx), 0.0f, chip_w);
  y[g] = rclampf(__fadd_rn(gy, dy), 0.0f, chip_h);
  atomicAdd(&st->moves, 1u);
}

__global__ void refine_init_kernel(RefineState *__restrict__ st) {
  RefineState s{};
  s.prev = FLT_MAX;
  *st = s;
}

}  // namespace fx

using namespace fx;

extern "C" int fx_refine_cfg_default(fx_refine_cfg *c) {
  if (!c) return FX_EINVAL;
  c->max_iterations = 100;
  c->move_distance = 5.0f;
  c->overflow_threshold = 1.0f;
  c->grid_cols = 256;
  c->grid_rows = 256;
  c->reserved0 = 0;
  return FX_OK;
}

extern "C" int fx_refine(fx_ctx *ctx, fx_design *d, const fx_refine_cfg *cfg,
                         float *x, float *y, fx_refine_stats *stats,
                         uint32_t *out_counts) {
  if (!ctx || !d || !cfg || (x == nullptr) != (y == nullptr) || cfg->grid_cols <= 0 ||
      cfg->grid_rows <= 0 || cfg->max_iterations < 0 ||
      (int64_t)cfg->grid_cols * cfg->grid_rows > (int64_t)1 << 26) {
    set_error("fx_refine: invalid arguments");
    return FX_EINVAL;
  }
  FX_CHECK_CUDA(cudaSetDevice(ctx->device));
  AllocScope alloc_scope(ctx->stream);
  cudaStream_t s = ctx->stream;
  if (x) FX_TRY(fx_design_set_positions(d, x, y));
  const int cols = cfg->grid_cols, rows = cfg->grid_rows, cells = cols * rows;
  // RoutingGrid::new (grid.rs:25-32)
  const float cw = d->chip_w / (float)cols, ch = d->chip_h / (float)rows;
  const float cap = (cw + ch) * 0.5f;
  float *px = d->x[d->cur].p, *py = d->y[d->cur].p;
  d->pos_in_box = false;  // moved positions are not re-checked against the die
  DevBuf<RefineState> state;
  FX_TRY(state.alloc(1));
  static_assert(sizeof(RefineState) <= sizeof(ctx->readback->refine[0]), "readback slot");
  auto slot = [&](int i) { return reinterpret_cast<RefineState *>(ctx->readback_dev->refine[i & 1]); };
  auto seen = [&](int i) {
    RefineState r;
    std::memcpy(&r, ctx->readback->refine[i & 1], sizeof r);
    return r;
  };
  refine_init_kernel<<<1, 1, 0, s>>>(state.p);
  FX_CHECK_LAUNCH();
  ctx->launches += 1;
  // Iteration it is queued before iteration it - 1's decision is read, so the
  // GPU does not wait for the host; once the device has stopped, what was
  // queued counts the same positions again and moves nothing.
  cudaEvent_t done[2] = {ctx->fork, ctx->join};
  RefineState last{};
  bool stopped = false;
  for (int it = 0; it < cfg->max_iterations && !stopped; ++it) {
    FX_TRY(congestion_run(ctx, d, px, py, cols, rows, s));
    refine_total_kernel<<<1, kTotalThreads, 0, s>>>(d->cong.counts.p, cells, cap,
                                                    cfg->overflow_threshold, 1, state.p, slot(it));
    FX_CHECK_LAUNCH();
    FX_CHECK_CUDA(cudaEventRecord(done[it & 1], s));
    refine_move_kernel<<<(d->n + 255) / 256, 256, 0, s>>>(
        px, py, d->n, d->cong.counts.p, cols, rows, cw, ch, cap, cfg->overflow_threshold,
        cfg->move_distance, d->chip_w, d->chip_h, state.p);
    FX_CHECK_LAUNCH();
    ctx->launches += 2;
    // (the first decision is waited for: a placement with nothing to refine is
    // not counted a third time)
    const int read = it > 0 ? it - 1 : 0;
    FX_CHECK_CUDA(cudaEventSynchronize(done[read & 1]));
    stopped = seen(read).stop != 0;
  }
  // the final count (the stopped loop's own, or that of the last moves)
  FX_TRY(congestion_run(ctx, d, px, py, cols, rows, s));
  refine_total_kernel<<<1, kTotalThreads, 0, s>>>(d->cong.counts.p, cells, cap,
                                                  cfg->overflow_threshold, 0, state.p, slot(0));
  FX_CHECK_LAUNCH();
  ctx->launches += 1;
  double hp = 0.0;
  FX_CHECK_CUDA(cudaMemcpyAsync(&hp, d->cong.result.p, 8, cudaMemcpyDeviceToHost, s));
  if (out_counts)
    FX_CHECK_CUDA(cudaMemcpyAsync(out_counts, d->cong.counts.p, (size_t)cells * 4,
                                  cudaMemcpyDeviceToHost, s));
  FX_CHECK_CUDA(cudaStreamSynchronize(s));
  last = seen(0);
  if (x) FX_TRY(fx_design_get_positions(d, x, y));
  if (stats) {
    stats->iterations = last.iters;
    stats->moves = last.moves;
    stats->total_overflow = last.total;
    stats->max_overflow = last.most;
    stats->hpwl = hp;
  }
  return FX_OK;
}
