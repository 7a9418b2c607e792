// fx_dct.cu -- the DCT Poisson solve by fast transforms (FX_DCT_SIMT and
// FX_DCT_I8, the FP32-accurate settings).
//
// The solve is the linear map of force_electrostatic.py:69-103: DCT-II of the
// charge along both axes, division by the eigenvalues, DCT-III back, centred
// differences. A length-N DCT-II is one length-N complex FFT of the reordered
// input (Makhoul, "A fast cosine transform in one and two dimensions", 1980:
// v[n] = x[2n], v[N-1-n] = x[2n+1], X[k] = Re(e^{-i pi k / 2N} V[k])), and two
// real rows share one complex FFT. That is O(G^2 log G) instead of the dense
// products' O(G^3), and the whole solve is three launches:
//   dct_rows_kernel   accumulated areas -> charge -> T1 = DCT along x
//   dct_cols_kernel   DCT along y, / eigenvalue, DCT-III along y, and the
//                     y differences, for a few columns per block: T1 -> (u, Dy u)
//   dct_field_kernel  DCT-III along x of both as one complex FFT per row, and
//                     the x differences: -> E_x, E_y (phi on request)
// All transform arithmetic is FP64; only the grids between the kernels are
// f32, as the operands of the dense products were. FP64 because the field
// differences a huge smooth potential: f32 butterflies would lose the digits
// the dense products lost (4e-5 relative at G = 640), here 1e-7. A constant
// charge has no potential (phi_hat[0, 0] = 0), so the transforms run on the
// density less its mean instead of less the target: the large kx = 0 entries
// of T1 would otherwise be rounded at the mean's scale (7.5e-7 of the field at
// G = 640).
//
// What bounds it: FP64 issue and shared memory about equally (an FFT of 1024
// points moves 128 KB through shared memory and spends ~70 kflop); the grids
// stay in L2 up to G = 2048. One butterfly of eight points per thread keeps
// all data of a stage in registers, so a stage needs one shared buffer and
// two barriers; the buffer is padded by one element in eight against bank
// conflicts of the stride-8 stores. Measured on a B200, the solve of one step
// (ncu, cold caches): 46 us at G = 1024 (310 us as int8-slice products), 157
// us at G = 2048 (1500 us).
#include <algorithm>
#include <cmath>

#include "fx_internal.h"
#include "fx_dct.cuh"

namespace fx {
namespace {

constexpr double kInvAreaScale = 1.0 / 4294967296.0;

__host__ __device__ __forceinline__ int pad8(int i) { return i + (i >> 3); }

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
// a * -i
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }

__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d) {
  const double2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = mul_mi(csub(b, d));
  a = cadd(s, u);
  b = cadd(t, v);
  c = csub(s, u);
  d = csub(t, v);
}

__device__ __forceinline__ void dft8(double2 v[8]) {
  dft4(v[0], v[2], v[4], v[6]);
  dft4(v[1], v[3], v[5], v[7]);
  constexpr double r = 0.70710678118654752440;
  const double2 o1 = make_double2(r * (v[3].x + v[3].y), r * (v[3].y - v[3].x));
  const double2 o2 = mul_mi(v[5]);
  const double2 o3 = make_double2(r * (v[7].y - v[7].x), -r * (v[7].x + v[7].y));
  const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = cadd(e0, o0);
  v[1] = cadd(e1, o1);
  v[2] = cadd(e2, o2);
  v[3] = cadd(e3, o3);
  v[4] = csub(e0, o0);
  v[5] = csub(e1, o1);
  v[6] = csub(e2, o2);
  v[7] = csub(e3, o3);
}

// Forward FFT of the N = 2^a * o points (o odd) in z (padded), by the N / 8
// threads j0 = 0 .. N/8 - 1 of the sequence; every thread of the block calls
// it with the same N. Self-sorting (Stockham) stages of radix 8, then 4 or 2,
// then the odd factor as one direct stage of length o (its points j, j + s,
// ... keep their places, so it needs no twiddles). tw[k] = e^{-2 pi i k / N}.
// Begins and ends with a barrier.
__device__ __forceinline__ void fft_block(double2 *z, int N, int odd, int j0,
                                          const double2 *__restrict__ tw) {
  const int n8 = N >> 3;
  int ls = 0, rem = N / odd;  // log2 of the stride, what is left of 2^a
  double2 v[8];
  __syncthreads();
  while (rem >= 8) {
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = z[pad8(j0 + r * n8)];
    dft8(v);
    const int q = j0 & ((1 << ls) - 1), p = j0 >> ls;
    if ((N >> ls) > 8) {
      const double2 w1 = tw[p << ls];
      const double2 w2 = cmul(w1, w1), w3 = cmul(w2, w1), w4 = cmul(w2, w2);
      v[1] = cmul(v[1], w1);
      v[2] = cmul(v[2], w2);
      v[3] = cmul(v[3], w3);
      v[4] = cmul(v[4], w4);
      v[5] = cmul(v[5], cmul(w4, w1));
      v[6] = cmul(v[6], cmul(w4, w2));
      v[7] = cmul(v[7], cmul(w4, w3));
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 8; ++t) z[pad8(q + ((8 * p + t) << ls))] = v[t];
    __syncthreads();
    ls += 3;
    rem >>= 3;
  }
  if (rem == 4) {
    const int n4 = N >> 2;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      double2 *b = v + 4 * i;
      const int j = j0 + i * n8;
#pragma unroll
      for (int r = 0; r < 4; ++r) b[r] = z[pad8(j + r * n4)];
      dft4(b[0], b[1], b[2], b[3]);
      if ((N >> ls) > 4) {
        const double2 w1 = tw[(j >> ls) << ls], w2 = cmul(w1, w1);
        b[1] = cmul(b[1], w1);
        b[2] = cmul(b[2], w2);
        b[3] = cmul(b[3], cmul(w2, w1));
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = j0 + i * n8, q = j & ((1 << ls) - 1), p = j >> ls;
#pragma unroll
      for (int t = 0; t < 4; ++t) z[pad8(q + ((4 * p + t) << ls))] = v[4 * i + t];
    }
    __syncthreads();
    ls += 2;
  } else if (rem == 2) {
    const int n2 = N >> 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = j0 + i * n8;
      const double2 a = z[pad8(j)], b = z[pad8(j + n2)];
      v[2 * i] = cadd(a, b);
      v[2 * i + 1] = csub(a, b);
      if ((N >> ls) > 2) v[2 * i + 1] = cmul(v[2 * i + 1], tw[(j >> ls) << ls]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = j0 + i * n8, q = j & ((1 << ls) - 1), p = j >> ls;
      z[pad8(q + ((2 * p) << ls))] = v[2 * i];
      z[pad8(q + ((2 * p + 1) << ls))] = v[2 * i + 1];
    }
    __syncthreads();
    ls += 1;
  }
  if (odd > 1) {
    const int s = 1 << ls;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = j0 + i * n8, j = e & (s - 1), t = e >> ls;
      double2 acc = z[pad8(j)];
      for (int r = 1, rt = t; r < odd; ++r) {
        const double2 c = cmul(z[pad8(j + (r << ls))], tw[rt << ls]);
        acc = cadd(acc, c);
        rt += t;
        if (rt >= odd) rt -= odd;
      }
      v[i] = acc;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) z[pad8(j0 + i * n8)] = v[i];
    __syncthreads();
  }
}

// Place of x in the reordered input: even x in front, odd x mirrored behind.
__device__ __forceinline__ int dct_place(int x, int N) {
  return (x & 1) ? N - 1 - (x >> 1) : (x >> 1);
}

// From the spectra of two real sequences in DCT-III form, h[k] = (a[k], b[k])
// and hm = h[N - k] (0 for k = 0), the FFT inputs of the inverse transform at
// k and N - k, with re and im swapped (the inverse FFT is the forward FFT of
// swapped data, swapped). c, s = cos, sin(pi k / 2N).
__device__ __forceinline__ void idct_pair(double2 h, double2 hm, double c, double s,
                                          double2 &zk, double2 &zm) {
  const double ra = c * h.x + s * hm.x, ia = s * h.x - c * hm.x;
  const double rb = c * h.y + s * hm.y, ib = s * h.y - c * hm.y;
  zk = make_double2(ia + rb, ra - ib);
  zm = make_double2(rb - ia, ra + ib);
}

// Rows: two per sequence. Threads x = S * N / 8.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
dct_rows_kernel(DctArgs a) {
  extern __shared__ double2 zsh[];
  const int N = a.G, n8 = N >> 3;
  const int seq = threadIdx.x / n8, j0 = threadIdx.x - seq * n8;
  const int row = 2 * (blockIdx.x * a.seqs + seq);
  double2 *z = zsh + seq * pad8(N);
  const size_t r0 = (size_t)row * N, r1 = r0 + N;
  // all loads before the stores that re-arm the accumulator: the compiler
  // may not move them across (211 to 40 us at G = 2048 otherwise)
  unsigned long long qa[8], qb[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    qa[i] = a.acc[r0 + j0 + i * n8];
    qb[i] = a.acc[r1 + j0 + i * n8];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int x = j0 + i * n8;
    const double va = (double)qa[i] * kInvAreaScale * a.inv_bin_area;
    const double vb = (double)qb[i] * kInvAreaScale * a.inv_bin_area;
    a.acc[r0 + x] = 0ull;
    a.acc[r1 + x] = 0ull;
    if (a.rho) {
      a.rho[r0 + x] = (float)(va - a.target);
      a.rho[r1 + x] = (float)(vb - a.target);
    }
    z[pad8(dct_place(x, N))] = make_double2(va - a.level, vb - a.level);
  }
  fft_block(z, N, a.odd, j0, a.tw);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = j0 + i * n8;
    const double2 p = z[pad8(k)], m = z[pad8(k ? N - k : 0)], w = a.qt[k];
    // V_a = (p + conj m) / 2, V_b = (p - conj m) / 2i; Re(e^{-i theta} V)
    a.t1[r0 + k] = (float)(0.5 * (w.x * (p.x + m.x) + w.y * (p.y - m.y)));
    a.t1[r1 + k] = (float)(0.5 * (w.x * (p.y + m.y) + w.y * (m.x - p.x)));
  }
}

// Columns: two per sequence, `seqs` sequences (1 or 2) per block.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
dct_cols_kernel(DctArgs a) {
  extern __shared__ double2 zsh[];
  const int N = a.G, n8 = N >> 3, T = blockDim.x, S = a.seqs;
  const int zs = pad8(N);
  const int c0 = blockIdx.x * 2 * S;
  const int lg = S - 1;  // log2(S) for 1 or 2
  // sequence fastest, so that a row's columns of the block are read together
  for (int e = threadIdx.x; e < N * S; e += T) {
    const int sq = e & (S - 1), y = e >> lg;
    const float2 v = *reinterpret_cast<const float2 *>(a.t1 + (size_t)y * N + c0 + 2 * sq);
    zsh[sq * zs + pad8(dct_place(y, N))] = make_double2((double)v.x, (double)v.y);
  }
  const int seq = threadIdx.x / n8, j0 = threadIdx.x - seq * n8;
  double2 *z = zsh + seq * zs;
  const int ca = c0 + 2 * seq;
  fft_block(z, N, a.odd, j0, a.tw);
  // spectrum, / eigenvalue, and the inverse transform's input, pair k, N - k
  const double ea = a.ax2[ca], eb = a.ax2[ca + 1], inv_n = -1.0 / (double)N;
  for (int k = j0; k <= N / 2; k += n8) {
    const int km = k ? N - k : 0;
    const double2 p = z[pad8(k)], m = z[pad8(km)], w = a.qt[k];
    const double sx = 0.5 * (p.x + m.x), dy = 0.5 * (p.y - m.y);
    const double sy = 0.5 * (p.y + m.y), dx = 0.5 * (m.x - p.x);
    const double lk = a.ay2[k], lm = a.ay2[km];
    double2 h = make_double2((w.x * sx + w.y * dy) * (inv_n / (lk + ea)),
                             (w.x * sy + w.y * dx) * (inv_n / (lk + eb)));
    double2 hm = make_double2((w.y * sx - w.x * dy) * (inv_n / (lm + ea)),
                              (w.y * sy - w.x * dx) * (inv_n / (lm + eb)));
    if (k == 0) {
      if (ca == 0) h.x = 0.0;  // no constant potential
      hm = make_double2(0.0, 0.0);
    }
    double2 zk, zm;
    idct_pair(h, hm, w.x, w.y, zk, zm);
    z[pad8(k)] = zk;
    if (km != k) z[pad8(km)] = zm;
  }
  fft_block(z, N, a.odd, j0, a.tw);
  // u and Dy u of the block's columns, interleaved (re and im are swapped)
  for (int e = threadIdx.x; e < N * S; e += T) {
    const int sq = e & (S - 1), y = e >> lg;
    const double2 *zq = zsh + sq * zs;
    const double2 u = zq[pad8(dct_place(y, N))];
    const double2 lo = y > 0 ? zq[pad8(dct_place(y - 1, N))] : u;
    const double2 hi = y < N - 1 ? zq[pad8(dct_place(y + 1, N))] : u;
    const double f = -a.wy * (y > 0 && y < N - 1 ? 0.5 : 1.0);
    *reinterpret_cast<float4 *>(a.uv + (size_t)y * N + c0 + 2 * sq) =
        make_float4((float)u.y, (float)(f * (hi.y - lo.y)), (float)u.x,
                    (float)(f * (hi.x - lo.x)));
  }
}

// Rows back: one complex FFT per row (u, Dy u) -> (phi, E_y).
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
dct_field_kernel(DctArgs a) {
  extern __shared__ double2 zsh[];
  const int N = a.G, n8 = N >> 3;
  const int seq = threadIdx.x / n8, j0 = threadIdx.x - seq * n8;
  double2 *z = zsh + seq * pad8(N);
  const size_t r = (size_t)(blockIdx.x * a.seqs + seq) * N;
  const double inv_n = 1.0 / (double)N;
  for (int k = j0; k <= N / 2; k += n8) {
    const int km = k ? N - k : 0;
    const float2 f = a.uv[r + k], g = a.uv[r + km];
    const double2 h = make_double2(f.x * inv_n, f.y * inv_n);
    const double2 hm = k ? make_double2(g.x * inv_n, g.y * inv_n) : make_double2(0.0, 0.0);
    const double2 w = a.qt[k];
    double2 zk, zm;
    idct_pair(h, hm, w.x, w.y, zk, zm);
    z[pad8(k)] = zk;
    if (km != k) z[pad8(km)] = zm;
  }
  fft_block(z, N, a.odd, j0, a.tw);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int x = j0 + i * n8;
    const double2 u = z[pad8(dct_place(x, N))];
    const double lo = x > 0 ? z[pad8(dct_place(x - 1, N))].y : u.y;
    const double hi = x < N - 1 ? z[pad8(dct_place(x + 1, N))].y : u.y;
    const double f = -a.wx * (x > 0 && x < N - 1 ? 0.5 : 1.0);
    a.ex[r + x] = (float)(f * (hi - lo));
    a.ey[r + x] = (float)u.x;
    if (a.phi) a.phi[r + x] = (float)u.y;
  }
}

using DctKernel = void (*)(DctArgs);

// Launches one of the three kernels for `total` sequences, `seqs` per block.
// Blocks of up to 512 threads may use 128 registers a thread; N / 8 of the
// grids above 4096 needs up to 1024 threads.
int dct_launch(DctKernel k512, DctKernel k1024, DctArgs a, int total, int seqs,
               cudaStream_t s) {
  const int threads = seqs * (a.G / 8);
  const int smem = seqs * pad8(a.G) * (int)sizeof(double2);
  DctKernel k = threads <= 512 ? k512 : k1024;
  if (smem > 48 * 1024) FX_TRY(raise_smem_limit((const void *)k, smem));
  a.seqs = seqs;
  k<<<total / seqs, threads, smem, s>>>(a);
  FX_CHECK_LAUNCH();
  return FX_OK;
}

}  // namespace

int dct_tables(int G, double wx, double wy, std::vector<double2> &tw,
               std::vector<double2> &qt, std::vector<double> &ax2,
               std::vector<double> &ay2) {
  const double pi = 3.14159265358979323846;
  tw.resize(G);
  qt.resize(G);
  ax2.resize(G);
  ay2.resize(G);
  for (int k = 0; k < G; ++k) {
    tw[k] = make_double2(std::cos(2.0 * pi * k / G), -std::sin(2.0 * pi * k / G));
    qt[k] = make_double2(std::cos(pi * k / (2.0 * G)), std::sin(pi * k / (2.0 * G)));
    const double ax = wx * std::cos(pi * k / G) - wx, ay = wy * std::cos(pi * k / G) - wy;
    ax2[k] = ax * ax;
    ay2[k] = ay * ay;
  }
  return FX_OK;
}

int dct_solve(fx_ctx *ctx, const DctArgs &args, cudaStream_t s) {
  DctArgs a = args;
  const int G = a.G;
  a.odd = G;
  while (a.odd % 2 == 0) a.odd /= 2;
  // Sequences per block: rows need 32 threads at least (N / 8 of them each);
  // columns take two sequences so that a block reads and writes whole
  // 32-byte sectors, one where shared memory (147 KB each at 8192) or the
  // 1024 threads of a block end.
  const int row_seqs = G >= 256 ? 1 : 2, col_seqs = G <= 4096 ? 2 : 1;
  FX_TRY(dct_launch(dct_rows_kernel<512>, dct_rows_kernel<1024>, a, G / 2, row_seqs, s));
  FX_TRY(dct_launch(dct_cols_kernel<512>, dct_cols_kernel<1024>, a, G / 2, col_seqs, s));
  FX_TRY(dct_launch(dct_field_kernel<512>, dct_field_kernel<1024>, a, G, row_seqs, s));
  ctx->launches += 3;
  return FX_OK;
}

}  // namespace fx
