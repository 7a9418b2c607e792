// fx_dct.cuh -- the fast-transform DCT Poisson solve (fx_dct.cu).
#pragma once
#include <vector>

#include "fx_internal.h"

namespace fx {

struct DctArgs {
  int G;               // bins per side, a multiple of 128 up to 8192
  int odd;             // odd part of G (set by dct_solve)
  int seqs;            // sequences per block (set by dct_solve)
  unsigned long long *acc;  // G x G fixed-point areas, read and zeroed
  double inv_bin_area, target;
  double level;        // taken off the density before the transforms
  double wx, wy;       // 1 / bin width, height
  const double2 *tw;   // G: e^{-2 pi i k / G}
  const double2 *qt;   // G: (cos, sin)(pi k / 2G)
  const double *ax2, *ay2;  // G each: the two parts of the eigenvalue
  float *rho;          // charge grid, or null
  float *t1;           // G x G scratch: row spectra
  float2 *uv;          // G x G scratch: (u, Dy u), spectral along x
  float *ex, *ey;      // field
  float *phi;          // potential, or null
};

// Host tables of a G-bin grid (the eigenvalues of force_electrostatic.py:72-86
// split by axis).
int dct_tables(int G, double wx, double wy, std::vector<double2> &tw,
               std::vector<double2> &qt, std::vector<double> &ax2,
               std::vector<double> &ay2);
// Areas -> field, in three launches on s.
int dct_solve(fx_ctx *ctx, const DctArgs &a, cudaStream_t s);

}  // namespace fx
