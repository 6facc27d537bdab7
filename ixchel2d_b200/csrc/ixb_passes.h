// ixb_passes.h -- many passes of the energy sweeps in one launch
// (ixb_passes_fast.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "ixb_grid.h"
#include "ixb_internal.h"

namespace ixb {

// coefficient arrays (field layout) of the energy rows: AI, AD, BS, BN, the
// relaxed diagonal, and the part of the right-hand side that is not T's
enum { C_AI = 0, C_AD, C_BS, C_BN, C_DG, C_R0, C_COUNT };

constexpr int kPassesPerLaunch = 4096;

struct PassArgs {
  Geo<double> G;
  const double* coef;  // C_COUNT fields of fsz elements
  size_t fsz;
  double keep;         // 1 - relaxation
  const BCEntry *first_x, *last_x, *first_y, *last_y;
  double *f0, *f1;     // f0 -> f1 -> f0 in every pass
  double* grad;        // transposed passes: += the first row's values, by x-line
  GridWaits waits;
  int passes;
  int lx, cx, ly, cy;  // lines per CTA and chunks per line of either direction
  int grid;
};

// energy rows at the velocities of io, whose `in` is the zero field
cudaError_t energy_coef_launch(const Geo<double>& G, const SweepIO<double>& io, double* coef, size_t fsz,
                               cudaStream_t st);
// Whether a grid's lines, factored in both directions, fit one CTA per SM;
// fills lx, cx, ly, cy, grid.
bool energy_passes_fit(int mi, int nj, int nsm, PassArgs* a);
// a.passes (T-y, T-x) passes, or their transposes (T-x first); the launches
// from number expire_from on get a.waits.expire
cudaError_t energy_passes_launch(bool reverse, const PassArgs& a, int expire_from, cudaStream_t st);

}  // namespace ixb
