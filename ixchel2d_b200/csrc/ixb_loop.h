// ixb_loop.h -- the resident SIMPLE loop: launch parameters shared by its
// kernels (ixb_loop.cuh) and the host side (ixb_api.cu).
#pragma once
#include <cuda_runtime.h>

#include "ixb_handle.h"

namespace ixb {

// Rows per chunk of the line solves, and lines per CTA of an x-sweep: a
// thread assembles a column of three cells in both directions.
constexpr int kLoopM = 3;
// Threads per CTA of the largest variant: one thread per column of an x-line
// of up to 768 rows, or six y-lines of up to 384 rows.  One CTA per SM.
constexpr int kLoopThreads = 768;
constexpr int kLoopLinesY = 8;

// Work per CTA: x_lines adjacent x-lines solved by gx threads each, y_lines
// adjacent y-lines solved by gy threads each.
struct LoopShape {
  int grid, threads;
  int x_lines, gx, y_lines, gy;
};

// What a launch runs: the loop, or one part of an outer pass (the host then
// reads its norms and applies the exit tests)
enum LoopPart { LOOP_ALL = 0, LOOP_MOMENTUM, LOOP_PRESSURE_FIRST, LOOP_PRESSURE, LOOP_CORRECT, LOOP_ENERGY,
                LOOP_RESIDUAL };

struct LoopArgs {
  Geo<double> G;
  double *u[2], *v[2], *T[2], *pc[2];
  double *p, *au, *av, *b_o, *resu;
  const double *u_ant, *v_ant, *T_ant;
  const double *fcon[3], *flin[3];
  const BCEntry* bc;
  int bcstride;
  Ctl* ctl;
  double* partials;  // [N_COUNT][grid]
  GridWaits waits;
  LoopShape s;
  double* norms;     // N_COUNT, written by a single-part launch
  int max_outer;     // outer passes this launch may run
  int part;          // LoopPart: the whole loop, or one part of it for the host-driven loop
};

// Whether the loop kernel covers an mi x nj grid on nsm SMs, and its shape.
bool loop_shape(int mi, int nj, int nsm, LoopShape* s);
cudaError_t loop_launch(int form, const LoopArgs& a, cudaStream_t st);
template <int SOLVER>
cudaError_t loop_launch_form(const LoopArgs& a, cudaStream_t st);

}  // namespace ixb
