// ixb_loop.cu -- host side of the resident SIMPLE loop: which grids it
// covers and how their lines spread over the GPU.
#include "ixb_loop.h"

#include <algorithm>

namespace ixb {

namespace {
int up32(int n) { return (n + 31) / 32 * 32; }
}  // namespace

// Three rows per thread and at most one tile of lines per CTA: x-lines of up
// to 768 rows, y-lines of up to 384, all lines resident at once.
bool loop_shape(int mi, int nj, int nsm, LoopShape* out) {
  LoopShape s{};
  const int lx = nj + 1, ly = mi + 1;  // lines of the widest sweep of each direction; also its rows the other way
  const int chunks_x = (mi + 1 + kLoopM - 1) / kLoopM, chunks_y = (nj + 1 + kLoopM - 1) / kLoopM;
  s.gx = up32(chunks_x);
  s.gy = chunks_y;
  // as few CTAs as three x-lines and four y-lines (one 32-byte sector of a
  // row) each allow: the grid barrier gets cheaper with fewer of them
  s.grid = std::min(nsm, std::max((lx + kLoopM - 1) / kLoopM, (ly + 3) / 4));
  s.x_lines = (lx + s.grid - 1) / s.grid;
  s.y_lines = (ly + s.grid - 1) / s.grid;
  if (s.x_lines > kLoopM || s.y_lines > kLoopLinesY) return false;
  s.threads = std::max(std::max(up32(mi + 1), s.x_lines * s.gx), up32(s.y_lines * s.gy));
  if (s.threads > kLoopThreads) return false;
  *out = s;
  return true;
}

cudaError_t loop_launch(int form, const LoopArgs& a, cudaStream_t st) {
  return form == SOLVER_MIXED ? loop_launch_form<SOLVER_MIXED>(a, st) : loop_launch_form<IXB_SOLVER_HYBRID>(a, st);
}

}  // namespace ixb
