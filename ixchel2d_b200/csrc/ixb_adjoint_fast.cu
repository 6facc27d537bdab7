// ixb_adjoint_fast.cu -- discrete adjoint of the energy iteration with the
// flow held fixed: the gradient of the hot-wall Nusselt number after K
// passes of the T sweeps (T-y then T-x, source/main.f90:985-1136) with
// respect to the Dirichlet value of every x-line on side a (the hot wall,
// x = 0).  The reference has no counterpart.
//
// With u, v frozen, every T sweep is affine in the temperatures: a line solve
// x = A^-1 (R T_in + f) with coefficients (AI, AD, BS, BN and the relaxed
// diagonal) that depend on the mesh and the velocities only, and f holding
// the boundary values.  The adjoint therefore needs no stored forward states:
// starting from the Nusselt number's weights, each sweep is reversed as
// mu = A^-T lambda (a transposed batched line solve) followed by
// lambda_in = R^T mu plus the lines the sweep copies, and the side-a
// boundary rows of the x-sweeps collect d Nu / d value += mu[row 0].
// A reversed sweep is one kernel that reads the sweep reversed before it as
// its mu and forms that one's R^T mu while it loads its right-hand sides, so
// that neither lambda nor the transposed rows pass through memory: 2
// launches and 6 loads per row and pass where staging, solving and
// scattering took 6 launches (256 x 256, 200 passes with the forward run:
// 7.8 ms then; with the passes resident, ixb_passes_fast.cu, 3.5 ms).
// Built with FMA contraction, like the fast forward assembly, whose
// coefficients it re-evaluates.  ixb_adjoint_energy_coupled extends this to
// K outer SIMPLE iterations of a flow that evolves but does not depend on
// the temperature, with checkpoints every C iterations.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstring>
#include <functional>
#include <vector>

#include "ixb_handle.h"
#include "ixb_nusselt.h"
#include "ixb_passes.h"

namespace ixb {
namespace {

struct Sweep {
  bool x;               // x-lines (fixed jj) or y-lines (fixed ii)
  int n;                // rows per line
  int nl;               // solved lines 2 .. nl+1
  const BCEntry* first;
  const BCEntry* last;
};

// lambda at a cell after sweep `s` was reversed: R^T mu + the lines it copies.
// `f` holds mu on the solved lines and lambda on the copied ones.
__device__ __forceinline__ double lambda_at(const Geo<double>& G, const Sweep& s, const double* coef, size_t fsz,
                                            double keep, const double* f, int ii, int jj) {
  const int L = s.x ? jj : ii, r = s.x ? ii - 1 : jj - 1, st = s.x ? G.LD : 1;
  const int c0 = G.at(ii, jj);
  auto solved = [&](int l) { return l >= 2 && l <= s.nl + 1; };
  const bool interior = r >= 1 && r <= s.n - 2;
  double v = 0.0;
  if (!solved(L)) v = __ldg(f + c0);
  else if (interior) v = coef[C_DG * fsz + c0] * keep * __ldg(f + c0);
  // rows of the neighbouring lines that read this cell through d
  if (interior && solved(L + 1)) v -= coef[(s.x ? C_BS : C_AI) * fsz + c0 + st] * __ldg(f + c0 + st);
  if (interior && solved(L - 1)) v -= coef[(s.x ? C_BN : C_AD) * fsz + c0 - st] * __ldg(f + c0 - st);
  return v;
}

__global__ void adj_lambda_kernel(const Geo<double> G, const Sweep s, const double* __restrict__ coef, size_t fsz,
                                  double keep, const double* __restrict__ f, double* __restrict__ lam) {
  const int ii = 1 + blockIdx.x * blockDim.x + threadIdx.x, jj = 1 + blockIdx.y;
  if (ii <= G.mi + 1) lam[G.at(ii, jj)] = lambda_at(G, s, coef, fsz, keep, f, ii, jj);
}

// One sweep reversed: CTA = TL adjacent lines, thread t: chunk t / TL (M rows)
// of line L0 + t % TL, in registers from the loads to mu.  The right-hand
// sides are lambda after the sweep `prev` (FIRST: `f` is lambda itself); the
// matrix is the transposed one (a'_r = c_{r-1}, b'_r = b_r, c'_r = a_{r+1}).
// Bound by latency: one wave of CTAs, a chunk's loads, the reduced system.
template <bool X, bool FIRST, int TL, int GT, int M>
__global__ void __launch_bounds__(TL * GT)
    adj_sweep_kernel(const Geo<double> G, const Sweep s, const Sweep prev, const double* __restrict__ coef, size_t fsz,
                     double keep, const double* __restrict__ f, double* __restrict__ mu, double* __restrict__ grad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* red = reinterpret_cast<double*>(smem_raw);
  const int t = threadIdx.x, l = t % TL, k = t / TL, L = 1 + blockIdx.x * TL + l;
  const bool active = L >= 2 && L <= s.nl + 1, there = L <= s.nl + 2;
  const double *ca = coef + (X ? C_AI : C_BS) * fsz, *cc = coef + (X ? C_AD : C_BN) * fsz, *cd = coef + C_DG * fsz;
  const int c00 = X ? G.at(1, L) : G.at(L, 1), st = X ? 1 : G.LD;
  int t0 = 1, t1 = 1;  // boundary row types
  if (active) { t0 = s.first[L].type; t1 = s.last[L].type; }
  Chunk<double, M> ch;
#pragma unroll
  for (int it = 0; it < M; ++it) {
    const int r = k * M + it, c0 = c00 + r * st;
    double a = 0.0, b = 1.0, c = 0.0, d = 0.0;
    if (there && r < s.n) {
      const int ii = X ? r + 1 : L, jj = X ? L : r + 1;
      d = FIRST ? __ldg(f + c0) : lambda_at(G, prev, coef, fsz, keep, f, ii, jj);
      if (!active) {
        mu[c0] = d;
        d = 0.0;
      } else {
        if (r == 0) b = t0 == 2 ? -1.0 : 1.0;
        else if (r < s.n - 1) b = __ldg(cd + c0);
        if (r == 1) a = t0 == 2 ? 1.0 : 0.0;
        else if (r > 1) a = __ldg(cc + c0 - st);
        if (r == s.n - 2) c = t1 == 2 ? -1.0 : 0.0;
        else if (r < s.n - 2) c = __ldg(ca + c0 + st);
      }
    }
    ch.a[it] = a; ch.b[it] = b; ch.c[it] = c; ch.d[it] = d;
  }
  ch.eliminate();
  double x0, xl;
  reduced_pcr<double, true>(red, TL * GT, TL, GT, t, k, active, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD, x0, xl,
                            [](bool q) { return (bool)__syncthreads_or(q); });
  ch.substitute(x0, xl);
  if (!active) return;
#pragma unroll
  for (int it = 0; it < M; ++it) {
    const int r = k * M + it;
    if (r < s.n) mu[c00 + r * st] = ch.d[it];
    if (X && r == 0) grad[L] += ch.d[it];
  }
}

struct SweepArgs {
  Geo<double> G;
  Sweep s, prev;
  const double* coef;
  size_t fsz;
  double keep;
  const double* f;
  double* mu;
  double* grad;
};

template <bool X, bool FIRST, int TL, int GT, int M>
cudaError_t adj_sweep_go(const SweepArgs& q, cudaStream_t st) {
  auto k = adj_sweep_kernel<X, FIRST, TL, GT, M>;
  const size_t smem = (size_t)9 * TL * GT * sizeof(double);
  cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  k<<<(q.s.nl + 2 + TL - 1) / TL, TL * GT, smem, st>>>(q.G, q.s, q.prev, q.coef, q.fsz, q.keep, q.f, q.mu, q.grad);
  return cudaGetLastError();
}

// The fewest threads that leave 3 rows each, up to 256 per x-line and 128 per
// y-line (four of them make 32-byte pieces of a row), then longer chunks;
// lines beyond those by 1024 threads.  A line has at most 6001 rows.
template <bool X, bool FIRST>
cudaError_t adj_sweep(const SweepArgs& q, cudaStream_t st) {
  constexpr int TL = X ? 1 : 4, GM = X ? 256 : 128;
  const int n = q.s.n;
  if (n <= 192) return adj_sweep_go<X, FIRST, TL, 64, 3>(q, st);
  if (n <= 384) return adj_sweep_go<X, FIRST, TL, 128, 3>(q, st);
  if (X && n <= 768) return adj_sweep_go<X, FIRST, TL, GM, 3>(q, st);
  if (n <= 4 * GM) return adj_sweep_go<X, FIRST, TL, GM, 4>(q, st);
  if (n <= 6 * GM) return adj_sweep_go<X, FIRST, TL, GM, 6>(q, st);
  if (n <= 8 * GM) return adj_sweep_go<X, FIRST, TL, GM, 8>(q, st);
  if (n <= 3072) return adj_sweep_go<X, FIRST, 1, 1024, 3>(q, st);
  return adj_sweep_go<X, FIRST, 1, 1024, 6>(q, st);
}

}  // namespace
}  // namespace ixb

using namespace ixb;

#define ACK(x)                   \
  do {                           \
    cudaError_t e_ = (x);        \
    if (e_ != cudaSuccess) {     \
      h->last_cuda = e_;         \
      return IXB_ECUDA;          \
    }                            \
  } while (0)
#define TRY(x)                   \
  do {                           \
    const int s_ = (x);          \
    if (s_ != IXB_OK) return s_; \
  } while (0)

namespace {

// Workspace, objective weights and reversed (T-y, T-x) passes shared by the
// two adjoint entry points.
struct AdjCtx {
  ixb_handle* h;
  size_t fsz = 0;
  double *coef = nullptr, *lam = nullptr, *mx = nullptr, *my = nullptr, *gd = nullptr;
  Geo<double> G{};
  Sweep sx{}, sy{};
  double keep = 0.0;     // 1 - relaxation
  bool started = false;  // the T-y sweep reversed last left its mu in my; else lam holds lambda

  int init(int j0, int j1) {
    const int mi = h->mi, nj = h->nj;
    fsz = h->fsz;
    const size_t need = (C_COUNT + 3) * fsz + (size_t)(nj + 2) + sizeof(GridWords) / sizeof(double);
    if (h->adj_size < need) {
      if (h->adj_pool) cudaFree(h->adj_pool);
      h->adj_pool = nullptr;
      h->adj_size = 0;
      ACK(cudaMalloc(&h->adj_pool, need * sizeof(double)));
      h->adj_size = need;
    }
    coef = h->adj_pool;
    lam = coef + C_COUNT * fsz;
    mx = lam + fsz;
    my = mx + fsz;
    gd = my + fsz;
    started = false;
    G = handle_geo(h);
    const BCEntry* base = h->bc + (size_t)2 * 4 * h->bcstride;  // T tables, sides a b c d
    sx = Sweep{true, mi + 1, nj - 1, base + 0 * (size_t)h->bcstride, base + 2 * (size_t)h->bcstride};
    sy = Sweep{false, nj + 1, mi - 1, base + 1 * (size_t)h->bcstride, base + 3 * (size_t)h->bcstride};
    keep = 1.0 - h->prm.rel_ener;
    // the objective's weights: Nu is linear in T (the wall-normal 3-point
    // derivative integrated panel by panel), evaluated here on unit fields
    std::vector<double> along(nj + 2, 0.0), across(mi + 2, 0.0);
    for (int j = 1; j <= nj + 1; ++j) along[j] = h->yp[j - 1];
    for (int i = 1; i <= mi + 1; ++i) across[i] = h->xp[i - 1];
    std::vector<double> w((size_t)fsz, 0.0);
    for (int k = j0; k <= j1 + 2; ++k)
      for (int l = 1; l <= 3; ++l)
        w[(size_t)(k - 1) * h->LD + (l - 1)] = nusselt_weight(along.data(), across.data(), mi + 1, j0, j1, k, l);
    ACK(cudaMemcpyAsync(lam, w.data(), fsz * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    ACK(cudaMemsetAsync(gd, 0, (nj + 2) * sizeof(double), h->stream));
    ACK(cudaStreamSynchronize(h->stream));  // w leaves scope
    return IXB_OK;
  }

  // coefficients of the energy rows at the handle's current velocities; the
  // last reversed sweep's lambda is formed with the ones it ran with first
  int coefficients() {
    if (started) {
      adj_lambda_kernel<<<dim3((h->mi + 1 + 127) / 128, h->nj + 1), 128, 0, h->stream>>>(G, sy, coef, fsz, keep, my, lam);
      ACK(cudaGetLastError());
      started = false;
    }
    SweepIO<double> io = handle_fixed_io(h, EQ_TX);
    io.in = h->zero;
    ACK(energy_coef_launch(G, io, coef, fsz, h->stream));
    return IXB_OK;
  }

  // one (T-y, T-x) pass, reversed: T-x first
  int pass() {
    const SweepArgs x{G, sx, sy, coef, fsz, keep, started ? my : lam, mx, gd};
    const SweepArgs y{G, sy, sx, coef, fsz, keep, mx, my, gd};
    ACK((started ? adj_sweep<true, false>(x, h->stream) : adj_sweep<true, true>(x, h->stream)));
    ACK((adj_sweep<false, false>(y, h->stream)));
    started = true;
    return IXB_OK;
  }

  int finish(double* grad) {
    const int nj = h->nj;
    std::vector<double> g(nj + 2);
    ACK(cudaMemcpyAsync(g.data(), gd, (nj + 2) * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    ACK(cudaStreamSynchronize(h->stream));
    for (int jj = 1; jj <= nj + 1; ++jj) grad[jj - 1] = g[jj];
    return IXB_OK;
  }
};

int check_range(const ixb_handle* h, int j0, int j1) {
  if (j0 < 1 || j1 < j0) return IXB_EINVAL;
  for (int k = j0; k <= j1; k += 2)
    if (k + 2 > h->nj + 1) return IXB_EINVAL;
  return IXB_OK;
}

}  // namespace

extern "C" int ixb_adjoint_energy(ixb_handle* h, int K, int j0, int j1, double* grad) {
  if (!h || K < 0 || !grad) return IXB_EINVAL;
  const int st0 = handle_ready(h);
  if (st0 != IXB_OK) return st0;
  TRY(check_range(h, j0, j1));
  AdjCtx A{h};
  TRY(A.init(j0, j1));
  TRY(A.coefficients());  // the frozen velocities
  // K passes of (T-y, T-x), reversed: the first reads the objective's weights;
  // the others run in one resident kernel where the grid fits it, else in a
  // WHILE graph kLoopUnroll at a time (rebuilt when the handle or its
  // workspace changes) and what is left as plain launches
  if (K > 0) TRY(A.pass());
  int left = std::max(K - 1, 0);
  PassArgs P{};
  if (left > 0 && handle_resident_passes(h, &P)) {
    P.coef = A.coef; P.f0 = A.my; P.f1 = A.mx; P.grad = A.gd; P.passes = left;
    int done = 0;
    TRY(handle_run_passes(h, true, P, reinterpret_cast<GridWords*>(A.gd + h->nj + 2), &done));
    left -= done;
  }
  const std::function<int()> pass = [&A]() -> int { return A.pass(); };
  if (left >= kLoopUnroll) {
    if (h->agraph_dirty || !h->agraph_exec || h->agraph_pool != h->adj_pool) {
      const int r = handle_build_loop_graph(h, pass, kLoopUnroll, &h->agraph, &h->agraph_exec);
      if (r != IXB_OK) return r;
      h->agraph_dirty = false;
      h->agraph_pool = h->adj_pool;
    }
    const int r = handle_run_loop_graph(h, h->agraph_exec, left / kLoopUnroll);
    if (r != IXB_OK) return r;
  }
  for (int k = 0; k < left % kLoopUnroll; ++k) TRY(pass());
  return A.finish(grad);
}

// The energy adjoint through K outer SIMPLE iterations whose flow evolves
// but does not depend on the temperature (Ri = Riy = 0: the buoyancy terms
// are exact zeros, so the velocities of every iteration are the same for
// any wall temperature).  T after K iterations is then a composition of
// affine T passes, the passes of iteration k with the coefficients of that
// iteration's velocities, and the gradient is exact.  Forward: K single
// outer iterations, recording each one's T passes and checkpointing the
// seven state fields every C iterations.  Reverse, segment by segment:
// restore the segment's checkpoint, recompute it storing u, v after every
// iteration, then reverse its iterations' T passes with their coefficients.
extern "C" int ixb_adjoint_energy_coupled(ixb_handle* h, int K, int C, int j0, int j1, double* grad,
                                          double* nu0) {
  if (!h || K < 1 || C < 1 || !grad) return IXB_EINVAL;
  const int st0 = handle_ready(h);
  if (st0 != IXB_OK) return st0;
  TRY(check_range(h, j0, j1));
  if (h->prm.Ri != 0.0 || h->prm.Riy != 0.0) return IXB_EINVAL;  // the flow would depend on T
  if (C > K) C = K;
  const size_t fsz = h->fsz, fb = fsz * sizeof(double);
  const int nseg = (K + C - 1) / C;
  // checkpoints: u v p T u_ant v_ant T_ant at iterations 0, C, 2C, ... and K
  double* pool = nullptr;
  const size_t ncp = (size_t)nseg + 1;
  ACK(cudaMalloc(&pool, (ncp * 7 + (size_t)2 * C) * fb));
  double* useg = pool + ncp * 7 * fsz;  // u after each iteration of a segment
  double* vseg = useg + (size_t)C * fsz;
  struct Saved { int iter_ecuaci, iter_simple; };
  std::vector<Saved> counters(ncp);
  auto fields = [h]() {
    return std::array<double*, 7>{h->u[h->cu], h->v[h->cv], h->p, h->T[h->cT], h->u_ant, h->v_ant, h->T_ant};
  };
  auto save = [&](size_t slot) -> int {
    const auto f = fields();
    for (int k = 0; k < 7; ++k)
      ACK(cudaMemcpyAsync(pool + (slot * 7 + k) * fsz, f[k], fb, cudaMemcpyDeviceToDevice, h->stream));
    counters[slot] = Saved{h->iter_ecuaci, h->iter_simple};
    return IXB_OK;
  };
  auto restore = [&](size_t slot) -> int {
    const auto f = fields();
    for (int k = 0; k < 7; ++k)
      ACK(cudaMemcpyAsync(f[k], pool + (slot * 7 + k) * fsz, fb, cudaMemcpyDeviceToDevice, h->stream));
    h->iter_ecuaci = counters[slot].iter_ecuaci;
    h->iter_simple = counters[slot].iter_simple;
    return IXB_OK;
  };
  int st = IXB_OK;
  std::vector<int> passes(K + 1, 0);  // T passes of iteration k
  auto run = [&]() -> int {
    // forward: K iterations, one call each (their T pass counts)
    TRY(save(0));
    for (int k = 1; k <= K; ++k) {
      ixb_report rep{};
      TRY(ixb_simple_iterations(h, 1, &rep));
      passes[k] = (int)rep.n_ener;
      if (k % C == 0 && k < K) TRY(save((size_t)(k / C)));
    }
    TRY(save(ncp - 1));  // the final state, restored at the end
    if (nu0) TRY(ixb_nusselt_x(h, j0, j1, nu0, nullptr));
    AdjCtx A{h};
    TRY(A.init(j0, j1));
    for (int seg = nseg - 1; seg >= 0; --seg) {
      const int k0 = seg * C, k1 = std::min(K, k0 + C);  // iterations k0+1 .. k1
      TRY(restore((size_t)seg));
      for (int k = k0 + 1; k <= k1; ++k) {
        ixb_report rep{};
        TRY(ixb_simple_iterations(h, 1, &rep));
        if ((int)rep.n_ener != passes[k]) return IXB_ESTATE;  // the recomputation must retrace the forward
        ACK(cudaMemcpyAsync(useg + (size_t)(k - k0 - 1) * fsz, h->u[h->cu], fb, cudaMemcpyDeviceToDevice, h->stream));
        ACK(cudaMemcpyAsync(vseg + (size_t)(k - k0 - 1) * fsz, h->v[h->cv], fb, cudaMemcpyDeviceToDevice, h->stream));
      }
      for (int k = k1; k > k0; --k) {
        ACK(cudaMemcpyAsync(h->u[h->cu], useg + (size_t)(k - k0 - 1) * fsz, fb, cudaMemcpyDeviceToDevice, h->stream));
        ACK(cudaMemcpyAsync(h->v[h->cv], vseg + (size_t)(k - k0 - 1) * fsz, fb, cudaMemcpyDeviceToDevice, h->stream));
        TRY(A.coefficients());
        for (int q = 0; q < passes[k]; ++q) TRY(A.pass());
      }
    }
    TRY(restore(ncp - 1));
    return A.finish(grad);
  };
  st = run();
  cudaStreamSynchronize(h->stream);
  cudaFree(pool);
  return st;
}
