// ixb_adjoint_simple.cu -- discrete adjoint of the full coupled SIMPLE outer
// iteration (momentum, pressure correction, velocity/pressure update and
// energy, main.f90:404-1136 with one pass of each equation per outer
// iteration), for flows that depend on the temperature through buoyancy
// (natural and mixed convection).  The gradient is that of the hot-wall
// Nusselt number (ixb_nusselt_x, wall x = 0) after K outer iterations with
// respect to the Dirichlet value of every x-line on side a.  The reference
// has no counterpart.
//
// Every sweep of the iteration maps its input state s (the swept field and
// the fields its rows read) to x_out, where A(s) x_out = d(s) on the solved
// lines and x_out = x_in on the others.  Its adjoint, given lambda (the
// adjoint of x_out):
//   mu = A(s)^-T lambda                      (transposed batched line solve)
//   s_bar += sum over rows r of  mu_r d(d_r)/ds - mu_r (x_{r-1} d(a_r)/ds
//            + x_r d(b_r)/ds + x_{r+1} d(c_r)/ds)
//   x_in_bar += lambda                       (on the unsolved lines)
// The row's derivatives are taken in reverse: for the weights (-mu x, mu) of
// (a, b, c, d) the adjoints of the row's coefficients, face velocities and
// stencil values follow by hand (about twice the row's own arithmetic, where
// one dual number per stencil value took thirteen times it), and are added to
// the stencil positions with atomic adds.  The rows are those of
// ixb_device.cuh in the fast form (the reference's formulas,
// mod_ec_momento.f90:365-1098, :145-355, mod_ec_energia.f90:119-443).  The
// velocity/pressure update (main.f90:931-962) has a hand-written adjoint.
//
// A reversed sweep is one kernel: a CTA evaluates its lines' rows, places
// them transposed in shared memory, solves, and scatters.  As row, transpose,
// line-solve and scatter kernels it was 44 launches per reversed iteration
// instead of 9, and bound by them up to 256x256 (128x128, 30 iterations, a
// checkpoint every 10: 20.3 ms per gradient then, 4.7 now).  The recomputed sweeps and
// the reversed ones are launched with programmatic serialisation: each is a
// few microseconds of latency, and the next one's launch overlaps it.
//
// Forward: K outer iterations (the library's loop, one pass of each equation),
// the state saved every C iterations.  Reverse, segment by segment from the
// last: restore the segment's checkpoint, recompute its iterations sweep by
// sweep, each writing its field of the store directly, then reverse the
// phases of each iteration from the last.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <cmath>
#include <cstring>
#include <vector>

#include "ixb_handle.h"
#include "ixb_nusselt.h"

namespace ixb {
namespace {

// ---------------------------------------------------------------------------
// stencils: the field and offset of every row input
// ---------------------------------------------------------------------------
enum Fld { F_U = 0, F_V, F_T, F_P, F_PC, F_AU, F_AV, F_COUNT, F_NONE = -1 };
struct Tap {
  int f, di, dj;
};
constexpr int NS = 13;  // stencil inputs of a row (the energy rows use 9)
// groups: 0 u rows, 1 v rows, 2 p' rows, 3 T rows
constexpr Tap kStencil[4][NS] = {
    {{F_U, 0, 0}, {F_U, 1, 0}, {F_U, -1, 0}, {F_U, 0, -1}, {F_U, 0, 1}, {F_V, 0, 0}, {F_V, 1, 0}, {F_V, 0, -1},
     {F_V, 1, -1}, {F_T, 0, 0}, {F_T, 1, 0}, {F_P, 0, 0}, {F_P, 1, 0}},
    {{F_V, 0, 0}, {F_V, 0, 1}, {F_V, 0, -1}, {F_V, -1, 0}, {F_V, 1, 0}, {F_U, 0, 0}, {F_U, 0, 1}, {F_U, -1, 0},
     {F_U, -1, 1}, {F_T, 0, 0}, {F_T, 0, 1}, {F_P, 0, 0}, {F_P, 0, 1}},
    {{F_PC, 0, 0}, {F_PC, 1, 0}, {F_PC, -1, 0}, {F_PC, 0, -1}, {F_PC, 0, 1}, {F_AU, -1, 0}, {F_AU, 0, 0},
     {F_AV, 0, -1}, {F_AV, 0, 0}, {F_U, 0, 0}, {F_U, -1, 0}, {F_V, 0, 0}, {F_V, 0, -1}},
    {{F_T, 0, 0}, {F_T, 1, 0}, {F_T, -1, 0}, {F_T, 0, -1}, {F_T, 0, 1}, {F_U, 0, 0}, {F_U, -1, 0}, {F_V, 0, 0},
     {F_V, 0, -1}, {F_NONE, 0, 0}, {F_NONE, 0, 0}, {F_NONE, 0, 0}, {F_NONE, 0, 0}}};
constexpr int eq_group(int eq) { return eq / 2; }
// the swept field of a group
constexpr int group_field(int g) { return g == 0 ? F_U : g == 1 ? F_V : g == 2 ? F_PC : F_T; }

// The pre-sweep state a sweep's rows read, its constants and boundary rows.
struct SweepState {
  const double* f[F_COUNT];   // u, v, T, p, p', au, av as the sweep reads them
  const double* x_out;        // the swept field after the sweep
  const double* ant;          // u_ant / v_ant / T_ant (null for p')
  const double* fcon;         // sources (null: none)
  const double* flin;
  const BCEntry* first;       // boundary rows (null: p', Dirichlet 0)
  const BCEntry* last;
  int eq, n, line_lo, line_hi, nfull;
};

struct AdjFields {
  double* f[F_COUNT];  // adjoints of u, v, T, p, p', au, av (field layout)
};

// The coefficients of a row (AI, AD, BS, BN negative, b the relaxed diagonal)
// and, with the face velocities (ui, ud, vs, vn) or au, av (p'), the
// derivative of each coefficient by its own face value.
struct Links {
  double AI, AD, BS, BN, b;
  double dI, dD, dS, dN;
  double dx, dy;  // the cell's widths
};

// Coefficient -(cond max(0, 1 - |vel| m)^5 + max(0, vel w)) and its derivative
// by vel; at the kinks of |.| and max the branch taken counts.
__device__ __forceinline__ void link_d(double cond, double m, double vel, double w, double& val, double& der) {
  const double t = fmax(0.0, fma(-fabs(vel), m, 1.0)), t2 = t * t, t4 = t2 * t2;
  const bool up = vel * w > 0.0;
  val = -fma(cond, t * t4, up ? vel * w : 0.0);
  const double dl = 5.0 * cond * t4 * m;
  der = (vel < 0.0 ? -dl : dl) - (up ? w : 0.0);
}

template <int GRP>
__device__ __forceinline__ Links links(const Geo<double>& G, const double (&x)[NS], double flin, int ii, int jj) {
  Links k;
  if constexpr (GRP == 0) {
    const double fi = G.met(M_FEXU, ii), fm = G.met(M_FEXU, ii - 1), fp = G.met(M_FEXP, ii);
    k.dx = G.met(M_DXU, ii);
    k.dy = G.met(M_DYU, jj);
    const double ud = fi * x[1] + (1.0 - fi) * x[0], ui = fm * x[0] + (1.0 - fm) * x[2];
    const double vn = fp * x[6] + (1.0 - fp) * x[5], vs = fp * x[8] + (1.0 - fp) * x[7];
    link_d(k.dy * G.met(M_GRDXP, ii), G.met(M_PEXP, ii), ui, k.dy, k.AI, k.dI);
    link_d(k.dy * G.met(M_GRDXP, ii + 1), G.met(M_PEXP, ii + 1), ud, -k.dy, k.AD, k.dD);
    link_d(k.dx * G.met(M_GRDYV, jj - 1), G.met(M_PEYV, jj - 1), vs, k.dx, k.BS, k.dS);
    link_d(k.dx * G.met(M_GRDYV, jj), G.met(M_PEYV, jj), vn, -k.dx, k.BN, k.dN);
  } else if constexpr (GRP == 1) {
    const double fp = G.met(M_FEYP, jj), fj = G.met(M_FEYV, jj), fm = G.met(M_FEYV, jj - 1);
    k.dx = G.met(M_DXV, ii);
    k.dy = G.met(M_DYV, jj);
    const double ud = fp * x[6] + (1.0 - fp) * x[5], ui = fp * x[8] + (1.0 - fp) * x[7];
    const double vn = fj * x[1] + (1.0 - fj) * x[0], vs = fm * x[0] + (1.0 - fm) * x[2];
    link_d(k.dy * G.met(M_GRDXU, ii - 1), G.met(M_PEXU, ii - 1), ui, k.dy, k.AI, k.dI);
    link_d(k.dy * G.met(M_GRDXU, ii), G.met(M_PEXU, ii), ud, -k.dy, k.AD, k.dD);
    link_d(k.dx * G.met(M_GRDYP, jj), G.met(M_PEYP, jj), vs, k.dx, k.BS, k.dS);
    link_d(k.dx * G.met(M_GRDYP, jj + 1), G.met(M_PEYP, jj + 1), vn, -k.dx, k.BN, k.dN);
  } else if constexpr (GRP == 2) {
    k.dx = G.met(M_DXP, ii);
    k.dy = G.met(M_DYP, jj);
    const double ri = fast_rcp(x[5]), rd = fast_rcp(x[6]), rs = fast_rcp(x[7]), rn = fast_rcp(x[8]);
    k.AI = -(k.dy * k.dy) * ri; k.AD = -(k.dy * k.dy) * rd;
    k.BS = -(k.dx * k.dx) * rs; k.BN = -(k.dx * k.dx) * rn;
    k.dI = -k.AI * ri; k.dD = -k.AD * rd; k.dS = -k.BS * rs; k.dN = -k.BN * rn;
    k.b = (-k.AI - k.AD - k.BS - k.BN) * G.inv_rel_pres;
    return k;
  } else {
    k.dx = G.met(M_DXP, ii);
    k.dy = G.met(M_DYP, jj);
    link_d(k.dy * G.met(M_HRDXU, ii - 1), G.met(M_PHXU, ii - 1), x[6], k.dy, k.AI, k.dI);
    link_d(k.dy * G.met(M_HRDXU, ii), G.met(M_PHXU, ii), x[5], -k.dy, k.AD, k.dD);
    link_d(k.dx * G.met(M_HRDYV, jj - 1), G.met(M_PHYV, jj - 1), x[8], k.dx, k.BS, k.dS);
    link_d(k.dx * G.met(M_HRDYV, jj), G.met(M_PHYV, jj), x[7], -k.dx, k.BN, k.dN);
  }
  const double S = k.dx * k.dy;
  k.b = (-k.AI - k.AD - k.BS - k.BN - S * flin + S * G.inv_dt) * (GRP == 3 ? G.inv_rel_ener : G.inv_rel_vel);
  return k;
}

// Adjoints g of the stencil values of a row for the weights wa, wb, wc, wd of
// (a, b, c, d); X: the row along x (a = AI, c = AD), else along y.
template <int GRP, bool X>
__device__ __forceinline__ void row_back(const Geo<double>& G, const Links& k, const double (&x)[NS], int ii, int jj,
                                         double wa, double wb, double wc, double wd, double (&g)[NS]) {
  const double rel = GRP == 2 ? G.rel_pres : GRP == 3 ? G.rel_ener : G.rel_vel;
  const double irel = GRP == 2 ? G.inv_rel_pres : GRP == 3 ? G.inv_rel_ener : G.inv_rel_vel;
#pragma unroll
  for (int q = 0; q < NS; ++q) g[q] = 0.0;
  // stencil indices of the west, east, south and north swept values
  constexpr int W = GRP == 1 ? 3 : 2, E = GRP == 1 ? 4 : 1, S = GRP == 1 ? 2 : 3, N = GRP == 1 ? 1 : 4;
  const double bb = (wb + wd * (1.0 - rel) * x[0]) * irel;  // what -AI, -AD, -BS, -BN of the diagonal receive
  const double AIb = (X ? wa : -wd * x[W]) - bb, ADb = (X ? wc : -wd * x[E]) - bb;
  const double BSb = (X ? -wd * x[S] : wa) - bb, BNb = (X ? -wd * x[N] : wc) - bb;
  g[0] += wd * k.b * (1.0 - rel);
  if (X) { g[S] += -wd * k.BS; g[N] += -wd * k.BN; }
  else { g[W] += -wd * k.AI; g[E] += -wd * k.AD; }
  const double ui = AIb * k.dI, ud = ADb * k.dD, vs = BSb * k.dS, vn = BNb * k.dN;
  if constexpr (GRP == 0) {
    const double fi = G.met(M_FEXU, ii), fm = G.met(M_FEXU, ii - 1), fp = G.met(M_FEXP, ii);
    g[1] += fi * ud; g[0] += (1.0 - fi) * ud;
    g[0] += fm * ui; g[2] += (1.0 - fm) * ui;
    g[6] += fp * vn; g[5] += (1.0 - fp) * vn;
    g[8] += fp * vs; g[7] += (1.0 - fp) * vs;
    const double tb = -wd * k.dx * k.dy * G.Ri;
    g[10] += fp * tb; g[9] += (1.0 - fp) * tb;
    g[11] += wd * k.dy; g[12] += -wd * k.dy;
  } else if constexpr (GRP == 1) {
    const double fp = G.met(M_FEYP, jj), fj = G.met(M_FEYV, jj), fm = G.met(M_FEYV, jj - 1);
    g[6] += fp * ud; g[5] += (1.0 - fp) * ud;
    g[8] += fp * ui; g[7] += (1.0 - fp) * ui;
    g[1] += fj * vn; g[0] += (1.0 - fj) * vn;
    g[0] += fm * vs; g[2] += (1.0 - fm) * vs;
    const double tb = -wd * k.dx * k.dy * G.Riy;
    g[10] += fp * tb; g[9] += (1.0 - fp) * tb;
    g[11] += wd * k.dx; g[12] += -wd * k.dx;
  } else if constexpr (GRP == 2) {
    g[5] += ui; g[6] += ud; g[7] += vs; g[8] += vn;
    g[10] += wd * k.dy; g[9] += -wd * k.dy;
    g[12] += wd * k.dx; g[11] += -wd * k.dx;
  } else {
    g[5] += ud; g[6] += ui; g[7] += vn; g[8] += vs;
  }
}

// f(q, tap) for every tap of a group, both compile-time constants
template <int GRP, class F, int... Q>
__device__ __forceinline__ void each_tap_(F&& f, std::integer_sequence<int, Q...>) {
  auto one = [&](auto q) {
    constexpr Tap t = kStencil[GRP][decltype(q)::value];
    if constexpr (t.f != F_NONE) f(q, std::integral_constant<int, t.f>{}, t.di, t.dj);
  };
  (one(std::integral_constant<int, Q>{}), ...);
}
template <int GRP, class F>
__device__ __forceinline__ void each_tap(F&& f) {
  each_tap_<GRP>(f, std::make_integer_sequence<int, NS>{});
}

template <int GRP>
__device__ __forceinline__ void load_stencil(const Geo<double>& G, const SweepState& s, int ii, int jj,
                                             double (&x)[NS]) {
  each_tap<GRP>([&](auto q, auto f, int di, int dj) { x[q] = __ldg(s.f[f] + G.at(ii + di, jj + dj)); });
}

// One sweep reversed.  A CTA takes TL adjacent lines, GT threads per line for
// the solve, m rows per thread (n <= GT*m), and RP times as many for the rows
// and the scatter (their stencil loads and link arithmetic, one row after
// another, were most of a reversed sweep at one thread per chunk).  lam: the swept field's adjoint after the sweep,
// read and cleared here; every contribution to it before the sweep goes to
// adj.f[swept field], another buffer, zero on entry (null: dropped, p' before
// its first sweep).  aux_bar (u-x, v-x): the adjoint of au or av, read and
// cleared.  grad (T-x): d / d value of the side-a boundary rows, += mu of row
// 0 (the row is (0, 1, 0 | value), or the Neumann row with the value as flux).
template <int EQ, int TL, int GT, int RP, int M>
__global__ void __launch_bounds__(TL * GT * RP)
    adj_sweep_kernel(const Geo<double> G, const SweepState s, double* __restrict__ lam, double* aux_bar, AdjFields adj,
                     double* grad, int m_, int mp_) {
  constexpr int GRP = eq_group(EQ);
  constexpr bool X = (EQ & 1) != 0;
  constexpr int NT = TL * GT * RP;
  IXB_PDL_ENTRY();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  const int m = M > 0 ? M : m_, mp = M > 0 ? (M | 1) : mp_;
  const int n = s.n, npad = GT * m, arr = GT * mp, LS = (int)line_smem_elems(GT, mp);
  const int L0 = 1 + blockIdx.x * TL;
  auto slot = [&](int l, int r) { return l * LS + (r / m) * mp + r % m; };
  auto cell = [&](int L, int r) { return X ? G.at(r + 1, L) : G.at(L, r + 1); };
  // rows, transposed: a'_r = c_{r-1}, b'_r = b_r, c'_r = a_{r+1}; identity rows pad the line
  for (int idx = threadIdx.x; idx < TL * npad; idx += NT) {
    const int l = X ? idx / npad : idx % TL, r = X ? idx - l * npad : idx / TL, L = L0 + l;
    if (L > s.nfull) continue;
    const bool solved = L >= s.line_lo && L <= s.line_hi;
    double a = 0.0, b = 1.0, c = 0.0, d = 0.0;
    if (r < n) {
      const int g = cell(L, r);
      d = lam[g];
      lam[g] = 0.0;
      if (!solved) {  // the sweep copies this line
        if (d != 0.0 && adj.f[group_field(GRP)]) atomicAdd(adj.f[group_field(GRP)] + g, d);
        continue;
      }
      if (r == 0 || r == n - 1) {
        const BCEntry* t = r == 0 ? s.first : s.last;
        if (t && t[L].type == 2) {
          if (r == 0) { b = -1.0; c = 1.0; }
          else { a = -1.0; }
        }
      } else {
        const int ii = X ? r + 1 : L, jj = X ? L : r + 1;
        double x[NS];
        load_stencil<GRP>(G, s, ii, jj, x);
        const Links k = links<GRP>(G, x, s.flin ? s.flin[g] : 0.0, ii, jj);
        a = X ? k.AI : k.BS; b = k.b; c = X ? k.AD : k.BN;
      }
    }
    if (!solved) continue;
    sm[slot(l, r) + arr] = b;
    sm[slot(l, r) + 3 * arr] = d;
    if (r == 0 || r >= n) sm[slot(l, r)] = 0.0;
    if (r >= n - 1) sm[slot(l, r) + 2 * arr] = 0.0;
    if (r + 1 < n) sm[slot(l, r + 1)] = c;
    if (r >= 1 && r < n) sm[slot(l, r - 1) + 2 * arr] = a;
  }
  __syncthreads();
  if (threadIdx.x < TL * GT) {
    // (lines barriers of their own, TL > 1, when not all threads solve)
    const int l = threadIdx.x / GT, L = L0 + l;
    chunk_solve<double, GT, (RP > 1 ? 2 : TL), M>(sm + l * LS, m, mp, L >= s.line_lo && L <= s.line_hi);
  }
  __syncthreads();
  // scatter of the interior rows
  for (int idx = threadIdx.x; idx < TL * n; idx += NT) {
    const int l = X ? idx / n : idx % TL, r = X ? idx - l * n : idx / TL, L = L0 + l;
    if (L < s.line_lo || L > s.line_hi) continue;
    const double mu = sm[slot(l, r) + 3 * arr];
    if (r == 0 && grad) grad[L] += mu;
    if (r == 0 || r == n - 1) continue;
    const int g = cell(L, r), st = X ? 1 : G.LD;
    const int ii = X ? r + 1 : L, jj = X ? L : r + 1;
    const double wa = -mu * __ldg(s.x_out + g - st), wc = -mu * __ldg(s.x_out + g + st);
    double wb = -mu * __ldg(s.x_out + g);
    if (aux_bar) {
      wb += aux_bar[g] * G.rel_vel;
      aux_bar[g] = 0.0;
    }
    if (wa == 0.0 && wb == 0.0 && wc == 0.0 && mu == 0.0) continue;
    double x[NS], out[NS];
    load_stencil<GRP>(G, s, ii, jj, x);
    const Links k = links<GRP>(G, x, s.flin ? s.flin[g] : 0.0, ii, jj);
    row_back<GRP, X>(G, k, x, ii, jj, wa, wb, wc, mu, out);
    each_tap<GRP>([&](auto q, auto f, int di, int dj) {
      double* to = adj.f[f];
      if (out[q] != 0.0 && (f != F_PC || to)) atomicAdd(to + G.at(ii + di, jj + dj), out[q]);
    });
  }
}

// x-lines one per CTA; y-lines two adjacent ones while that gives a CTA per SM
// at most, else four (32-byte pieces of a row).  Three rows per thread of the
// solve up to 768 rows, longer chunks beyond.
template <int EQ>
cudaError_t adj_sweep_launch(const Geo<double>& G, const SweepState& s, double* lam, double* aux_bar,
                             const AdjFields& adj, double* grad, int nsm, cudaStream_t st) {
  constexpr bool X = (EQ & 1) != 0;
  auto go = [&](auto k, int tl, int g, int rp, int m) -> cudaError_t {
    const size_t smem = line_smem_elems(g, m | 1) * sizeof(double) * tl;
    if (smem > 48 * 1024) {  // beyond the default limit
      const cudaError_t e = allow_smem(k);
      if (e != cudaSuccess) return e;
    }
    return launch_pdl(true, k, (s.nfull + tl - 1) / tl, tl * g * rp, smem, st, G, s, lam, aux_bar, adj, grad, m, m | 1);
  };
  if constexpr (X) {
    if (s.n <= 192) return go(adj_sweep_kernel<EQ, 1, 64, 3, 3>, 1, 64, 3, 3);
    if (s.n <= 384) return go(adj_sweep_kernel<EQ, 1, 128, 3, 3>, 1, 128, 3, 3);
    if (s.n <= 768) return go(adj_sweep_kernel<EQ, 1, 256, 3, 3>, 1, 256, 3, 3);
  } else {
    const bool two = s.nfull <= 2 * nsm;
    if (s.n <= 192 && two) return go(adj_sweep_kernel<EQ, 2, 64, 3, 3>, 2, 64, 3, 3);
    if (s.n <= 192) return go(adj_sweep_kernel<EQ, 4, 64, 3, 3>, 4, 64, 3, 3);
    if (s.n <= 384 && two) return go(adj_sweep_kernel<EQ, 2, 128, 3, 3>, 2, 128, 3, 3);
    if (s.n <= 384) return go(adj_sweep_kernel<EQ, 4, 128, 1, 3>, 4, 128, 1, 3);
    if (s.n <= 1024) return go(adj_sweep_kernel<EQ, 4, 128, 1, 0>, 4, 128, 1, (s.n + 127) / 128);
  }
  return go(adj_sweep_kernel<EQ, 1, 256, 1, 0>, 1, 256, 1, std::max(3, (s.n + 255) / 256));
}

cudaError_t adj_sweep(const Geo<double>& G, const SweepState& s, double* lam, double* aux_bar, const AdjFields& adj,
                      double* grad, int nsm, cudaStream_t st) {
  switch (s.eq) {
    case EQ_UY: return adj_sweep_launch<EQ_UY>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_UX: return adj_sweep_launch<EQ_UX>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_VY: return adj_sweep_launch<EQ_VY>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_VX: return adj_sweep_launch<EQ_VX>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_PY: return adj_sweep_launch<EQ_PY>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_PX: return adj_sweep_launch<EQ_PX>(G, s, lam, aux_bar, adj, grad, nsm, st);
    case EQ_TY: return adj_sweep_launch<EQ_TY>(G, s, lam, aux_bar, adj, grad, nsm, st);
    default: return adj_sweep_launch<EQ_TX>(G, s, lam, aux_bar, adj, grad, nsm, st);
  }
}

// pressure and velocity correction (main.f90:931-962) out of place: u3, v3, p1
// from u2, v2, p0; entries the update leaves alone are copied
__global__ void correct_to_kernel(const Geo<double> G, const double* __restrict__ u2, const double* __restrict__ v2,
                                  const double* __restrict__ p0, const double* __restrict__ pc,
                                  const double* __restrict__ au, const double* __restrict__ av, double* __restrict__ u3,
                                  double* __restrict__ v3, double* __restrict__ p1) {
  IXB_PDL_ENTRY();
  const int ii = 1 + blockIdx.x * blockDim.x + threadIdx.x, jj = 1 + blockIdx.y;
  if (ii > G.mi + 1) return;
  const int c0 = G.at(ii, jj);
  const bool in = ii >= 2 && ii <= G.mi && jj >= 2 && jj <= G.nj;
  const double q = in ? pc[c0] : 0.0;
  p1[c0] = in ? p0[c0] + G.p_update * q : p0[c0];
  u3[c0] = in && ii <= G.mi - 1 ? u2[c0] + G.met(M_DYU, jj) * (q - pc[c0 + 1]) * fast_rcp(au[c0]) : u2[c0];
  v3[c0] = in && jj <= G.nj - 1 ? v2[c0] + G.met(M_DXV, ii) * (q - pc[c0 + G.LD]) * fast_rcp(av[c0]) : v2[c0];
}

__global__ void fill_kernel(double* f, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) f[i] = v;
}

// Adjoint of the velocity and pressure update (main.f90:931-962, correct_cell):
//   p += p_update p';  u(ii,jj) += dyu (p'(ii,jj) - p'(ii+1,jj)) / au;
//   v(ii,jj) += dxv (p'(ii,jj) - p'(ii,jj+1)) / av.
// u_bar, v_bar and p_bar pass through; p'_bar, au_bar and av_bar collect.
__global__ void adj_correct_kernel(const Geo<double> G, const double* __restrict__ pc, const double* __restrict__ au,
                                   const double* __restrict__ av, const double* __restrict__ ub,
                                   const double* __restrict__ vb, const double* __restrict__ pb, double* pcb,
                                   double* aub, double* avb) {
  IXB_PDL_ENTRY();
  const int ni = G.mi - 1;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ni * (G.nj - 1)) return;
  const int ii = 2 + idx % ni, jj = 2 + idx / ni;
  const int c0 = G.at(ii, jj);
  atomicAdd(pcb + c0, G.p_update * pb[c0]);
  if (ii <= G.mi - 1) {
    const double w = ub[c0];
    if (w != 0.0) {
      const int ce = G.at(ii + 1, jj);
      const double q = G.met(M_DYU, jj) / au[c0];
      atomicAdd(pcb + c0, w * q);
      atomicAdd(pcb + ce, -w * q);
      aub[c0] -= w * q * (pc[c0] - pc[ce]) / au[c0];
    }
  }
  if (jj <= G.nj - 1) {
    const double w = vb[c0];
    if (w != 0.0) {
      const int cn = G.at(ii, jj + 1);
      const double q = G.met(M_DXV, ii) / av[c0];
      atomicAdd(pcb + c0, w * q);
      atomicAdd(pcb + cn, -w * q);
      avb[c0] -= w * q * (pc[c0] - pc[cn]) / av[c0];
    }
  }
}

}  // namespace
}  // namespace ixb

using namespace ixb;

#define SCK(x)                   \
  do {                           \
    cudaError_t e_ = (x);        \
    if (e_ != cudaSuccess) {     \
      h->last_cuda = e_;         \
      return IXB_ECUDA;          \
    }                            \
  } while (0)
#define STRY(x)                  \
  do {                           \
    const int s_ = (x);          \
    if (s_ != IXB_OK) return s_; \
  } while (0)

namespace {

// The fields of one outer iteration, each written by the phase that produces
// it (S_U0 .. S_T0: the state before it; the state after it is the next
// iteration's S_U0 .. S_T0).
enum Snap { S_U0 = 0, S_V0, S_P0, S_T0, S_U1, S_U2, S_AU, S_V1, S_V2, S_AV, S_PC1, S_PC2, S_T1, S_COUNT };

struct SimpleAdjoint {
  ixb_handle* h;
  size_t fsz = 0;
  Geo<double> G{};
  double* pool = nullptr;   // everything below
  double* store = nullptr;  // C + 1 iterations x S_COUNT fields
  double* ckpt = nullptr;   // segments x (u, v, p, T)
  AdjFields adj{};
  double* other[F_COUNT] = {};  // second buffers of the swept fields' adjoints
  double* gd = nullptr;

  ~SimpleAdjoint() {
    if (pool) cudaFreeAsync(pool, h->stream);
    if (h && h->stream) cudaStreamSynchronize(h->stream);
  }

  int init(int C, int segments) {
    fsz = h->fsz;
    G = handle_geo(h);
    const size_t nadj = F_COUNT + 4, ngd = (size_t)h->nj + 2;
    const size_t total = ((size_t)(C + 1) * S_COUNT + (size_t)segments * 4 + nadj) * fsz + ngd;
    const cudaError_t e = scratch_alloc(SCRATCH_HANDLES, reinterpret_cast<void**>(&pool), total * sizeof(double), h->stream);
    if (e != cudaSuccess) {
      cudaGetLastError();
      pool = nullptr;
      return e == cudaErrorMemoryAllocation ? IXB_ENOMEM : IXB_ECUDA;
    }
    h->scratch_used = true;
    store = pool;
    ckpt = store + (size_t)(C + 1) * S_COUNT * fsz;
    double* a = ckpt + (size_t)segments * 4 * fsz;
    // adjoints and gradient start from zero; fields of the store from zero
    // too, but for au and av, whose unswept entries are 1e40 (main.f90:309-310)
    SCK(cudaMemsetAsync(a, 0, (nadj * fsz + ngd) * sizeof(double), h->stream));
    for (int k = 0; k < F_COUNT; ++k, a += fsz) adj.f[k] = a;
    for (int f : {F_U, F_V, F_T, F_PC}) { other[f] = a; a += fsz; }
    gd = a;
    SCK(cudaMemsetAsync(store, 0, (size_t)(C + 1) * S_COUNT * fsz * sizeof(double), h->stream));
    for (int it = 0; it < C; ++it)
      for (int f : {S_AU, S_AV}) {
        fill_kernel<<<148, 256, 0, h->stream>>>(slot(it, f), fsz, 1.e40);
        SCK(cudaGetLastError());
      }
    return IXB_OK;
  }
  double* slot(int it, int k) const { return store + ((size_t)it * S_COUNT + k) * fsz; }

  int copy(double* dst, const double* src) {
    SCK(cudaMemcpyAsync(dst, src, fsz * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    return IXB_OK;
  }
  int save(double* dst) {
    STRY(copy(dst, h->u[h->cu]));
    STRY(copy(dst + fsz, h->v[h->cv]));
    STRY(copy(dst + 2 * fsz, h->p));
    return copy(dst + 3 * fsz, h->T[h->cT]);
  }
  // the state of checkpoint k into the store
  int load(int k) {
    for (int q = 0; q < 4; ++q) STRY(copy(slot(0, S_U0 + q), ckpt + ((size_t)k * 4 + q) * fsz));
    return IXB_OK;
  }
  // count iterations from checkpoint k by the library's loop; it stops at
  // values that are not finite, the sweeps of the store carry them along
  int forward(int k, int count) {
    STRY(save(ckpt + (size_t)k * 4 * fsz));
    const int st = handle_single_passes(h, count);
    if (st != IXB_ENONFINITE) return st;
    STRY(load(k));
    for (int it = 0; it < count; ++it) STRY(iterate(it));
    STRY(copy(h->u[h->cu], slot(count, S_U0)));
    STRY(copy(h->v[h->cv], slot(count, S_V0)));
    STRY(copy(h->p, slot(count, S_P0)));
    return copy(h->T[h->cT], slot(count, S_T0));
  }

  // Iteration `it` of the store, sweep by sweep, one pass of each equation:
  // reads the state in its slots S_U0 .. S_T0, fills its other slots and the
  // next iteration's S_U0 .. S_T0.
  int iterate(int it) {
    auto S = [&](int k) { return slot(it, k); };
    auto sw = [&](int eq, const double* in, double* out, const double* u, const double* v, double* aux) -> int {
      SweepIO<double> io = handle_fixed_io(h, eq);
      io.in = in; io.out = out; io.aux = aux;
      io.u = u; io.v = v; io.T = S(S_T0); io.p = S(S_P0); io.pc = in;
      io.au = S(S_AU); io.av = S(S_AV);
      return handle_sweep_to(h, eq, io, true);
    };
    const double *u0 = S(S_U0), *v0 = S(S_V0);
    STRY(sw(EQ_UY, u0, S(S_U1), u0, v0, nullptr));
    STRY(sw(EQ_UX, S(S_U1), S(S_U2), S(S_U1), v0, S(S_AU)));
    STRY(sw(EQ_VY, v0, S(S_V1), S(S_U2), v0, nullptr));
    STRY(sw(EQ_VX, S(S_V1), S(S_V2), S(S_U2), S(S_V1), S(S_AV)));
    STRY(sw(EQ_PY, h->zero, S(S_PC1), S(S_U2), S(S_V2), nullptr));
    STRY(sw(EQ_PX, S(S_PC1), S(S_PC2), S(S_U2), S(S_V2), h->b_o));
    double *u3 = slot(it + 1, S_U0), *v3 = slot(it + 1, S_V0);
    const dim3 grid((h->mi + 1 + 127) / 128, h->nj + 1);
    SCK(launch_pdl(true, correct_to_kernel, grid, 128, 0, h->stream, G, S(S_U2), S(S_V2), S(S_P0), S(S_PC2), S(S_AU),
                   S(S_AV), u3, v3, slot(it + 1, S_P0)));
    STRY(sw(EQ_TY, S(S_T0), S(S_T1), u3, v3, nullptr));
    return sw(EQ_TX, S(S_T1), slot(it + 1, S_T0), u3, v3, nullptr);
  }

  // the boundary tables of variable var (0 u, 1 v, 2 T) for x- or y-lines
  void tables(SweepState& s, int var) {
    const bool x = (s.eq & 1) != 0;
    const BCEntry* base = h->bc + (size_t)var * 4 * h->bcstride;
    s.first = base + (size_t)(x ? 0 : 1) * h->bcstride;
    s.last = base + (size_t)(x ? 2 : 3) * h->bcstride;
  }
  SweepState state(int eq, int it) {
    SweepState s{};
    s.eq = eq;
    const SweepShape sh = sweep_shape(eq, h->mi, h->nj, 8, 1, 128);
    s.n = sh.n;
    s.line_lo = sh.line_lo;
    s.line_hi = sh.line_hi;
    s.nfull = sh.nfull;
    auto S = [&](int k) { return slot(it, k); };
    switch (eq) {
      case EQ_UY: case EQ_UX:
        s.f[F_U] = S(eq == EQ_UY ? S_U0 : S_U1); s.f[F_V] = S(S_V0); s.f[F_T] = S(S_T0); s.f[F_P] = S(S_P0);
        s.x_out = S(eq == EQ_UY ? S_U1 : S_U2); s.flin = h->flin[0];
        tables(s, 0);
        break;
      case EQ_VY: case EQ_VX:
        s.f[F_V] = S(eq == EQ_VY ? S_V0 : S_V1); s.f[F_U] = S(S_U2); s.f[F_T] = S(S_T0); s.f[F_P] = S(S_P0);
        s.x_out = S(eq == EQ_VY ? S_V1 : S_V2); s.flin = h->flin[1];
        tables(s, 1);
        break;
      case EQ_PY: case EQ_PX:
        s.f[F_PC] = eq == EQ_PY ? h->zero : S(S_PC1); s.f[F_AU] = S(S_AU); s.f[F_AV] = S(S_AV);
        s.f[F_U] = S(S_U2); s.f[F_V] = S(S_V2);
        s.x_out = S(eq == EQ_PY ? S_PC1 : S_PC2);
        break;
      default:
        s.f[F_T] = S(eq == EQ_TY ? S_T0 : S_T1); s.f[F_U] = slot(it + 1, S_U0); s.f[F_V] = slot(it + 1, S_V0);
        s.x_out = eq == EQ_TY ? S(S_T1) : slot(it + 1, S_T0); s.flin = h->flin[2];
        tables(s, 2);
        break;
    }
    return s;
  }

  // One sweep reversed: the adjoint of the swept field moves to its other
  // buffer (keep false: it is dropped); the other fields' adjoints collect.
  int sweep_back(int eq, int it, double* aux_bar, double* grad, bool keep = true) {
    const int f = eq == EQ_UY || eq == EQ_UX ? F_U : eq == EQ_VY || eq == EQ_VX ? F_V : eq == EQ_PY || eq == EQ_PX ? F_PC : F_T;
    double* lam = adj.f[f];
    std::swap(adj.f[f], other[f]);
    AdjFields a = adj;
    if (!keep) a.f[f] = nullptr;
    SCK(adj_sweep(G, state(eq, it), lam, aux_bar, a, grad, h->nsm, h->stream));
    return IXB_OK;
  }

  // One outer iteration reversed, from its stored phases.
  int iteration_back(int it) {
    STRY(sweep_back(EQ_TX, it, nullptr, gd));
    STRY(sweep_back(EQ_TY, it, nullptr, nullptr));
    const int ncell = (h->mi - 1) * (h->nj - 1);
    SCK(launch_pdl(true, adj_correct_kernel, (ncell + 255) / 256, 256, 0, h->stream, G, slot(it, S_PC2), slot(it, S_AU),
                   slot(it, S_AV), adj.f[F_U], adj.f[F_V], adj.f[F_P], adj.f[F_PC], adj.f[F_AU], adj.f[F_AV]));
    STRY(sweep_back(EQ_PX, it, nullptr, nullptr));
    STRY(sweep_back(EQ_PY, it, nullptr, nullptr, false));  // p' starts from the zero field
    STRY(sweep_back(EQ_VX, it, adj.f[F_AV], nullptr));     // av is written by the v-x sweep
    STRY(sweep_back(EQ_VY, it, nullptr, nullptr));
    STRY(sweep_back(EQ_UX, it, adj.f[F_AU], nullptr));     // au is written by the u-x sweep
    return sweep_back(EQ_UY, it, nullptr, nullptr);
  }

  // lambda_T = d Nu / d T: the Nusselt number is linear in T; its weights
  // are evaluated on unit fields with the shared host/device formula
  int objective(int j0, int j1) {
    const int mi = h->mi, nj = h->nj;
    std::vector<double> along(nj + 2, 0.0), across(mi + 2, 0.0);
    for (int j = 1; j <= nj + 1; ++j) along[j] = h->yp[j - 1];
    for (int i = 1; i <= mi + 1; ++i) across[i] = h->xp[i - 1];
    std::vector<double> w(fsz, 0.0);
    for (int k = j0; k <= j1 + 2; ++k)
      for (int l = 1; l <= 3; ++l)
        w[(size_t)(k - 1) * h->LD + (l - 1)] = nusselt_weight(along.data(), across.data(), mi + 1, j0, j1, k, l);
    SCK(cudaMemcpyAsync(adj.f[F_T], w.data(), fsz * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    SCK(cudaStreamSynchronize(h->stream));
    return IXB_OK;
  }
};

}  // namespace

extern "C" int ixb_adjoint_simple(ixb_handle* h, int K, int C, int j0, int j1, double* grad, double* nu0) {
  if (!h || K < 1 || C < 1) return IXB_EINVAL;
  STRY(handle_ready(h));
  if (h->prec != IXB_PREC_FP64) return IXB_EINVAL;  // the refined form's line solves are another map
  if (j0 < 1 || j1 < j0) return IXB_EINVAL;
  for (int k = j0; k <= j1; k += 2)
    if (k + 2 > h->nj + 1) return IXB_EINVAL;
  const int segments = (K + C - 1) / C;
  SimpleAdjoint A{h};
  STRY(A.init(std::min(C, K), segments));
  // forward, with a checkpoint at the start of every segment
  for (int sgm = 0; sgm < segments; ++sgm) STRY(A.forward(sgm, std::min(C, K - sgm * C)));
  double nu = 0.0;
  STRY(ixb_nusselt_x(h, j0, j1, &nu, nullptr));
  if (nu0) *nu0 = nu;
  if (!grad) return IXB_OK;
  STRY(A.objective(j0, j1));
  for (int sgm = segments - 1; sgm >= 0; --sgm) {
    STRY(A.load(sgm));
    const int count = std::min(C, K - sgm * C);
    for (int it = 0; it < count; ++it) STRY(A.iterate(it));
    for (int it = count - 1; it >= 0; --it) STRY(A.iteration_back(it));
  }
  std::vector<double> g((size_t)h->nj + 2);
  SCK(cudaMemcpyAsync(g.data(), A.gd, g.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  SCK(cudaStreamSynchronize(h->stream));
  for (int jj = 1; jj <= h->nj + 1; ++jj) grad[jj - 1] = g[jj];
  return IXB_OK;
}
