// ixb_passes_fast.cu -- many passes of the two energy sweeps (T-y then T-x,
// source/main.f90:985-1136) with the velocities held fixed, or of their
// transposes (ixb_adjoint_energy), in one cooperative launch.
//
// With u, v fixed the rows' matrices are the same in every pass and only
// their right-hand sides change, linearly with the field:
//   d_r = p0 + pc f(c) + pm f(c - s) + pp f(c + s)
// (s: across the line forward, along it transposed).  Every CTA keeps the
// lines it owns in both directions factored: each thread one chunk of three
// rows per direction, its right-hand side and elimination factors in
// registers, the reduced system's factors of every PCR step in shared memory.
// A sweep then loads nine values (transposed five) per thread, moves one word
// per thread and PCR step instead of three, divides nothing, and ends with a
// grid barrier.  The fields ping-pong through L2.
// Bound by latency: loads, PCR steps, the barrier (about 3.4 us per sweep at 256 x 256).
#include <cuda_runtime.h>

#include <algorithm>

#include "ixb_grid.cuh"
#include "ixb_internal.h"
#include "ixb_passes.h"
#include "ixb_sweep.cuh"

namespace ixb {
namespace {

constexpr int PM = 3;        // rows per thread
constexpr int PLEVELS = 8;   // PCR steps of up to 256 chunks
constexpr int PQ = 3 + 3 * PLEVELS + 2;  // factors in shared memory per thread and direction
constexpr int PMAXT = 448;

__global__ void energy_coef_kernel(const Geo<double> G, const SweepIO<double> io, double* __restrict__ coef,
                                   size_t fsz) {
  const int ni = G.mi - 1;  // ii = 2..mi, jj = 2..nj
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ni * (G.nj - 1)) return;
  const int ii = 2 + idx % ni, jj = 2 + idx / ni;
  const CellView<double, double> cell{G, io, ii, jj};
  const Row<double> rx = assemble_tx<true>(G, cell);  // a = AI, c = AD, b = diagonal
  const Row<double> ry = assemble_ty<true>(G, cell);  // a = BS, c = BN
  const int c0 = G.at(ii, jj);
  coef[C_AI * fsz + c0] = rx.a;
  coef[C_AD * fsz + c0] = rx.c;
  coef[C_BS * fsz + c0] = ry.a;
  coef[C_BN * fsz + c0] = ry.c;
  coef[C_DG * fsz + c0] = rx.b;
  coef[C_R0 * fsz + c0] = rx.d;  // io.in is the zero field: what does not depend on T
}

// One thread's chunk of one direction.
struct Chunk3 {
  double p0[PM], pc[PM], pm[PM], pp[PM];
  double inv, r, a2r, r0, c0r, a1, c1;
  int c0;       // field offset of its first row
  int k, pos;   // chunk of the line; TS apart in the exchange arrays
  int rows;     // rows inside the line (0: no chunk)
  int levels;
};

// Loads and factors the chunk (all threads call it: it holds barriers).
template <bool REV, bool X>
__device__ __forceinline__ void factor(Chunk3& h, const PassArgs& A, double* q, double* ex) {
  const Geo<double>& G = A.G;
  const int T = blockDim.x, t = threadIdx.x;
  const int n = X ? G.mi + 1 : G.nj + 1, lines = X ? G.nj - 1 : G.mi - 1;  // solved lines 2 .. lines+1
  const int per = X ? A.lx : A.ly, cn = X ? A.cx : A.cy;
  const int l = X ? t / cn : t % per, k = X ? t % cn : t / per, TS = X ? 1 : per;
  const int L = 2 + blockIdx.x * per + l, st = X ? 1 : G.LD;
  const bool mine = l < per && k < cn && L <= lines + 1;
  const BCEntry *bf = X ? A.first_x : A.first_y, *bl = X ? A.last_x : A.last_y;
  const double *AI = A.coef + C_AI * A.fsz, *AD = A.coef + C_AD * A.fsz, *BS = A.coef + C_BS * A.fsz,
               *BN = A.coef + C_BN * A.fsz, *DG = A.coef + C_DG * A.fsz, *R0 = A.coef + C_R0 * A.fsz;
  const double *lo = X ? AI : BS, *up = X ? AD : BN, *lo2 = X ? BS : AI, *up2 = X ? BN : AD;
  h.k = k;
  h.pos = t;
  h.rows = mine ? min(PM, n - k * PM) : 0;
  h.c0 = mine ? (X ? G.at(k * PM + 1, L) : G.at(L, k * PM + 1)) : 0;
  double a[PM], b[PM], c[PM];
#pragma unroll
  for (int i = 0; i < PM; ++i) {
    const int r = k * PM + i, g = h.c0 + i * st;
    a[i] = c[i] = 0.0;
    b[i] = 1.0;
    h.p0[i] = h.pc[i] = h.pm[i] = h.pp[i] = 0.0;
    if (i >= h.rows) continue;
    const bool edge = r == 0 || r == n - 1;
    if (edge) {
      const Row<double> e = r == 0 ? bc_first_row<double>(bf, L) : bc_last_row<double>(bl, L);
      a[i] = e.a; b[i] = e.b; c[i] = e.c;
      if (!REV) h.p0[i] = e.d;
    } else {
      a[i] = lo[g]; b[i] = DG[g]; c[i] = up[g];
      h.pc[i] = b[i] * A.keep;
      if (!REV) { h.p0[i] = R0[g]; h.pm[i] = -lo2[g]; h.pp[i] = -up2[g]; }
    }
    if (REV) {
      // transposed rows, and the rows of the other direction's lines that read
      // this cell through d (on a line that sweep copies nothing else arrives:
      // the sweep before it reads no boundary row's value)
      a[i] = r == 0 ? 0.0 : r == 1 ? bc_first_row<double>(bf, L).c : up[g - st];
      c[i] = r == n - 1 ? 0.0 : r == n - 2 ? bc_last_row<double>(bl, L).a : lo[g + st];
      if (r >= 2) h.pm[i] = -up[g - st];
      if (r <= n - 3) h.pp[i] = -lo[g + st];
    }
  }
  h.inv = fast_rcp(b[1]);
  h.a1 = a[1] * h.inv;
  h.c1 = c[1] * h.inv;
  h.r = fast_rcp(fma(-a[2], h.c1, b[2]));
  h.a2r = a[2] * h.r;
  double oA = -h.a2r * h.a1, oC = c[2] * h.r;
  h.r0 = fast_rcp(fma(-c[0], h.a1, b[0]));
  h.c0r = c[0] * h.r0;
  const double eA = a[0] * h.r0, eC = -h.c0r * h.c1;
  q += t;
  q[(PQ - 2) * T] = eA;
  q[(PQ - 1) * T] = eC;
  // the couplings of the steps of reduced_pcr: last rows by their own and the next chunk's first row, then among
  // themselves (all steps: whether one still counts depends on the right-hand sides, which change with every pass)
  double *xa = ex, *xc = ex + T;
  xa[t] = eA;
  xc[t] = eC;
  __syncthreads();
  const bool has = h.rows > 0;
  double hA = 0.0, hC = 0.0;
  if (has && k + 1 < cn) { hA = xa[t + TS]; hC = xc[t + TS]; }
  double r = fast_rcp(fma(-oC, hA, fma(-oA, eC, 1.0)));
  q[0] = oA * r; q[T] = oC * r; q[2 * T] = r;
  oA = -oA * eA * r;
  oC = -oC * hC * r;
  int lev = 0;
  for (int s = 1; s < cn; s <<= 1, ++lev) {
    double* pa = ex + ((lev & 1) ? 0 : 2) * T;  // the other pair: its readers are past a barrier
    pa[t] = oA;
    pa[T + t] = oC;
    __syncthreads();
    double lA = 0.0, lC = 0.0;
    hA = hC = 0.0;
    if (has && k >= s) { lA = pa[t - s * TS]; lC = pa[T + t - s * TS]; }
    if (has && k + s < cn) { hA = pa[t + s * TS]; hC = pa[T + t + s * TS]; }
    r = fast_rcp(fma(-oC, hA, fma(-oA, lC, 1.0)));
    double* ql = q + (3 + 3 * lev) * T;
    ql[0] = oA * r; ql[T] = oC * r; ql[2 * T] = r;
    oA = -oA * lA * r;
    oC = -oC * hC * r;
  }
  h.levels = lev;
  __syncthreads();
}

// One sweep of the CTA's lines of a direction: src -> dst.  Returns the first
// row's value (chunk 0's x_0).
template <bool REV, bool X>
__device__ __forceinline__ double pass_sweep(const Chunk3& h, const PassArgs& A, const double* q, double* ex,
                                             double* src, double* dst) {
  const int T = blockDim.x, t = threadIdx.x, LD = A.G.LD;
  const int n = X ? A.G.mi + 1 : A.G.nj + 1, cn = X ? A.cx : A.cy, TS = X ? 1 : A.ly;
  const int st = X ? 1 : LD, cr = REV ? st : (X ? LD : 1);
  const bool has = h.rows > 0;
  double d[PM];
  if (has) {
    double f[PM], fm[PM], fp[PM];
#pragma unroll
    for (int i = 0; i < PM; ++i) {
      // factors that are zero read a cell inside: across the line that of an
      // interior row, along it the line's first or last
      const int r = min(max(h.k * PM + i, REV ? 0 : 1), REV ? n - 1 : n - 2), g = h.c0 + (r - h.k * PM) * st;
      f[i] = __ldcg(src + g);
      fm[i] = __ldcg(src + (REV && r == 0 ? g : g - cr));
      fp[i] = __ldcg(src + (REV && r == n - 1 ? g : g + cr));
    }
#pragma unroll
    for (int i = 0; i < PM; ++i) d[i] = fma(h.pp[i], fp[i], fma(h.pm[i], fm[i], fma(h.pc[i], f[i], h.p0[i])));
  } else {
    d[0] = d[1] = d[2] = 0.0;
  }
  q += t;
  const double dn = d[1] * h.inv;
  double oD = fma(-h.a2r, dn, d[2] * h.r);
  const double eD = fma(-h.c0r, dn, d[0] * h.r0);
  ex[t] = eD;
  __syncthreads();
  {
    const double hD = has && h.k + 1 < cn ? ex[t + TS] : 0.0;
    oD = fma(-q[T], hD, fma(-q[0], eD, oD * q[2 * T]));
  }
  int buf = 1;
  for (int lev = 0, s = 1; lev < h.levels; ++lev, s <<= 1) {
    double* e = ex + buf * T;
    buf ^= 1;
    e[t] = oD;
    const double* ql = q + (3 + 3 * lev) * T;
    const double qa = ql[0], qc = ql[T], qr = ql[2 * T];
    __syncthreads();
    const double lD = has && h.k >= s ? e[t - s * TS] : 0.0;
    const double hD = has && h.k + s < cn ? e[t + s * TS] : 0.0;
    oD = fma(-qc, hD, fma(-qa, lD, oD * qr));
  }
  double* e = ex + buf * T;
  e[t] = oD;
  __syncthreads();
  const double xm = has && h.k > 0 ? e[t - TS] : 0.0;
  const double x0 = fma(-q[(PQ - 1) * T], oD, fma(-q[(PQ - 2) * T], xm, eD));
  const double x1 = fma(-h.c1, oD, fma(-h.a1, x0, dn));
  if (h.rows > 0) dst[h.c0] = x0;
  if (h.rows > 1) dst[h.c0 + st] = x1;
  if (h.rows > 2) dst[h.c0 + 2 * st] = oD;
  if (!REV && !X) {  // the T-x sweep copies these rows back (x-lines 1 and nj+1); no sweep reads them
    if (has && h.k == 0) src[h.c0] = x0;
    const int last = n - 1 - h.k * PM;
    if (has && last < PM) src[h.c0 + last * st] = last == 0 ? x0 : last == 1 ? x1 : oD;
  }
  return x0;
}

template <bool REV>
__global__ void __launch_bounds__(PMAXT, 1) energy_pass_kernel(const __grid_constant__ PassArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int T = blockDim.x;
  grid_arrive(A.waits);
  double* qx = reinterpret_cast<double*>(smem_raw);
  double* qy = qx + PQ * T;
  double* ex = qy + PQ * T;
  Chunk3 hx, hy;
  factor<REV, true>(hx, A, qx, ex);
  factor<REV, false>(hy, A, qy, ex);
  if (!grid_meet(A.waits)) return;
  unsigned target = 0;
  double grad = 0.0;
  for (int p = 0; p < A.passes; ++p) {
    if (REV) grad += pass_sweep<REV, true>(hx, A, qx, ex, A.f0, A.f1);
    else pass_sweep<REV, false>(hy, A, qy, ex, A.f0, A.f1);
    if (!grid_sync(A.waits, target)) return;
    if (REV) pass_sweep<REV, false>(hy, A, qy, ex, A.f1, A.f0);
    else pass_sweep<REV, true>(hx, A, qx, ex, A.f1, A.f0);
    if (!grid_sync(A.waits, target)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) A.waits.words->passes += A.passes;
  if (REV && hx.rows > 0 && hx.k == 0) A.grad[2 + blockIdx.x * A.lx + threadIdx.x / A.cx] += grad;
}

int threads_of(const PassArgs& a) { return (std::max(a.lx * a.cx, a.ly * a.cy) + 31) / 32 * 32; }
size_t smem_of(int threads) { return (size_t)(2 * PQ + 4) * threads * sizeof(double); }

}  // namespace

// One CTA per SM holds the lines of both directions: up to 256 chunks per
// line and 448 threads (the factors of more do not fit in shared memory),
// 445 x 445 on 148 SMs.  Per pass against two launches: 256 x 256 6.8 against
// 9.8 us forward and 6.7 against 10.4 transposed, 64 x 64 5.6 against 7.6 and
// 5.2 against 8.4; factoring costs about a pass, so the forward run takes it
// from four passes on.
bool energy_passes_fit(int mi, int nj, int nsm, PassArgs* a) {
  PassArgs p{};
  p.cx = (mi + 1 + PM - 1) / PM;
  p.cy = (nj + 1 + PM - 1) / PM;
  p.lx = (nj - 1 + nsm - 1) / nsm;
  p.ly = (mi - 1 + nsm - 1) / nsm;
  if (p.cx > (1 << PLEVELS) || p.cy > (1 << PLEVELS) || threads_of(p) > PMAXT) return false;
  p.grid = std::max((nj - 1 + p.lx - 1) / p.lx, (mi - 1 + p.ly - 1) / p.ly);
  if (a) { a->cx = p.cx; a->cy = p.cy; a->lx = p.lx; a->ly = p.ly; a->grid = p.grid; }
  return true;
}

cudaError_t energy_coef_launch(const Geo<double>& G, const SweepIO<double>& io, double* coef, size_t fsz,
                               cudaStream_t st) {
  const int n = (G.mi - 1) * (G.nj - 1);
  energy_coef_kernel<<<(n + 255) / 256, 256, 0, st>>>(G, io, coef, fsz);
  return cudaGetLastError();
}

// A launch runs up to kPassesPerLaunch passes (a bounded kernel time).
cudaError_t energy_passes_launch(bool reverse, const PassArgs& a, int expire_from, cudaStream_t st) {
  const int T = threads_of(a);
  const size_t smem = smem_of(T);
  auto k = reverse ? energy_pass_kernel<true> : energy_pass_kernel<false>;
  cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  PassArgs q = a;
  int launch = 0;
  for (int left = a.passes; left > 0; left -= q.passes, ++launch) {
    q.passes = std::min(left, kPassesPerLaunch);
    q.waits.expire = launch >= expire_from ? a.waits.expire : GRID_EXPIRE_NONE;
    if ((e = cudaMemsetAsync(q.waits.words, 0, 2 * sizeof(unsigned), st)) != cudaSuccess) return e;
    void* params[] = {&q};
    if ((e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(q.grid), dim3(T), params, smem, st)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ixb
