// ixb_loop.cuh -- the SIMPLE loop as one resident kernel: every phase of the
// outer iteration (source/main.f90:395-1217), the inner loops and their exit
// tests, with a grid barrier between phases.
//
// A sweep is a few microseconds of dependent latencies on every SM (stencil
// loads, row arithmetic, line solve, write-back), so what separates two
// sweeps weighs as much as a third of one: as graph nodes it was a kernel
// boundary, the norm's last-CTA reduction and the loops' conditional nodes.
// Here one CTA per SM stays for up to max_outer outer passes; phases are
// separated by a grid barrier, and after a barrier every warp sums the norm's
// per-CTA partials in the same order and takes the reference's exit test
// itself.
//
// Within a phase the stencil loads were what took longest (rows assembled
// one after another, each waiting for its loads and the metrics').  So:
//  * a thread assembles a column of up to three cells (fixed ii, jj .. jj+2) in
//    both directions: neighbouring cells share its loads (28 field loads per
//    three cells instead of 42), which go out a row ahead of the arithmetic;
//    in an x-sweep the column crosses the CTA's lines and a warp reads 32
//    consecutive ii;
//  * the metrics and the boundary rows of the CTA's lines stay in shared
//    memory for the whole launch;
//  * the u residual of an outer pass (main.f90:1169-1199) needs what the next
//    pass's first u-y sweep loads, so it is taken there; that sweep writes
//    only the other buffer, so nothing is lost when the outer test then ends
//    the loop.
// The arithmetic is that of the fused sweep kernels.
//
// Measured per outer iteration of a developed field, graph of fused sweeps ->
// this kernel (binary64 / refined): 64x64 53.1 / 53.9 -> 42.9 / 43.8 us, 161x97
// 58.0 / 57.9 -> 47.0 / 48.7 us, 256x256 67.5 / 68.0 -> 55.2 / 57.4 us, 701x301
// 83.3 / 87.8 -> 82.2 / 84.6 us (and with several passes per inner loop the
// graph pays a conditional body each, this kernel nothing).
// Bound by latencies: at 701x301 a warp's issue waits for barriers (the steps
// of the reduced systems, the grid barrier) 9.8 cycles of some 15, for loads
// 2.7, with 30 % of the issue slots and 0.6 % of the DRAM rate in use.
#pragma once
#include "ixb_grid.cuh"
#include "ixb_loop.h"
#include "ixb_sweep.cuh"

namespace ixb {

// Barrier `id` (1..15) of n threads (whole warps) that tells whether q holds
// in any of them; a single warp needs no hardware barrier.
__device__ __forceinline__ bool group_or(int id, int n, bool q) {
  if (n == 32) {
    const bool r = __any_sync(0xffffffffu, q);
    __syncwarp();
    return r;
  }
  return barrier_or(id, n, q);
}

// Sum of one norm's partials, the same bits in every thread: each warp adds
// the CTAs' partials in the same order.
__device__ __forceinline__ double sum_partials(const double* p) {
  const int lane = threadIdx.x & 31, n = gridDim.x;
  double s = 0.0;
  for (int i0 = 0; i0 < n; i0 += 160) {  // five loads in flight
    double v[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int i = i0 + q * 32 + lane;
      v[q] = i < n ? reinterpret_cast<const Live*>(p)[i].v : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) s += v[q];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// this CTA's share of two sums of squares -> partials
__device__ __forceinline__ void post_partials(double a, double* pa, double b, double* pb) {
  __shared__ double red[2][kLoopThreads / 32];
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { red[0][w] = a; red[1][w] = b; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    a = lane < nw ? red[0][lane] : 0.0;
    b = lane < nw ? red[1][lane] : 0.0;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
      pa[blockIdx.x] = a;
      if (pb) pb[blockIdx.x] = b;
    }
  }
}

// ---------------------------------------------------------------------------
// shared memory of a CTA, filled once per launch
// ---------------------------------------------------------------------------
// metrics the fast rows read, by direction (dxv = dxp and dyu = dyp)
enum { SX_DXP = 0, SX_DXU, SX_FEXP, SX_FEXU, SX_GRDXP, SX_GRDXU, SX_HRDXU, SX_PEXP, SX_PEXU, SX_PHXU, SX_COUNT };
enum { SY_DYP = 0, SY_DYV, SY_FEYP, SY_FEYV, SY_GRDYV, SY_GRDYP, SY_HRDYV, SY_PEYV, SY_PEYP, SY_PHYV, SY_COUNT };

__host__ __device__ constexpr int sx_of(int m) {
  return m == M_DXP || m == M_DXV ? SX_DXP : m == M_DXU ? SX_DXU : m == M_FEXP ? SX_FEXP : m == M_FEXU ? SX_FEXU
         : m == M_GRDXP ? SX_GRDXP : m == M_GRDXU ? SX_GRDXU : m == M_HRDXU ? SX_HRDXU : m == M_PEXP ? SX_PEXP
         : m == M_PEXU ? SX_PEXU : SX_PHXU;
}
__host__ __device__ constexpr int sy_of(int m) {
  return m == M_DYP || m == M_DYU ? SY_DYP : m == M_DYV ? SY_DYV : m == M_FEYP ? SY_FEYP : m == M_FEYV ? SY_FEYV
         : m == M_GRDYV ? SY_GRDYV : m == M_GRDYP ? SY_GRDYP : m == M_HRDYV ? SY_HRDYV : m == M_PEYV ? SY_PEYV
         : m == M_PEYP ? SY_PEYP : SY_PHYV;
}

// one boundary row: type 2 (neum) or not, and its value
struct BcS { double val; int neum; };

// Everything the phases share, at the start of the CTA's dynamic shared
// memory.  The phases are functions of their own (not inlined): a register
// allocation over all of them at once spilled ten times as much as theirs.
struct LoopCtx {
  LoopArgs A;
  double* mx;  // SX_COUNT arrays of sx
  double* my;  // SY_COUNT arrays of sy
  int sx, sy;
  // this CTA's x-lines (first, count) of fields with nj+1 lines and of v (nj)
  int x0, xn, x0v, xnv;
  BcS bcx[3][2][kLoopM];  // [variable][first, last][line of the CTA]
  BcS bcy[3][2][kLoopLinesY];
  unsigned char* lines;   // staged lines / reduced systems
};
__device__ __forceinline__ LoopCtx& loop_ctx() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return *reinterpret_cast<LoopCtx*>(smem_raw);
}
// index range of a metric array: 0 .. n+3 (columns reach two cells past a
// line's last row; the entries beyond the mesh are zeros)
__host__ __device__ constexpr int loop_pitch(int n) { return (n + 5) | 1; }
__host__ __device__ constexpr size_t up16(size_t n) { return (n + 15) & ~(size_t)15; }
__host__ __device__ constexpr size_t loop_fixed_bytes(int mi, int nj) {
  return up16(sizeof(LoopCtx)) +
         up16(((size_t)SX_COUNT * loop_pitch(mi) + (size_t)SY_COUNT * loop_pitch(nj)) * sizeof(double));
}

// fields of one sweep (SweepIO's, without the norms)
struct LoopIO {
  const double *in, *u, *v, *T, *p, *au, *av, *ant, *fcon, *flin;
  double *out, *aux;
  const double* prev;
  int var;         // boundary tables: 0 u, 1 v, 2 T, -1 p'
  bool zero_in;    // p' before its first sweep: zero, not read
};

__device__ __forceinline__ double live(const double* p, int i) { return reinterpret_cast<const Live*>(p)[i].v; }

// ---------------------------------------------------------------------------
// columns of cells
// ---------------------------------------------------------------------------
// values of one field around the current cell of a column, [di + 1][dj + 1],
// and the next row's, already on their way
struct Window { double f[3][3], nx[3]; };

// What a column's current cell reads, and its place.  Entries an equation
// does not use are never read, and their loads are dropped.
struct Column {
  Window in, u, v, T, p, au, av;
  double ant, nant;
  int ii, jj, o;  // the cell and its offset
};

// the view of a column's current cell (see CellView)
template <int EQ>
struct ColumnView {
  const Column& c;
  const LoopIO& io;
  int LD;
  __device__ __forceinline__ double in(int di, int dj) const { return c.in.f[di + 1][dj + 1]; }
  __device__ __forceinline__ double u(int di, int dj) const { return c.u.f[di + 1][dj + 1]; }
  __device__ __forceinline__ double v(int di, int dj) const { return c.v.f[di + 1][dj + 1]; }
  // u rows read T only with a buoyancy along x (no mode of the reference has one)
  __device__ __forceinline__ double T(int di, int dj) const {
    if constexpr (EQ == EQ_UY || EQ == EQ_UX) return live(io.T, c.o + dj * LD + di);
    else return c.T.f[di + 1][dj + 1];
  }
  __device__ __forceinline__ double p(int di, int dj) const { return c.p.f[di + 1][dj + 1]; }
  __device__ __forceinline__ double au(int di, int dj) const { return c.au.f[di + 1][dj + 1]; }
  __device__ __forceinline__ double av(int di, int dj) const { return c.av.f[di + 1][dj + 1]; }
  __device__ __forceinline__ double u_ant() const { return c.ant; }
  __device__ __forceinline__ double v_ant() const { return c.ant; }
  __device__ __forceinline__ double T_ant() const { return c.ant; }
  __device__ __forceinline__ double fcon() const { return io.fcon ? __ldg(io.fcon + c.o) : 0.0; }
  __device__ __forceinline__ double flin() const { return io.flin ? __ldg(io.flin + c.o) : 0.0; }
  __device__ __forceinline__ double mx(int which, int d) const {
    const LoopCtx& X = loop_ctx();
    return X.mx[sx_of(which) * X.sx + c.ii + d];
  }
  __device__ __forceinline__ double my(int which, int d) const {
    const LoopCtx& X = loop_ctx();
    return X.my[sy_of(which) * X.sy + c.jj + d];
  }
};

// Fields of sweep EQ: y-sweeps read buffer 0 and write buffer 1, x-sweeps the
// other way, so every pass ends in buffer 0.  first (p'): the pass starts
// from p' = 0.
template <int EQ>
__device__ __forceinline__ LoopIO loop_io(const LoopArgs& A, bool first) {
  constexpr int VAR = EQ == EQ_UY || EQ == EQ_UX ? 0 : EQ == EQ_VY || EQ == EQ_VX ? 1 : EQ == EQ_PY || EQ == EQ_PX ? -1 : 2;
  constexpr int X = EqIsX<EQ>::value ? 1 : 0;
  LoopIO io{};
  io.var = VAR;
  double* const* f = VAR == 0 ? A.u : VAR == 1 ? A.v : VAR == 2 ? A.T : A.pc;
  io.in = f[X];
  io.out = f[1 - X];
  io.u = A.u[0]; io.v = A.v[0]; io.T = A.T[0]; io.p = A.p; io.au = A.au; io.av = A.av;
  if (VAR >= 0) { io.fcon = A.fcon[VAR < 0 ? 0 : VAR]; io.flin = A.flin[VAR < 0 ? 0 : VAR]; }
  io.ant = VAR == 0 ? A.u_ant : VAR == 1 ? A.v_ant : A.T_ant;
  io.aux = EQ == EQ_UX ? A.au : EQ == EQ_VX ? A.av : A.b_o;
  io.prev = EQ == EQ_VX ? A.v[0] : EQ == EQ_TX ? A.T[0] : EQ == EQ_PX && !first ? A.pc[0] : nullptr;
  io.zero_in = EQ == EQ_PY && first;
  return io;
}

// Walk along a column.  Loads run a row ahead of the arithmetic (few
// registers hold them, and the three columns' sectors are asked for together:
// loading a whole column before its neighbours measured 88 against 84 us per
// outer iteration at 701x301, the neighbours' sectors being evicted from L1
// in between).  Rows are clamped to 1..jmax.
template <int EQ>
struct ColumnWalk {
  static constexpr bool P = EQ == EQ_PY || EQ == EQ_PX, T = EQ == EQ_TY || EQ == EQ_TX, U = EQ == EQ_UY || EQ == EQ_UX,
                        V = EQ == EQ_VY || EQ == EQ_VX;
  const LoopIO& io;
  int LD, jmax;
  __device__ __forceinline__ int row(const Column& c, int jj) const {
    return (min(max(jj, 1), jmax) - 1) * LD + c.ii - 1;
  }
  __device__ __forceinline__ void three(double (&x)[3], const double* f, int o) const {
#pragma unroll
    for (int d = 0; d < 3; ++d) x[d] = live(f, o + d - 1);
  }
  __device__ __forceinline__ void put(Window& w, int dj, const double* f, int o) const {
#pragma unroll
    for (int d = 0; d < 3; ++d) w.f[d][dj + 1] = live(f, o + d - 1);
  }
  // first cell (ii, jj)
  __device__ __forceinline__ void start(Column& c, int ii, int jj) const {
    c.ii = ii;
    c.jj = jj;
    const int o[3] = {row(c, jj - 1), row(c, jj), row(c, jj + 1)};
    c.o = o[1];
    if (P && io.zero_in) {
#pragma unroll
      for (int d = 0; d < 3; ++d) c.in.f[d][0] = c.in.f[d][1] = c.in.f[d][2] = c.in.nx[d] = 0.0;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      if (!(P && io.zero_in)) put(c.in, r - 1, io.in, o[r]);
      if (!U) put(c.u, r - 1, io.u, o[r]);
      if (!V) put(c.v, r - 1, io.v, o[r]);
      if (P) { put(c.au, r - 1, io.au, o[r]); put(c.av, r - 1, io.av, o[r]); }
      if (U || V) put(c.p, r - 1, io.p, o[r]);
      if (V) put(c.T, r - 1, io.T, o[r]);
    }
    if (!P) c.ant = __ldg(io.ant + o[1]);
  }
  // the row a field is read at next: jj+2 where the cell reads its north row, else jj+1
  __device__ __forceinline__ void fetch(Column& c) const {
    const int o1 = row(c, c.jj + 1), o2 = row(c, c.jj + 2);
    if (!(P && io.zero_in)) {
      c.in.nx[0] = live(io.in, o1 - 1);
      c.in.nx[1] = live(io.in, o2);
      c.in.nx[2] = live(io.in, o1 + 1);
    }
    if (V) three(c.u.nx, io.u, o2);
    else if (!U) three(c.u.nx, io.u, o1);
    if (!V) three(c.v.nx, io.v, o1);
    if (P) { three(c.au.nx, io.au, o1); three(c.av.nx, io.av, o1); }
    if (U || V) three(c.p.nx, io.p, V ? o2 : o1);
    if (V) three(c.T.nx, io.T, o2);
    if (!P) c.nant = __ldg(io.ant + o1);
  }
  __device__ __forceinline__ void shift(double (&f)[3], double nx, bool north) const {
    f[0] = f[1];
    if (north) { f[1] = f[2]; f[2] = nx; }
    else f[1] = nx;
  }
  __device__ __forceinline__ void advance(Column& c) const {
    shift(c.in.f[1], c.in.nx[1], true);
    c.in.f[0][1] = c.in.nx[0];
    c.in.f[2][1] = c.in.nx[2];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!U) shift(c.u.f[d], c.u.nx[d], V);
      if (!V) shift(c.v.f[d], c.v.nx[d], false);
      if (V) shift(c.T.f[d], c.T.nx[d], true);
      if (U || V) shift(c.p.f[d], c.p.nx[d], V);
      if (P) { shift(c.au.f[d], c.au.nx[d], false); shift(c.av.f[d], c.av.nx[d], false); }
    }
    if (!P) c.ant = c.nant;
    ++c.jj;
    c.o = row(c, c.jj);
  }
};

// boundary row (see bc_first_row / bc_last_row); p' rows are Dirichlet 0
__device__ __forceinline__ Row<double> loop_bc_row(const BcS& e, bool first) {
  if (e.neum) return first ? Row<double>{0.0, -1.0, 1.0, e.val} : Row<double>{-1.0, 1.0, 0.0, e.val};
  return Row<double>{0.0, 1.0, 0.0, e.val};
}

// The phases keep their code small: the loop runs through all of it once per
// outer pass on every SM, and code beyond the instruction cache is fetched
// again each time (the same sweeps with their three cells unrolled were 240 KB
// and took 113 us per outer iteration at 701x301, against 84 us).  So the
// cells of a column are a loop, only the assembly exists per equation, and the
// line solves and write-backs are shared by all sweeps of a direction.

// x-sweep: thread t assembles column ii = t + 1 of the CTA's lines into shared
// memory (line q: rows a | b | c | d in chunk order).  Returns this thread's
// share of the sum of squares of b_o (p'-x).
template <int EQ, int SOLVER>
__device__ __noinline__ double assemble_x(const bool first) {
  using ST = SweepTypes<SOLVER, EQ>;
  using S = typename ST::S;
  const LoopCtx& sh = loop_ctx();
  const LoopArgs& A = sh.A;
  const Geo<double>& G_ = A.G;
  const LoopIO io = loop_io<EQ>(A, first);
  const int n = EQ == EQ_UX ? G_.mi : G_.mi + 1, lo = 2, hi = EQ == EQ_VX ? G_.nj - 1 : G_.nj;
  const int arr = A.s.gx * kLoopM;
  const int L0 = EQ == EQ_VX ? sh.x0v : sh.x0, nl = EQ == EQ_VX ? sh.xnv : sh.xn;
  const int t = threadIdx.x;
  S* ln = reinterpret_cast<S*>(sh.lines) + t;
  double acc_bo = 0.0;
  if (t < n) {
    const bool edge = t == 0 || t == n - 1;
    Column c;
    const ColumnWalk<EQ> walk{io, G_.LD, min(hi + 1, L0 + nl)};
    walk.start(c, min(max(t + 1, 2), n - 1), L0);
    const ColumnView<EQ> cell{c, io, G_.LD};
#pragma unroll 1
    for (int q = 0; q < nl; ++q) {
      walk.fetch(c);
      double aux = 0.0;
      Row<double> row = assemble_cell<EQ, true>(G_, cell, aux);
      if (edge)
        row = io.var < 0 ? Row<double>{0.0, 1.0, 0.0, 0.0} : loop_bc_row(sh.bcx[io.var][t == 0 ? 0 : 1][q], t == 0);
      if constexpr (ST::DC) {
        // boundary columns are assembled at their neighbour: their own value sits beside it
        const double x0 = t == 0 ? cell.in(-1, 0) : t == n - 1 ? cell.in(1, 0) : cell.in(0, 0);
        const double xm = t == n - 1 ? cell.in(0, 0) : cell.in(-1, 0), xp = t == 0 ? cell.in(0, 0) : cell.in(1, 0);
        row_defect(row, xm, x0, xp);
      }
      if constexpr (ST::MIX) row_scale(row);
      ln[0] = S(row.a); ln[arr] = S(row.b); ln[2 * arr] = S(row.c); ln[3 * arr] = S(row.d);
      ln += 4 * arr;
      if constexpr (EqHasAux<EQ>::value) {
        const int L = L0 + q;
        if (!edge && L >= lo && L <= hi) {
          io.aux[(L - 1) * G_.LD + t] = aux;
          if (EQ == EQ_PX) acc_bo += aux * aux;
        }
      }
      walk.advance(c);
    }
  }
  // identity rows pad every line to gx chunks
  for (int r = n + t; r < arr; r += blockDim.x)
    for (int q = 0; q < nl; ++q) {
      S* p = reinterpret_cast<S*>(sh.lines) + (size_t)q * 4 * arr + r;
      p[0] = S(0); p[arr] = S(1); p[2 * arr] = S(0); p[3 * arr] = S(0);
    }
  return acc_bo;
}

// Line solve and write-back of an x-sweep: group gid of gx threads (this
// thread's chunk: k) solves line L0 + gid of the staged ones if it lies in
// 2..hi, then thread t writes column t of the nl lines.  old: the swept field
// (a defect correction adds to it; unsolved lines keep it), dc: the former.
// Returns this thread's share of the sum of squares of new - prev.
template <class S>
__device__ __noinline__ double solve_x(const int gid, const int k, const int n, const int hi, const int L0, const int nl,
                                       const double* old, const bool dc, double* out, const double* prev,
                                       const bool norm) {
  constexpr int M = kLoopM;
  const LoopCtx& sh = loop_ctx();
  const int gx = sh.A.s.gx, arr = gx * M, LD = sh.A.G.LD, t = threadIdx.x;
  S* lines = reinterpret_cast<S*>(sh.lines);
  double o[M], p[M];  // read early: the solve hides their latency
#pragma unroll
  for (int q = 0; q < M; ++q) {
    const int L = L0 + q, g = (L - 1) * LD + t;
    const bool in = q < nl && t < n;
    o[q] = in && (dc || L < 2 || L > hi) ? live(old, g) : 0.0;
    p[q] = in && prev ? live(prev, g) : 0.0;
  }
  __syncthreads();
  if (gid < nl && L0 + gid >= 2 && L0 + gid <= hi) {
    S* ln = lines + (size_t)gid * 4 * arr;
    auto sync = [&](bool q) { return group_or(1 + gid, gx, q); };
    Chunk<S, M> ch;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const int r = k * M + i;  // M is odd: the threads of a warp hit different banks
      ch.a[i] = ln[r]; ch.b[i] = ln[arr + r]; ch.c[i] = ln[2 * arr + r]; ch.d[i] = ln[3 * arr + r];
    }
    ch.eliminate();
    sync(false);  // the rows are in registers: their memory serves the reduced system
    S x0, xl;
    reduced_pcr<S, sizeof(S) == 8>(ln, gx, 1, gx, k, k, true, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD, x0, xl, sync);
    ch.substitute(x0, xl);
    sync(false);
#pragma unroll
    for (int i = 0; i < M; ++i) ln[k * M + i] = ch.d[i];
  }
  __syncthreads();
  double acc = 0.0;
  if (t < n) {
#pragma unroll
    for (int q = 0; q < M; ++q) {
      const int L = L0 + q;
      if (q >= nl) break;
      double x = o[q];
      if (L >= 2 && L <= hi) {
        x += double(lines[(size_t)q * 4 * arr + t]);
        if (norm && t >= 1 && t <= n - 2) { const double dv = x - p[q]; acc += dv * dv; }
      }
      out[(L - 1) * LD + t] = x;
    }
  }
  __syncthreads();  // the next sweep's assembly reuses the lines' memory
  return acc;
}

template <int EQ, int SOLVER>
__device__ __forceinline__ double2 loop_x(const bool first, const int gid, const int k) {
  using ST = SweepTypes<SOLVER, EQ>;
  const double bo = assemble_x<EQ, SOLVER>(first);
  const LoopCtx& sh = loop_ctx();
  const LoopArgs& A = sh.A;
  const LoopIO io = loop_io<EQ>(A, first);
  const double acc = solve_x<typename ST::S>(
      gid, k, EQ == EQ_UX ? A.G.mi : A.G.mi + 1, EQ == EQ_VX ? A.G.nj - 1 : A.G.nj, EQ == EQ_VX ? sh.x0v : sh.x0,
      EQ == EQ_VX ? sh.xnv : sh.xn, io.in, ST::DC, io.out, io.prev, EQ != EQ_UX);
  return double2{acc, bo};
}

// y-sweep: thread t assembles the three rows of chunk k = t / y_lines of line
// 1 + blockIdx.x * y_lines + l, l = t % y_lines, into its own slots of shared
// memory (row it: a, b, c, d at (4*it + 0..3) * used + t).  res (u-y): also the u
// residual of the fields before the sweep; returns this thread's share of its
// sum of squares.
template <int EQ, int SOLVER>
__device__ __noinline__ double assemble_y(const bool first, const int l, const int k, const int used, const bool res) {
  using ST = SweepTypes<SOLVER, EQ>;
  using S = typename ST::S;
  constexpr int M = kLoopM;
  const LoopCtx& sh = loop_ctx();
  const LoopArgs& A = sh.A;
  const Geo<double>& G_ = A.G;
  const LoopIO io = loop_io<EQ>(A, first);
  const int n = EQ == EQ_VY ? G_.nj : G_.nj + 1, hi = EQ == EQ_UY ? G_.mi - 1 : G_.mi;
  const int L = 1 + blockIdx.x * A.s.y_lines + l;
  S* slot = reinterpret_cast<S*>(sh.lines) + threadIdx.x;
  double acc_res = 0.0;
  if (!(k < A.s.gy && k * M < n && L >= 2 && L <= hi)) {
#pragma unroll 1
    for (int it = 0; it < M; ++it) {
      slot[0] = S(0); slot[used] = S(1); slot[2 * used] = S(0); slot[3 * used] = S(0);
      slot += 4 * used;
    }
    return 0.0;
  }
  Column c;
  const ColumnWalk<EQ> walk{io, G_.LD, n};
  walk.start(c, L, k * M + 1);
  const ColumnView<EQ> cell{c, io, G_.LD};
#pragma unroll 1
  for (int it = 0; it < M; ++it) {
    const int r = k * M + it;
    walk.fetch(c);
    double aux;
    Row<double> row = assemble_cell<EQ, true>(G_, cell, aux);
    if (r == 0 || r >= n - 1)
      row = r >= n ? Row<double>{0.0, 1.0, 0.0, 0.0}
            : io.var < 0 ? Row<double>{0.0, 1.0, 0.0, 0.0}
                         : loop_bc_row(sh.bcy[io.var][r == 0 ? 0 : 1][l], r == 0);
    if constexpr (ST::DC || EQ == EQ_UY) {
      Row<double> def = row;
      row_defect(def, cell.in(0, -1), cell.in(0, 0), cell.in(0, 1));
      if constexpr (EQ == EQ_UY) {
        // u residual: the defect of the row (its relaxation terms cancel at the values it holds)
        if (res && r >= 1 && r <= n - 2) {
          A.resu[r * G_.LD + (L - 1)] = def.d;
          acc_res += def.d * def.d;
        }
      }
      if (ST::DC && r < n) row = def;
    }
    if constexpr (ST::MIX) row_scale(row);
    slot[0] = S(row.a); slot[used] = S(row.b); slot[2 * used] = S(row.c); slot[3 * used] = S(row.d);
    slot += 4 * used;
    walk.advance(c);
  }
  return acc_res;
}

// Line solve and write-back of a y-sweep (lines of n rows, 2..hi solved,
// hi + 1 in the field); old, dc, out as in solve_x.
template <class S>
__device__ __noinline__ void solve_y(const int l, const int k, const int used, const int n, const int hi,
                                     const double* old, const bool dc, double* out) {
  constexpr int M = kLoopM;
  const LoopCtx& sh = loop_ctx();
  const int gy = sh.A.s.gy, TL = sh.A.s.y_lines, LD = sh.A.G.LD;
  const int L = 1 + blockIdx.x * TL + l;
  const bool active = k < gy && L >= 2 && L <= hi, mine = k < gy && k * M < n && L <= hi + 1;
  S* red = reinterpret_cast<S*>(sh.lines);
  auto sync = [&](bool q) { return group_or(1, used, q); };
  Chunk<S, M> ch;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const S* slot = red + 4 * i * used + threadIdx.x;
    ch.a[i] = slot[0]; ch.b[i] = slot[used]; ch.c[i] = slot[2 * used]; ch.d[i] = slot[3 * used];
  }
  ch.eliminate();
  double o[M];  // read early: nothing else hides their latency
#pragma unroll
  for (int i = 0; i < M; ++i)
    o[i] = mine && old && (dc || !active) ? live(old, min(k * M + i, n - 1) * LD + (L - 1)) : 0.0;
  sync(false);  // every thread holds its rows: their memory serves the reduced system
  S x0, xl;
  reduced_pcr<S, sizeof(S) == 8>(red, TL * gy, TL, gy, threadIdx.x, k, active, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD,
                                 x0, xl, sync);
  ch.substitute(x0, xl);
  if (mine) {
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const int r = k * M + i;
      if (r < n) out[r * LD + (L - 1)] = active ? o[i] + double(ch.d[i]) : o[i];
    }
  }
}

template <int EQ, int SOLVER>
__device__ __forceinline__ double loop_y(const bool first, const int l, const int k, const bool res) {
  using ST = SweepTypes<SOLVER, EQ>;
  const LoopArgs& A = loop_ctx().A;
  const int used = (A.s.y_lines * A.s.gy + 31) & ~31;
  if ((int)threadIdx.x >= used) return 0.0;
  const double acc = assemble_y<EQ, SOLVER>(first, l, k, used, res);
  const LoopIO io = loop_io<EQ>(A, first);
  solve_y<typename ST::S>(l, k, used, EQ == EQ_VY ? A.G.nj : A.G.nj + 1, EQ == EQ_UY ? A.G.mi - 1 : A.G.mi,
                          io.zero_in ? nullptr : io.in, ST::DC, io.out);
  return acc;
}

// pressure and velocity correction (main.f90:931-962) of this CTA's cells
template <bool FAST>
__device__ __noinline__ void loop_correct() {
  const LoopArgs& A = loop_ctx().A;
  const Geo<double>& G = A.G;
  const int ni = G.mi - 1, total = ni * (G.nj - 1);
  const Live* pc = reinterpret_cast<const Live*>(A.pc[0]);
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const int jq = idx / ni, ii = 2 + (idx - jq * ni), jj = 2 + jq;
    const int c0 = G.at(ii, jj);
    const double p0 = A.p[c0], pc0 = pc[c0].v, pce = pc[c0 + 1].v, pcn = pc[c0 + G.LD].v;
    const double u0 = A.u[0][c0], au0 = A.au[c0], v0 = A.v[0][c0], av0 = A.av[c0];
    const double dyu = G.met(M_DYU, jj), dxv = G.met(M_DXV, ii);
    A.p[c0] = p0 + G.p_update * pc0;
    if (ii <= G.mi - 1) A.u[0][c0] = u0 + qdiv<FAST>(dyu * (pc0 - pce), au0);
    if (jj <= G.nj - 1) A.v[0][c0] = v0 + qdiv<FAST>(dxv * (pc0 - pcn), av0);
  }
}

// The loop's state and inputs, in shared memory; thread 0 of every CTA keeps
// its own copy of the same values.
struct LoopState {
  double conv_u, conv_p, conv_t, conv_resi, conv_paso;
  int iter_max, simple_max, fixed;
  int iter_ecuaci, iter_simple, inner_done, outer_done, status, exit_code;
  long long n_simple, n_momen, n_pres, n_ener;
  double err_u, err_p, err_t, maxbo, residuo;
  int go, passes, next;  // next: what the CTA does (LoopNext)
};
enum LoopNext { NEXT_AGAIN = 0, NEXT_ON, NEXT_STOP };

// End of an inner pass (ctl_inner_step).
__device__ __forceinline__ int loop_inner_test(LoopState& s, double err, double extra, double conv) {
  bool again;
  const int done = s.inner_done + 1;
  if (!finite_d(err) || !finite_d(extra)) { s.status = IXB_ENONFINITE; again = false; }
  else if (err < conv) { s.iter_ecuaci = 0; again = false; }
  else if (s.iter_ecuaci > s.iter_max) { s.iter_ecuaci = 0; again = false; }
  else { s.iter_ecuaci++; again = true; }
  if (again && (long long)done >= (long long)s.iter_max + 2) { s.status = IXB_ETIMEOUT; again = false; }
  s.inner_done = again ? done : 0;
  return s.status ? NEXT_STOP : again ? NEXT_AGAIN : NEXT_ON;
}

// End of an outer pass (ctl_outer_step).
__device__ __forceinline__ int loop_outer_test(LoopState& s, double res, int max_outer) {
  s.residuo = res;
  s.n_simple++;
  s.outer_done++;
  if (!finite_d(res)) {
    s.status = IXB_ENONFINITE;
  } else if (s.fixed > 0) {
    s.go = s.outer_done < s.fixed;
  } else {
    if (s.maxbo < s.conv_paso && res < s.conv_resi) { s.iter_simple = 0; s.exit_code = 1; s.go = 0; }
    else if (s.iter_simple > s.simple_max) { s.iter_simple = 0; s.exit_code = 2; s.go = 0; }
    else { s.iter_simple++; s.go = 1; }
    if (s.go && (long long)s.outer_done >= (long long)s.simple_max + 2) { s.status = IXB_ETIMEOUT; s.go = 0; }
  }
  return s.status || !s.go || ++s.passes >= max_outer ? NEXT_STOP : NEXT_ON;
}

template <int SOLVER, int NT>
__global__ void __launch_bounds__(NT, 1) simple_loop_kernel(const __grid_constant__ LoopArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Ctl* c = A.ctl;
  if (A.part == LOOP_ALL && c->stop) return;  // an earlier launch of this run ended it
  grid_arrive(A.waits);
  const int mi = A.G.mi, nj = A.G.nj;
  const int ly = threadIdx.x % A.s.y_lines, ky = threadIdx.x / A.s.y_lines;
  const int gid = threadIdx.x / A.s.gx, kx = threadIdx.x - gid * A.s.gx;
  {
    LoopCtx& sh = loop_ctx();
    const unsigned b = blockIdx.x, nb = gridDim.x;  // at most 384 lines on at most a few hundred CTAs
    const int x0 = 1 + b * (nj + 1) / nb, x0v = 1 + b * nj / nb;
    const int sx = loop_pitch(mi), sy = loop_pitch(nj);
    double* const mx = reinterpret_cast<double*>(smem_raw + up16(sizeof(LoopCtx)));
    double* const my = mx + SX_COUNT * sx;
    if (threadIdx.x == 0) {
      sh.A = A;
      sh.mx = mx;
      sh.my = my;
      sh.sx = sx;
      sh.sy = sy;
      sh.x0 = x0;
      sh.xn = 1 + (b + 1) * (nj + 1) / nb - x0;
      sh.x0v = x0v;
      sh.xnv = 1 + (b + 1) * nj / nb - x0v;
      sh.lines = smem_raw + loop_fixed_bytes(mi, nj);
    }
    const int mxs[SX_COUNT] = {M_DXP, M_DXU, M_FEXP, M_FEXU, M_GRDXP, M_GRDXU, M_HRDXU, M_PEXP, M_PEXU, M_PHXU};
    const int mys[SY_COUNT] = {M_DYP, M_DYV, M_FEYP, M_FEYV, M_GRDYV, M_GRDYP, M_HRDYV, M_PEYV, M_PEYP, M_PHYV};
#pragma unroll
    for (int q = 0; q < SX_COUNT; ++q)
      for (int i = threadIdx.x; i < sx; i += blockDim.x) mx[q * sx + i] = i >= 1 && i <= mi + 1 ? A.G.met(mxs[q], i) : 0.0;
#pragma unroll
    for (int q = 0; q < SY_COUNT; ++q)
      for (int i = threadIdx.x; i < sy; i += blockDim.x) my[q * sy + i] = i >= 1 && i <= nj + 1 ? A.G.met(mys[q], i) : 0.0;
    // boundary rows of this CTA's lines
    constexpr int NX = 3 * 2 * kLoopM, NY = 3 * 2 * kLoopLinesY;
    for (int q = threadIdx.x; q < NX + NY; q += blockDim.x) {
      const bool x = q < NX;
      const int per = x ? kLoopM : kLoopLinesY, w = x ? q : q - NX;
      const int line = w % per, last = (w / per) & 1, var = w / (2 * per);
      const int L = line + (x ? (var == 1 ? x0v : x0) : 1 + (int)b * A.s.y_lines);
      const int side = x ? (last ? 2 : 0) : (last ? 3 : 1);
      BcS e{0.0, 0};
      if (L < A.bcstride) {
        const BCEntry t = A.bc[((size_t)var * 4 + side) * A.bcstride + L];
        e = BcS{t.val, t.type == 2};
      }
      if (x) sh.bcx[var][last][line] = e;
      else sh.bcy[var][last][line] = e;
    }
  }
  __shared__ LoopState s;
  if (threadIdx.x == 0) {
    s.conv_u = c->conv_u; s.conv_p = c->conv_p; s.conv_t = c->conv_t;
    s.conv_resi = c->conv_resi; s.conv_paso = c->conv_paso;
    s.iter_max = c->iter_ecuaci_max; s.simple_max = c->iter_simple_max; s.fixed = c->fixed_count;
    s.iter_ecuaci = c->iter_ecuaci; s.iter_simple = c->iter_simple; s.inner_done = 0; s.outer_done = c->outer_done;
    s.status = 0; s.exit_code = 0;
    s.n_simple = c->n_simple; s.n_momen = c->n_momen; s.n_pres = c->n_pres; s.n_ener = c->n_ener;
    s.err_u = c->err_u; s.err_p = c->err_p; s.err_t = c->err_t; s.maxbo = c->maxbo; s.residuo = c->residuo;
    s.go = 1; s.passes = 0;
  }
  if (!grid_meet(A.waits)) return;
  unsigned target = 0;
  double* const part = A.partials;
  const int np = gridDim.x;
#define IXB_GRID_SYNC() \
  if (!grid_sync(A.waits, target)) return
  const int part_only = A.part;
  // a single-part launch leaves its norms in A.norms and ends
  auto publish = [&](int id, double v) {
    if (blockIdx.x == 0) A.norms[id] = v;
  };
  // the norms of a pass and what follows from them: `test` runs on thread 0
  // with the sums of norms a and b (b < 0: none)
  auto decide = [&](int a, int b, auto test) -> int {
    if (threadIdx.x < 32) {
      const double va = sqrt(sum_partials(part + a * np));
      const double vb = b >= 0 ? sqrt(sum_partials(part + b * np)) : 0.0;
      if (threadIdx.x == 0) {
        if (part_only) {
          publish(a, va);
          if (b >= 0) publish(b, vb);
          s.next = NEXT_STOP;
        } else {
          s.next = test(va, vb);
        }
      }
    }
    __syncthreads();
    return s.next;
  };
  bool pending = part_only == LOOP_RESIDUAL;  // an outer pass is done but for its residual and test
  bool first = part_only != LOOP_PRESSURE;    // of the pressure passes
  int stage = part_only == LOOP_ALL || part_only == LOOP_MOMENTUM || part_only == LOOP_RESIDUAL ? 0
              : part_only == LOOP_CORRECT ? 2 : part_only == LOOP_ENERGY ? 3 : 1;
  for (;;) {
    if (stage == 0) {
      // momentum pass (main.f90:404-740); an outer pass's first u-y sweep also
      // takes the residual of the outer pass before
      const double ar = loop_y<EQ_UY, SOLVER>(false, ly, ky, pending);
      if (pending) post_partials(ar, part + N_RES * np, 0.0, nullptr);
      IXB_GRID_SYNC();
      if (pending) {
        pending = false;
        if (decide(N_RES, -1, [&](double r, double) { return loop_outer_test(s, r, A.max_outer); }) == NEXT_STOP) break;
      }
      loop_x<EQ_UX, SOLVER>(false, gid, kx);
      IXB_GRID_SYNC();
      loop_y<EQ_VY, SOLVER>(false, ly, ky, false);
      IXB_GRID_SYNC();
      post_partials(loop_x<EQ_VX, SOLVER>(false, gid, kx).x, part + N_DV * np, 0.0, nullptr);
      IXB_GRID_SYNC();
      const int next = decide(N_DV, -1, [&](double e, double) {
        s.err_u = e;
        s.n_momen++;
        return loop_inner_test(s, e, 0.0, s.conv_u);
      });
      if (next == NEXT_STOP) break;
      if (next == NEXT_ON) { stage = 1; first = true; }
    } else if (stage == 1) {
      // pressure correction pass, the first one from p' = 0 (main.f90:745-924)
      loop_y<EQ_PY, SOLVER>(first, ly, ky, false);
      IXB_GRID_SYNC();
      const double2 a = loop_x<EQ_PX, SOLVER>(first, gid, kx);
      post_partials(a.x, part + N_DP * np, a.y, part + N_BO * np);
      IXB_GRID_SYNC();
      first = false;
      const int next = decide(N_DP, N_BO, [&](double e, double bo) {
        s.err_p = e;
        s.maxbo = bo;
        s.n_pres++;
        return loop_inner_test(s, e, bo, s.conv_p);
      });
      if (next == NEXT_STOP) break;
      if (next == NEXT_ON) stage = 2;
    } else if (stage == 2) {
      loop_correct<true>();
      if (part_only) break;
      IXB_GRID_SYNC();
      stage = 3;
    } else {
      // energy pass (main.f90:975-1156)
      loop_y<EQ_TY, SOLVER>(false, ly, ky, false);
      IXB_GRID_SYNC();
      post_partials(loop_x<EQ_TX, SOLVER>(false, gid, kx).x, part + N_DT * np, 0.0, nullptr);
      IXB_GRID_SYNC();
      const int next = decide(N_DT, -1, [&](double e, double) {
        s.err_t = e;
        s.n_ener++;
        return loop_inner_test(s, e, 0.0, s.conv_t);
      });
      if (next == NEXT_STOP) break;
      if (next == NEXT_ON) { stage = 0; pending = true; }
    }
  }
#undef IXB_GRID_SYNC
  if (!part_only && blockIdx.x == 0 && threadIdx.x == 0) {
    c->iter_ecuaci = s.iter_ecuaci;
    c->iter_simple = s.iter_simple;
    c->outer_done = s.outer_done;
    c->inner_done = 0;
    c->exit_code = s.exit_code;
    c->status = s.status;
    c->n_simple = s.n_simple; c->n_momen = s.n_momen; c->n_pres = s.n_pres; c->n_ener = s.n_ener;
    c->err_u = s.err_u; c->err_p = s.err_p; c->err_t = s.err_t; c->maxbo = s.maxbo; c->residuo = s.residuo;
    c->stop = s.status != 0 || !s.go;
  }
}

template <int SOLVER, int NT>
cudaError_t loop_go(const LoopArgs& a, cudaStream_t st) {
  auto k = simple_loop_kernel<SOLVER, NT>;
  using S = typename SweepTypes<SOLVER, EQ_UX>::S;
  const size_t line = std::max(a.s.x_lines * a.s.gx, (a.s.y_lines * a.s.gy + 31) / 32 * 32);
  const size_t smem = loop_fixed_bytes(a.G.mi, a.G.nj) + 12 * line * sizeof(S);
  cudaError_t e = allow_smem(k);
  if (e != cudaSuccess) return e;
  LoopArgs args = a;
  void* params[] = {&args};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(a.s.grid), dim3(a.s.threads), params, smem,
                                     st);
}

// The fewest-thread variant that holds the CTA: the register file is shared
// by fewer threads, and a column's loads (28 values) all stay in flight.
template <int SOLVER>
cudaError_t loop_launch_form(const LoopArgs& a, cudaStream_t st) {
  if (a.s.threads <= 256) return loop_go<SOLVER, 256>(a, st);
  if (a.s.threads <= 384) return loop_go<SOLVER, 384>(a, st);
  if (a.s.threads <= 512) return loop_go<SOLVER, 512>(a, st);
  return loop_go<SOLVER, kLoopThreads>(a, st);
}

}  // namespace ixb
