// ixb_device.cuh -- device-side data structures, coefficient assembly and
// line solvers of the SIMPLE hot path.
//
// Layout in HBM: every 2-D field (u, v, p, T, p', the *_ant copies, au, av,
// b_o, Resu, sources) is one array of (nj+2) rows x LD doubles, LD >= mi+1
// with LD = 4 modulo 16 (ixb_create), with Fortran index (ii,jj) at
// (jj-1)*LD + (ii-1).  Adjacent ii are adjacent in memory, so x-lines are
// contiguous and the y-lines of a tile of adjacent ii are read as coalesced
// row segments.  1-D metrics are 1-based arrays (element 0 unused).
//
// Arithmetic of the assembly follows the reference statements operand by
// operand (the library is built with -fmad=false), so the coefficients are
// bit-identical to the reference's IEEE evaluation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ixb {

// First statement of every kernel of the SIMPLE loop: wait for the previous
// kernel of the stream (programmatic dependent launch) and let the next one
// be placed.
#define IXB_PDL_ENTRY()                        \
  do {                                         \
    cudaGridDependencySynchronize();           \
    cudaTriggerProgrammaticLaunchCompletion(); \
  } while (0)

// metric arrays inside one device buffer, each `mstride` long, 1-based.
// M_HXU/M_HYV are the energy equation's face diffusivities
// hmean(ge,ge,fexu(k)) / hmean(ge,ge,feyv(k)), filled by the table kernel.  The
// fast form forms the diffusive conductances gamma*delta/d of the 2-D tables
// below from 1-D factors (a uniform gamma makes them separable): M_GRDXP =
// gamma_momen/dxp, M_GRDYV = gamma_momen/dyv, M_GRDXU = gamma_momen/dxu,
// M_GRDYP = gamma_momen/dyp, M_HRDXU = M_HXU/dxu, M_HRDYV = M_HYV/dyv.  M_PE*
// are the factors of |velocity| in 0.1|Peclet| (0.1 * spacing / diffusivity):
// of gamma_momen with dxp, dyv, dxu and dyp, and of the energy faces (M_PHXU,
// M_PHYV).
enum Metric {
  M_DXP = 0, M_DYP, M_DXU, M_DYU, M_DXV, M_DYV, M_FEXP, M_FEYP, M_FEXU, M_FEYV,
  M_HXU, M_HYV, M_GRDXP, M_GRDYV, M_GRDXU, M_GRDYP, M_HRDXU, M_HRDYV,
  M_PEXP, M_PEYV, M_PEXU, M_PEYP, M_PHXU, M_PHYV, M_COUNT
};

// Mesh-constant 2-D tables (field layout).  With the uniform diffusion
// coefficients of the reference (main.f90:226-239) every harmonic face
// diffusivity and every diffusive conductance gamma*delta/d of the assembly
// is a function of the mesh alone; the table kernel evaluates each one once,
// with the reference's operands in the reference's order, so reading a table
// entry gives the same bits as recomputing it in the cell loop.
//   T_GU (ii,jj)  u: gamman at (ii,jj); gammas(ii,jj) = T_GU(ii,jj-1)
//   T_CU1(ii,jj)  u: gammai*deltay/di;  AD conductance = T_CU1(ii+1,jj)
//   T_CU2(ii,jj)  u: gamman*deltax/dn;  BS conductance = T_CU2(ii,jj-1)
//   T_GV (ii,jj)  v: gammad at (ii,jj); gammai(ii,jj) = T_GV(ii-1,jj)
//   T_CV1(ii,jj)  v: gammai*deltayv/di; AD conductance = T_CV1(ii+1,jj)
//   T_CV2(ii,jj)  v: gammas*deltaxv/ds; BN conductance = T_CV2(ii,jj+1)
//   T_CT1(ii,jj)  T: gammai*deltayp/di; AD conductance = T_CT1(ii+1,jj)
//   T_CT2(ii,jj)  T: gamman*deltaxp/dn; BS conductance = T_CT2(ii,jj-1)
//   (the fast form takes its Peclet numbers from the M_PE* factors: the face
//   diffusivities of a uniform gamma are gamma itself up to rounding)
enum Table { T_GU = 0, T_CU1, T_CU2, T_GV, T_CV1, T_CV2, T_CT1, T_CT2, T_COUNT };

// sweeps: the eight line-solve phases of main.f90
enum Eq { EQ_UY = 0, EQ_UX, EQ_VY, EQ_VX, EQ_PY, EQ_PX, EQ_TY, EQ_TX, EQ_COUNT };

struct BCEntry {  // effective boundary row of one line (last covering segment wins)
  double val;
  int type;       // 0 none, 1 diri, 2 neum
  int pad;
};

struct BatchNorm {          // per-instance norms of a batched launch
  double* partials;         // one per work item of the launch (null: no norm)
  unsigned int* counter;    // one per instance
  double* result;           // one per instance
};

struct NormSlot {        // deterministic two-level sum of squares
  double* partials;      // one per CTA
  unsigned int* counter; // CTAs finished (reset by the last one)
  double* result;        // sqrt(sum) written by the last CTA
};

// Read-only loads of the assembly: every array an assembly reads is left
// untouched by the kernel that reads it, so the non-coherent path applies
// and the compiler may batch the loads ahead of the shared-memory stores.
template <class R>
__device__ __forceinline__ R ldg(const R* p, int i) { return __ldg(p + i); }
// the same load converted to the assembly's arithmetic type (a no-op when
// the field and the arithmetic are both binary64)
template <class R, class F>
__device__ __forceinline__ R ld(const F* p, int i) { return R(__ldg(p + i)); }
// A binary64 field that other CTAs of the same launch write between grid
// barriers (the loop kernel): ordinary loads, which see those writes, in
// place of the read-only path.
struct Live { double v; };
template <class R>
__device__ __forceinline__ R ld(const Live* p, int i) { return p[i].v; }
template <class R>
struct Geo {
  int mi, nj, LD, mstride;
  int tstride;     // elements per 2-D table (fields stay below 2^31 elements)
  const R* m;      // M_COUNT 1-D arrays
  const R* tab;    // T_COUNT 2-D tables
  R gm, ge, Ri, Riy, dt, rel_vel, rel_pres, rel_ener, p_update;
  R inv_dt, inv_rel_vel, inv_rel_pres, inv_rel_ener;  // fast form
  __device__ __forceinline__ R met(int which, int k) const { return __ldg(m + which * mstride + k); }
  __device__ __forceinline__ int at(int ii, int jj) const { return (jj - 1) * LD + (ii - 1); }
  __device__ __forceinline__ R t(int which, int ii, int jj) const { return __ldg(tab + which * tstride + at(ii, jj)); }
};

template <class R>
struct SweepIO {
  const R *u, *v, *T, *p, *pc;        // current fields
  const double *u_ant, *v_ant, *T_ant;
  const R *au, *av;
  const double *fcon, *flin;          // sources of this equation (null when none)
  const R* in;                        // swept field, current values
  double* out;                        // swept field, new values
  const double* prev;                 // field at the start of the inner pass (null: zero)
  double* aux;                        // au (u-x), av (v-x), b_o (p'-x)
  const BCEntry* bc_first;            // indexed by line
  const BCEntry* bc_last;
  NormSlot nrm0;                      // ||out - prev|| over interior rows of solved lines
  NormSlot nrm1;                      // ||b_o|| (p'-x)
};

// What an assembly reads at and around cell (ii,jj): the swept field `in`,
// the other fields, the previous time level and the sources at the cell, the
// 1-D metrics and the mesh tables, all by offset.  CellView loads each value
// where it is asked for; the resident loop's column view holds three cells'
// values in registers (ixb_loop.cuh).
template <class R, class F>
struct CellView {
  const Geo<R>& G;
  const SweepIO<F>& io;
  int ii, jj;
  __device__ __forceinline__ int at(int di, int dj) const { return G.at(ii + di, jj + dj); }
  __device__ __forceinline__ R in(int di, int dj) const { return ld<R>(io.in, at(di, dj)); }
  __device__ __forceinline__ R u(int di, int dj) const { return ld<R>(io.u, at(di, dj)); }
  __device__ __forceinline__ R v(int di, int dj) const { return ld<R>(io.v, at(di, dj)); }
  __device__ __forceinline__ R T(int di, int dj) const { return ld<R>(io.T, at(di, dj)); }
  __device__ __forceinline__ R p(int di, int dj) const { return ld<R>(io.p, at(di, dj)); }
  __device__ __forceinline__ R au(int di, int dj) const { return ld<R>(io.au, at(di, dj)); }
  __device__ __forceinline__ R av(int di, int dj) const { return ld<R>(io.av, at(di, dj)); }
  __device__ __forceinline__ R u_ant() const { return ld<R>(io.u_ant, at(0, 0)); }
  __device__ __forceinline__ R v_ant() const { return ld<R>(io.v_ant, at(0, 0)); }
  __device__ __forceinline__ R T_ant() const { return ld<R>(io.T_ant, at(0, 0)); }
  // no sources: no loads (the values would be +0)
  __device__ __forceinline__ R fcon() const { return io.fcon ? ld<R>(io.fcon, at(0, 0)) : R(0); }
  __device__ __forceinline__ R flin() const { return io.flin ? ld<R>(io.flin, at(0, 0)) : R(0); }
  __device__ __forceinline__ R mx(int which, int di) const { return G.met(which, ii + di); }  // metrics along x
  __device__ __forceinline__ R my(int which, int dj) const { return G.met(which, jj + dj); }  // and along y
  __device__ __forceinline__ R tab(int which, int di, int dj) const { return G.t(which, ii + di, jj + dj); }
};

// Diffusive conductances.  The exact form reads the 2-D table entry (the
// reference's operands in its order); the fast form multiplies the cell's 1-D
// mesh factor by a 1-D reciprocal factor, an L1-resident load in place of a
// 2-D table read, which differs from the table by rounding:
//   u: T_CU1(ii,jj) = dyu(jj) * GRDXP(ii);   T_CU2(ii,jj) = dxu(ii) * GRDYV(jj)
//   v: T_CV1(ii,jj) = dyv(jj) * GRDXU(ii-1); T_CV2(ii,jj) = dxv(ii) * GRDYP(jj)
//   T: T_CT1(ii,jj) = dyp(jj) * HRDXU(ii-1); T_CT2(ii,jj) = dxp(ii) * HRDYV(jj)

template <class R>
struct Row { R a, b, c, d; };

// math on either binary32 or binary64 operands without promotion
__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fabsT(float x) { return fabsf(x); }
__device__ __forceinline__ double fabsT(double x) { return fabs(x); }
__device__ __forceinline__ float fmaxT(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double fmaxT(double a, double b) { return fmax(a, b); }

// DMAX1(0, (1 - 0.1|P|)**5): the integer power as binary powering x*((x*x)*(x*x))
template <class R>
__device__ __forceinline__ R plaw(R pe) {
  R t = R(1) - R(0.1) * fabsT(pe);
  R t2 = t * t;
  R t5 = t * (t2 * t2);
  return fmaxT(R(0), t5);
}
template <class R>
__device__ __forceinline__ R dmax0(R x) { return fmaxT(R(0), x); }
// max(0, x) by the sign bit (three integer operations; the binary64 maximum
// takes the binary64 pipe, which the fast rows keep busy).  NaN gives +0 or NaN,
// by its own sign bit (fmax: +0): a row with a velocity that is not a number
// carries it through the field values of its right-hand side.
__device__ __forceinline__ double pos(double x) {
  const int hi = __double2hiint(x), keep = ~(hi >> 31);
  return __hiloint2double(hi & keep, __double2loint(x) & keep);
}
// Fast form of a neighbour coefficient (with its sign): conductance
// max(0, 1 - 0.1|Pe|)^5 plus the upwind part of the flux, 0.1|Pe| = |vel| m.
__device__ __forceinline__ double plaw_fast(double vel, double m) {
  const double t = pos(fma(-fabs(vel), m, 1.0)), t2 = t * t;
  return t * (t2 * t2);
}
__device__ __forceinline__ double link_fast(double cond, double law, double flux) {
  return -fma(cond, law, pos(flux));
}

// harmonic face interpolation g1*g2/(g1*(1-f)+g2*f) of the reference
// (e.g. source/mod_ec_momento.f90:462-465) with its operand order
template <class R>
__device__ __forceinline__ R hmean(R g1, R g2, R f) {
  return (g1 * g2) / (g1 * (R(1) - f) + g2 * f);
}

// Reciprocal for the fast form: Newton-Raphson refinement
// r <- r + r(1 - x r) of a hardware reciprocal estimate (two steps for
// binary64, one for binary32).
__device__ __forceinline__ double fast_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  r = fma(r, fma(-x, r, 1.0), r);
  return r;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(r, fmaf(-x, r, 1.0f), r);
}

// a / b.  EXACT (FAST=false): the IEEE quotient of the reference.  FAST:
// a * rb with rb ~ 1/b precomputed (or, when rb is not given, estimated).
template <bool FAST, class R>
__device__ __forceinline__ R qdiv(R a, R b, R rb) { if constexpr (FAST) return a * rb; else return a / b; }
template <bool FAST, class R>
__device__ __forceinline__ R qdiv(R a, R b) { if constexpr (FAST) return a * fast_rcp(b); else return a / b; }

// ---------------------------------------------------------------------------
// u momentum (ensambla_velu_x/_y, source/mod_ec_momento.f90:365-724)
// ---------------------------------------------------------------------------
// The four neighbour coefficients of the u row (:512-526), face velocities
// interpolated as in :447-455, diffusivities and conductances from the
// tables (gammai = gammad = gamma_momen).
// Without buoyancy (coefficient 0) the fast form leaves T unread.
template <bool FAST, class R, class V>
__device__ __forceinline__ void u_parts(const Geo<R>& G, const V& c, R& AI, R& AD, R& BS, R& BN, R& deltax, R& deltay,
                                        R& temp_int) {
  const R fexu_i = c.mx(M_FEXU, 0), fexu_m = c.mx(M_FEXU, -1);
  const R fexp_i = c.mx(M_FEXP, 0);
  R ud = fexu_i * c.in(1, 0) + (R(1) - fexu_i) * c.in(0, 0);
  R ui = fexu_m * c.in(0, 0) + (R(1) - fexu_m) * c.in(-1, 0);
  R vn = fexp_i * c.v(1, 0) + (R(1) - fexp_i) * c.v(0, 0);
  R vs = fexp_i * c.v(1, -1) + (R(1) - fexp_i) * c.v(0, -1);
  deltax = c.mx(M_DXU, 0);
  deltay = c.my(M_DYU, 0);
  if constexpr (FAST) {
    // the face diffusivities are harmonic means of a uniform gamma_momen
    // (ixb_params holds one value), i.e. gamma_momen up to rounding
    temp_int = R(0);
    if (G.Ri != R(0)) temp_int = fexp_i * c.T(1, 0) + (R(1) - fexp_i) * c.T(0, 0);
    AI = link_fast(deltay * c.mx(M_GRDXP, 0), plaw_fast(ui, c.mx(M_PEXP, 0)), ui * deltay);
    AD = link_fast(deltay * c.mx(M_GRDXP, 1), plaw_fast(ud, c.mx(M_PEXP, 1)), -ud * deltay);
    BS = link_fast(deltax * c.my(M_GRDYV, -1), plaw_fast(vs, c.my(M_PEYV, -1)), vs * deltax);
    BN = link_fast(deltax * c.my(M_GRDYV, 0), plaw_fast(vn, c.my(M_PEYV, 0)), -vn * deltax);
  } else {
    const R g = G.gm;
    const R gamman = c.tab(T_GU, 0, 0), gammas = c.tab(T_GU, 0, -1);
    R di = c.mx(M_DXP, 0), dd = c.mx(M_DXP, 1), ds = c.my(M_DYV, -1), dn = c.my(M_DYV, 0);
    temp_int = fexp_i * c.T(1, 0) + (R(1) - fexp_i) * c.T(0, 0);
    AI = -(c.tab(T_CU1, 0, 0) * plaw(ui * di / g) + dmax0(ui * deltay));
    AD = -(c.tab(T_CU1, 1, 0) * plaw(ud * dd / g) + dmax0(-ud * deltay));
    BS = -(c.tab(T_CU2, 0, -1) * plaw(vs * ds / gammas) + dmax0(vs * deltax));
    BN = -(c.tab(T_CU2, 0, 0) * plaw(vn * dn / gamman) + dmax0(-vn * deltax));
  }
}

// X form (ensambla_velu_x): a=AI c=AD b=AC d=Rx, aux = au = AC*rel
template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_ux(const Geo<R>& G, const V& c, R& au) {
  R AI, AD, BS, BN, dx, dy, tint;
  u_parts<FAST>(G, c, AI, AD, BS, BN, dx, dy, tint);
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = AI;
  r.c = AD;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dx * dy * flin + qdiv<FAST>(dx * dy, G.dt, G.inv_dt), G.rel_vel,
                   G.inv_rel_vel);
  r.d = -BS * c.in(0, -1) - BN * c.in(0, 1) - dx * dy * G.Ri * tint + dx * dy * fcon +
        qdiv<FAST>(dx * dy * c.u_ant(), G.dt, G.inv_dt) + (c.p(0, 0) - c.p(1, 0)) * dy +
        r.b * (R(1) - G.rel_vel) * c.in(0, 0);
  au = r.b * G.rel_vel;
  return r;
}

// Y form (ensambla_velu_y): a=BS c=BN b=BC d=Ry
template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_uy(const Geo<R>& G, const V& c) {
  R AI, AD, BS, BN, dx, dy, tint;
  u_parts<FAST>(G, c, AI, AD, BS, BN, dx, dy, tint);
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = BS;
  r.c = BN;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dx * dy * flin + qdiv<FAST>(dx * dy, G.dt, G.inv_dt), G.rel_vel,
                   G.inv_rel_vel);
  r.d = -AI * c.in(-1, 0) - AD * c.in(1, 0) - dx * dy * G.Ri * tint + dx * dy * fcon +
        qdiv<FAST>(dx * dy * c.u_ant(), G.dt, G.inv_dt) + (c.p(0, 0) - c.p(1, 0)) * dy +
        r.b * (R(1) - G.rel_vel) * c.in(0, 0);
  return r;
}

// ---------------------------------------------------------------------------
// v momentum (ensambla_velv_x/_y, source/mod_ec_momento.f90:736-1098)
// ---------------------------------------------------------------------------
template <bool FAST, class R, class V>
__device__ __forceinline__ void v_parts(const Geo<R>& G, const V& c, R& AI, R& AD, R& BS, R& BN, R& temp_int) {
  const R feyp_j = c.my(M_FEYP, 0);
  const R feyv_j = c.my(M_FEYV, 0), feyv_m = c.my(M_FEYV, -1);
  R ud = feyp_j * c.u(0, 1) + (R(1) - feyp_j) * c.u(0, 0);
  R ui = feyp_j * c.u(-1, 1) + (R(1) - feyp_j) * c.u(-1, 0);
  R vn = feyv_j * c.in(0, 1) + (R(1) - feyv_j) * c.in(0, 0);
  R vs = feyv_m * c.in(0, 0) + (R(1) - feyv_m) * c.in(0, -1);
  const R dyv = c.my(M_DYV, 0), dxv = c.mx(M_DXV, 0);
  if constexpr (FAST) {
    temp_int = R(0);
    if (G.Riy != R(0)) temp_int = feyp_j * c.T(0, 1) + (R(1) - feyp_j) * c.T(0, 0);
    AI = link_fast(dyv * c.mx(M_GRDXU, -1), plaw_fast(ui, c.mx(M_PEXU, -1)), ui * dyv);
    AD = link_fast(dyv * c.mx(M_GRDXU, 0), plaw_fast(ud, c.mx(M_PEXU, 0)), -ud * dyv);
    BS = link_fast(dxv * c.my(M_GRDYP, 0), plaw_fast(vs, c.my(M_PEYP, 0)), vs * dxv);
    BN = link_fast(dxv * c.my(M_GRDYP, 1), plaw_fast(vn, c.my(M_PEYP, 1)), -vn * dxv);
  } else {
    const R g = G.gm;  // gamman = gammas = gamma_momen (:854-858)
    const R gammad = c.tab(T_GV, 0, 0), gammai = c.tab(T_GV, -1, 0);
    R di = c.mx(M_DXU, -1), dd = c.mx(M_DXU, 0), ds = c.my(M_DYP, 0), dn = c.my(M_DYP, 1);
    temp_int = feyp_j * c.T(0, 1) + (R(1) - feyp_j) * c.T(0, 0);
    AI = -(c.tab(T_CV1, 0, 0) * plaw(ui * di / gammai) + dmax0(ui * dyv));
    AD = -(c.tab(T_CV1, 1, 0) * plaw(ud * dd / gammad) + dmax0(-ud * dyv));
    BS = -(c.tab(T_CV2, 0, 0) * plaw(vs * ds / g) + dmax0(vs * dxv));
    BN = -(c.tab(T_CV2, 0, 1) * plaw(vn * dn / g) + dmax0(-vn * dxv));
  }
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_vx(const Geo<R>& G, const V& c, R& av) {
  R AI, AD, BS, BN, tint;
  v_parts<FAST>(G, c, AI, AD, BS, BN, tint);
  const R dxv = c.mx(M_DXV, 0), dyv = c.my(M_DYV, 0);
  const R dxdy = dxv * dyv;
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = AI;
  r.c = AD;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dxdy * flin + qdiv<FAST>(dxdy, G.dt, G.inv_dt), G.rel_vel, G.inv_rel_vel);
  r.d = -BS * c.in(0, -1) - BN * c.in(0, 1) - dxdy * G.Riy * tint + dxdy * fcon +
        qdiv<FAST>(dxdy * c.v_ant(), G.dt, G.inv_dt) + (c.p(0, 0) - c.p(0, 1)) * dxv +
        r.b * (R(1) - G.rel_vel) * c.in(0, 0);
  av = r.b * G.rel_vel;
  return r;
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_vy(const Geo<R>& G, const V& c) {
  R AI, AD, BS, BN, tint;
  v_parts<FAST>(G, c, AI, AD, BS, BN, tint);
  const R dxv = c.mx(M_DXV, 0), dyv = c.my(M_DYV, 0);
  const R dxdy = dxv * dyv;
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = BS;
  r.c = BN;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dxdy * flin + qdiv<FAST>(dxdy, G.dt, G.inv_dt), G.rel_vel, G.inv_rel_vel);
  r.d = -AI * c.in(-1, 0) - AD * c.in(1, 0) - dxdy * G.Riy * tint + dxdy * fcon +
        qdiv<FAST>(dxdy * c.v_ant(), G.dt, G.inv_dt) + (c.p(0, 0) - c.p(0, 1)) * dxv +
        r.b * (R(1) - G.rel_vel) * c.in(0, 0);
  return r;
}

// ---------------------------------------------------------------------------
// energy (ensambla_energia_x/_y, source/mod_ec_energia.f90:119-443).  The
// calls in main.f90:989 and :1060 bind fexu/feyv to the dummies fexpo/feypo.
// ---------------------------------------------------------------------------
template <bool FAST, class R, class V>
__device__ __forceinline__ void t_parts(const Geo<R>& G, const V& c, R& AI, R& AD, R& BS, R& BN) {
  const R ud = c.u(0, 0), ui = c.u(-1, 0);
  const R vn = c.v(0, 0), vs = c.v(0, -1);
  const R dyp = c.my(M_DYP, 0), dxp = c.mx(M_DXP, 0);
  if constexpr (FAST) {
    AI = link_fast(dyp * c.mx(M_HRDXU, -1), plaw_fast(ui, c.mx(M_PHXU, -1)), ui * dyp);
    AD = link_fast(dyp * c.mx(M_HRDXU, 0), plaw_fast(ud, c.mx(M_PHXU, 0)), -ud * dyp);
    BS = link_fast(dxp * c.my(M_HRDYV, -1), plaw_fast(vs, c.my(M_PHYV, -1)), vs * dxp);
    BN = link_fast(dxp * c.my(M_HRDYV, 0), plaw_fast(vn, c.my(M_PHYV, 0)), -vn * dxp);
  } else {
    const R di = c.mx(M_DXU, -1), dd = c.mx(M_DXU, 0), ds = c.my(M_DYV, -1), dn = c.my(M_DYV, 0);
    const R gammad = c.mx(M_HXU, 0);
    const R gammai = c.mx(M_HXU, -1);
    const R gamman = c.my(M_HYV, 0);
    const R gammas = c.my(M_HYV, -1);
    AI = -(c.tab(T_CT1, 0, 0) * plaw(ui * di / gammai) + dmax0(ui * dyp));
    AD = -(c.tab(T_CT1, 1, 0) * plaw(ud * dd / gammad) + dmax0(-ud * dyp));
    BS = -(c.tab(T_CT2, 0, -1) * plaw(vs * ds / gammas) + dmax0(vs * dxp));
    BN = -(c.tab(T_CT2, 0, 0) * plaw(vn * dn / gamman) + dmax0(-vn * dxp));
  }
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_tx(const Geo<R>& G, const V& c) {
  R AI, AD, BS, BN;
  t_parts<FAST>(G, c, AI, AD, BS, BN);
  const R dxdy = c.mx(M_DXP, 0) * c.my(M_DYP, 0);
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = AI;
  r.c = AD;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dxdy * flin + qdiv<FAST>(dxdy, G.dt, G.inv_dt), G.rel_ener, G.inv_rel_ener);
  r.d = -BS * c.in(0, -1) - BN * c.in(0, 1) + dxdy * fcon + qdiv<FAST>(dxdy * c.T_ant(), G.dt, G.inv_dt) +
        r.b * (R(1) - G.rel_ener) * c.in(0, 0);
  return r;
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_ty(const Geo<R>& G, const V& c) {
  R AI, AD, BS, BN;
  t_parts<FAST>(G, c, AI, AD, BS, BN);
  const R dxdy = c.mx(M_DXP, 0) * c.my(M_DYP, 0);
  const R flin = c.flin(), fcon = c.fcon();
  Row<R> r;
  r.a = BS;
  r.c = BN;
  r.b = qdiv<FAST>(-AI - AD - BS - BN - dxdy * flin + qdiv<FAST>(dxdy, G.dt, G.inv_dt), G.rel_ener, G.inv_rel_ener);
  r.d = -AI * c.in(-1, 0) - AD * c.in(1, 0) + dxdy * fcon + qdiv<FAST>(dxdy * c.T_ant(), G.dt, G.inv_dt) +
        r.b * (R(1) - G.rel_ener) * c.in(0, 0);
  return r;
}

// ---------------------------------------------------------------------------
// pressure correction (ensambla_corr_pres_x/_y, source/mod_ec_momento.f90:145-355)
// ---------------------------------------------------------------------------
// Mass source b_o = (u_w - u_e) dy + (v_s - v_n) dx of the p' rows, always
// in the fields' precision (binary64) with binary64 metrics, whatever the
// precision of the coefficients.
template <class R, class V>
__device__ __forceinline__ double mass_residual(const Geo<R>& G, const V& c) {
  const double ud = c.u(0, 0), ui = c.u(-1, 0), vn = c.v(0, 0), vs = c.v(0, -1);
  return (ui - ud) * double(c.my(M_DYP, 0)) + (vs - vn) * double(c.mx(M_DXP, 0));
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_px(const Geo<R>& G, const V& c, double& bo) {
  const R ai = c.au(-1, 0), ad = c.au(0, 0), as = c.av(0, -1), an = c.av(0, 0);
  const R dyp = c.my(M_DYP, 0), dxp = c.mx(M_DXP, 0);
  Row<R> r;
  r.a = -qdiv<FAST>(dyp * dyp, ai);
  r.c = -qdiv<FAST>(dyp * dyp, ad);
  const R BS = -qdiv<FAST>(dxp * dxp, as);
  const R BN = -qdiv<FAST>(dxp * dxp, an);
  r.b = qdiv<FAST>(-r.a - r.c - BS - BN, G.rel_pres, G.inv_rel_pres);
  bo = mass_residual(G, c);
  r.d = -BS * c.in(0, -1) - BN * c.in(0, 1) + R(bo) + (R(1) - G.rel_pres) * r.b * c.in(0, 0);
  return r;
}

template <bool FAST, class R, class V>
__device__ __forceinline__ Row<R> assemble_py(const Geo<R>& G, const V& c) {
  const R ai = c.au(-1, 0), ad = c.au(0, 0), as = c.av(0, -1), an = c.av(0, 0);
  const R dyp = c.my(M_DYP, 0), dxp = c.mx(M_DXP, 0);
  const R AI = -qdiv<FAST>(dyp * dyp, ai);
  const R AD = -qdiv<FAST>(dyp * dyp, ad);
  Row<R> r;
  r.a = -qdiv<FAST>(dxp * dxp, as);
  r.c = -qdiv<FAST>(dxp * dxp, an);
  r.b = qdiv<FAST>(-AI - AD - r.a - r.c, G.rel_pres, G.inv_rel_pres);
  const R bo = R(mass_residual(G, c));
  r.d = -AI * c.in(-1, 0) - AD * c.in(1, 0) + bo + (R(1) - G.rel_pres) * r.b * c.in(0, 0);
  return r;
}

// ---------------------------------------------------------------------------
// u residual (residuo_u, source/mod_ec_momento.f90:1107-1266) of the cell's
// u (`in` of the view).  With a uniform gamma the reference's different south
// numerator (:1208) has the same value as in ensambla_velu_x, so it shares
// the u coefficients.
// ---------------------------------------------------------------------------
template <bool FAST, class R, class V>
__device__ __forceinline__ R residual_u(const Geo<R>& G, const V& c) {
  R AI, AD, BS, BN, dxu, dyu, temp_int;
  u_parts<FAST>(G, c, AI, AD, BS, BN, dxu, dyu, temp_int);
  AI = -AI; AD = -AD; BS = -BS; BN = -BN;
  const R fl = c.flin(), fc = c.fcon();
  R AC = AI + AD + BS + BN - dxu * dyu * fl + qdiv<FAST>(dxu * dyu, G.dt, G.inv_dt);
  return AI * c.in(-1, 0) - AC * c.in(0, 0) + AD * c.in(1, 0) + BS * c.in(0, -1) + BN * c.in(0, 1) -
         dxu * dyu * G.Ri * temp_int + dxu * dyu * fc + qdiv<FAST>(dxu * dyu * c.u_ant(), G.dt, G.inv_dt) +
         (c.p(0, 0) - c.p(1, 0)) * dyu;
}
// the same from field pointers; T_WRITTEN: T was written earlier in the
// calling kernel (a fused T-x sweep evaluating the residual of the rows it
// solved), so it is read with ordinary coherent loads
template <class R, bool T_WRITTEN>
struct ResidView : CellView<R, R> {
  __device__ __forceinline__ R T(int di, int dj) const {
    const int k = this->at(di, dj);
    return T_WRITTEN ? this->io.T[k] : ldg(this->io.T, k);
  }
};
template <bool FAST, class R, bool T_WRITTEN = false>
__device__ __forceinline__ R residual_u(const Geo<R>& G, const R* u, const R* v, const R* T, const R* p,
                                        const R* u_ant, const R* fcon, const R* flin, int ii, int jj) {
  SweepIO<R> io{};
  io.in = u; io.v = v; io.T = T; io.p = p; io.u_ant = u_ant; io.fcon = fcon; io.flin = flin;
  return residual_u<FAST>(G, ResidView<R, T_WRITTEN>{{G, io, ii, jj}});
}

// ---------------------------------------------------------------------------
// Line solvers on a line staged in shared memory.
// Row r of the (padded) line lives in chunk r / m at slot r % m; each row
// array is [G][mp] with mp odd, so G threads walking their chunks in step
// hit distinct banks.
// ---------------------------------------------------------------------------

// Sequential Thomas, one thread, the exact operation order of
// tridiagonal (source/mod_solucionador.f90:25-47).  Solution left in sd.
template <class R>
__device__ void thomas_exact(R* sa, R* sb, R* sc, R* sd, int n, int m, int mp) {
  int lane = 0, k = 0;
  int prev = 0;  // offset of row i-1
  for (int i = 1; i < n; ++i) {
    if (++k == m) { k = 0; ++lane; }
    const int o = lane * mp + k;
    const R q = sa[o] / sb[prev];
    sd[o] = sd[o] - q * sd[prev];
    sb[o] = sb[o] - q * sc[prev];
    prev = o;
  }
  sd[prev] = sd[prev] / sb[prev];
  int nxt = prev;
  for (int i = n - 2; i >= 0; --i) {
    if (--k < 0) { k = m - 1; --lane; }
    const int o = lane * mp + k;
    sd[o] = (sd[o] - sc[o] * sd[nxt]) / sb[o];
    nxt = o;
  }
}

// Shared-memory footprint (elements) of one line: the four row arrays of G
// chunks (pitch mp), plus the reduced system (two sets of the 2G normalised
// rows a, c, d).
__host__ __device__ constexpr size_t line_smem_elems(int G, int mp) { return (size_t)4 * G * mp + (size_t)12 * G; }

// Barrier `id` (1..15) of n threads (whole warps); returns whether q holds in
// any of them.
__device__ __forceinline__ bool barrier_or(int id, int n, bool q) {
  int r;
  asm volatile(
      "{ .reg .pred p, a; setp.ne.s32 a, %3, 0; barrier.cta.red.or.pred p, %1, %2, a; selp.s32 %0, 1, 0, p; }"
      : "=r"(r)
      : "r"(id), "r"(n), "r"((int)q)
      : "memory");
  return r != 0;
}

// Barrier of the G threads that solve one line when a CTA holds TL lines of
// whole warps (a named barrier per line, so lines do not wait for each
// other), else of the whole CTA.
template <int G, int TL>
__device__ __forceinline__ bool line_sync(bool q) {
  if constexpr (TL > 1 && TL <= 8 && G % 32 == 0) return barrier_or(1 + (int)threadIdx.x / G, G, q);
  else return __syncthreads_or(q);
}

// One parallel-cyclic-reduction step of a row with unit diagonal,
// x + A x_lo + C x_hi = D, against its two neighbours' rows.
template <class R>
__device__ __forceinline__ void pcr_row(R& A, R& C, R& D, R lA, R lC, R lD, R hA, R hC, R hD) {
  const R r = fast_rcp(fmaT(-C, hA, fmaT(-A, lC, R(1))));
  const R nA = -A * lA * r, nC = -C * hC * r, nD = fmaT(-C, hD, fmaT(-A, lD, D)) * r;
  A = nA; C = nC; D = nD;
}

// Reduced system of a partitioned line solve: the first and last rows of G
// chunks, each with unit diagonal, coupled to the neighbouring chunks' end
// rows (row 2k: eA x_{2k-1} + x_{2k} + eC x_{2k+1} = eD; row 2k+1 likewise
// with oA, oC, oD).  Thread k of a line supplies rows 2k, 2k+1 and receives
// their solutions x0, xl by parallel cyclic reduction over shared memory.
//
// The solve is bound by shared-memory bandwidth (nothing else in it comes
// close), so a thread keeps its own rows in registers and exchanges only
// what its neighbours read.  The first step (row distance 1) couples even
// and odd rows; every later one couples rows of one parity at distance h in
// k, i.e. two independent systems of G rows.
//  * HALF: only the odd (last) rows are reduced further and the even ones
//    follow by substitution: 9 shared-memory words per step and thread.
//  * otherwise both parities: 18 words, the operations of a plain 2G-row
//    cyclic reduction in its order (binary32 p' lines are solved outright,
//    so the form whose rounding they had is kept).
// The textbook form (rows re-read every step) moved 24 words.
//
// Each step squares the couplings (they are below one in diagonally dominant
// rows), and the loop ends after a step whose neighbours added no more to any
// row of the line than a part t of that row's own right-hand side (pcr_more),
// t^2 being far below rounding.  Then nothing more can be seen in any
// component, however small it is beside the others.  For let |A D_lo| + |C D_hi|
// <= t |D| in every row of x + K x = D, K the couplings.  With the |D| as weights
// K has the maximum norm t at most, so |x| <= |D| / (1 - t).  The step gives
// x + K' x = D' where K' is K^2 without its diagonal, over 1 - that diagonal, and
// |D'| >= |D| (1 - t) / (1 + t^2); hence |x - D'| <= t^2 |D'| up to terms of t^3:
// dropping the steps that would follow costs a part t^2 of each component.
// (A line that decays from its boundary value goes on until its last chunks
// have theirs; a test of the couplings' size alone left them at zero.  A row of
// zeros has to get exact zeros.)  The test rides on the barrier that publishes
// the next rows.  701x301, per outer iteration, against all steps: 82.2 against
// 88.9 us binary64, 84.6 against 96.3 us refined.
//
// N elements per array in `red` (9N used with HALF, else 12N); the rows of
// neighbouring chunks are TS elements apart.  All threads of the line(s)
// call `sync(q)`, which orders shared memory between them and returns
// whether q holds in any of them; `active` false: barriers only.
//
// Whether more steps are needed after the one of x + A x_lo + C x_hi = D (not a
// number: yes, it has to reach the whole line).  t^2 is 2^-58 in binary64, 2^-44
// in binary32: the last bits are those of all steps.
template <class R>
__device__ __forceinline__ bool pcr_more(R A, R C, R D, R lD, R hD) {
  const R t = sizeof(R) == 8 ? R(1.862645149230957e-9) : R(2.384185791015625e-7);  // 2^-29, 2^-22
  return !(fabsT(A * lD) + fabsT(C * hD) <= t * fabsT(D));
}

template <class R, bool HALF, class Sync>
__device__ __forceinline__ void reduced_pcr(R* red, const int N, const int TS, const int G, const int pos,
                                            const int k, const bool active, R eA, R eC, R eD, R oA, R oC, R oD,
                                            R& x0, R& xl, Sync sync) {
  const bool lo1 = active && k > 0, hi1 = active && k + 1 < G;
  if constexpr (HALF) {
    if (active) { red[pos] = eA; red[N + pos] = eC; red[2 * N + pos] = eD; }
    sync(false);
    R hA = R(0), hC = R(0), hD = R(0);
    if (hi1) { hA = red[pos + TS]; hC = red[N + pos + TS]; hD = red[2 * N + pos + TS]; }
    pcr_row(oA, oC, oD, eA, eC, eD, hA, hC, hD);
    R* cur = red + 3 * N;
    R* nxt = red + 6 * N;
    bool more = true;
#pragma unroll 1
    for (int h = 1; h < G; h <<= 1) {
      if (active) { cur[pos] = oA; cur[N + pos] = oC; cur[2 * N + pos] = oD; }
      if (!sync(active && more)) break;
      R lA = R(0), lC = R(0), lD = R(0);
      hA = hC = hD = R(0);
      if (active && k >= h) {
        const int q = pos - h * TS;
        lA = cur[q]; lC = cur[N + q]; lD = cur[2 * N + q];
      }
      if (active && k + h < G) {
        const int q = pos + h * TS;
        hA = cur[q]; hC = cur[N + q]; hD = cur[2 * N + q];
      }
      more = pcr_more(oA, oC, oD, lD, hD);
      pcr_row(oA, oC, oD, lA, lC, lD, hA, hC, hD);
      R* t = cur; cur = nxt; nxt = t;
    }
    xl = oD;
    if (active) cur[pos] = xl;  // a buffer nobody reads any more: no step follows the one it was published for
    sync(false);
    const R xm = lo1 ? cur[pos - TS] : R(0);
    x0 = fmaT(-eC, xl, fmaT(-eA, xm, eD));
  } else {
    R* cur = red;
    R* nxt = red + 6 * N;
    if (active) {
      cur[pos] = eA; cur[N + pos] = eC; cur[2 * N + pos] = eD;
      cur[3 * N + pos] = oA; cur[4 * N + pos] = oC; cur[5 * N + pos] = oD;
    }
    sync(false);
    {
      R lA = R(0), lC = R(0), lD = R(0), hA = R(0), hC = R(0), hD = R(0);
      if (lo1) { lA = cur[3 * N + pos - TS]; lC = cur[4 * N + pos - TS]; lD = cur[5 * N + pos - TS]; }
      if (hi1) { hA = cur[pos + TS]; hC = cur[N + pos + TS]; hD = cur[2 * N + pos + TS]; }
      const R e0A = eA, e0C = eC, e0D = eD;
      pcr_row(eA, eC, eD, lA, lC, lD, oA, oC, oD);
      pcr_row(oA, oC, oD, e0A, e0C, e0D, hA, hC, hD);
    }
    bool more = true;
#pragma unroll 1
    for (int h = 1; h < G; h <<= 1) {
      R* t = cur; cur = nxt; nxt = t;
      if (active) {
        cur[pos] = eA; cur[N + pos] = eC; cur[2 * N + pos] = eD;
        cur[3 * N + pos] = oA; cur[4 * N + pos] = oC; cur[5 * N + pos] = oD;
      }
      if (!sync(active && more)) break;
      R lA = R(0), lC = R(0), lD = R(0), hA = R(0), hC = R(0), hD = R(0);
      R mA = R(0), mC = R(0), mD = R(0), gA = R(0), gC = R(0), gD = R(0);
      if (active && k >= h) {
        const int q = pos - h * TS;
        lA = cur[q]; lC = cur[N + q]; lD = cur[2 * N + q];
        mA = cur[3 * N + q]; mC = cur[4 * N + q]; mD = cur[5 * N + q];
      }
      if (active && k + h < G) {
        const int q = pos + h * TS;
        hA = cur[q]; hC = cur[N + q]; hD = cur[2 * N + q];
        gA = cur[3 * N + q]; gC = cur[4 * N + q]; gD = cur[5 * N + q];
      }
      more = pcr_more(eA, eC, eD, lD, hD) || pcr_more(oA, oC, oD, mD, gD);
      pcr_row(eA, eC, eD, lA, lC, lD, hA, hC, hD);
      pcr_row(oA, oC, oD, mA, mC, mD, gA, gC, gD);
    }
    x0 = eD;
    xl = oD;
  }
}

// One chunk of M >= 3 rows in registers, eliminated to its first and last
// rows (modified Thomas) and back-substituted once their solutions are
// known; the operations of chunk_solve in its order.
template <class R, int M>
struct Chunk {
  R a[M], b[M], c[M], d[M];
  R eA, eC, eD, oA, oC, oD;
  __device__ __forceinline__ void eliminate() {
    const R inv = fast_rcp(b[1]);
    R ap = a[1] * inv, cp = c[1] * inv, dp = d[1] * inv;
    a[1] = ap; c[1] = cp; d[1] = dp;
#pragma unroll
    for (int i = 2; i < M; ++i) {
      const R ai = a[i];
      const R r = fast_rcp(fmaT(-ai, cp, b[i]));
      ap = -ai * ap * r;
      dp = fmaT(-ai, dp, d[i]) * r;
      cp = c[i] * r;
      a[i] = ap; c[i] = cp; d[i] = dp;
    }
    R an = a[M - 2], cn = c[M - 2], dn = d[M - 2];
#pragma unroll
    for (int i = M - 3; i >= 1; --i) {
      const R ci = c[i];
      dn = fmaT(-ci, dn, d[i]);
      an = fmaT(-ci, an, a[i]);
      cn = -ci * cn;
      a[i] = an; c[i] = cn; d[i] = dn;
    }
    const R r0 = fast_rcp(fmaT(-c[0], an, b[0]));
    eA = a[0] * r0; eC = -c[0] * cn * r0; eD = fmaT(-c[0], dn, d[0]) * r0;
    oA = ap; oC = cp; oD = dp;
  }
  // the solution replaces d
  __device__ __forceinline__ void substitute(R x0, R xl) {
    d[0] = x0;
#pragma unroll
    for (int i = 1; i < M - 1; ++i) d[i] = fmaT(-c[i], xl, fmaT(-a[i], x0, d[i]));
    d[M - 1] = xl;
  }
};

// Partitioned line solve of the TL lines staged in shared memory, G threads
// per line (thread t: line t / G, chunk k = t % G, rows k*m .. k*m+m-1 at
// offset k*mp of the line's row arrays).  Every thread eliminates its chunk
// (m >= 3 rows) down to two rows coupled only to the neighbouring chunks'
// end rows (a forward and a backward "modified Thomas" sweep), in registers
// when the chunk is compile-time (M > 0); the 2G reduced rows of each line
// are then solved by reduced_pcr, and every thread back-substitutes its
// chunk.  This is the Thomas-PCR hybrid of Laszlo, Giles and Appleyard (ACM
// TOMS 42(4), 2016).  Reciprocals use fast_rcp (two Newton steps).  The
// solution replaces the right-hand side.  Called by all TL*G threads;
// threads of lines with `active` false only take part in the barriers.
// ALIAS (compile-time chunk): the reduced system takes the place of the
// coefficients, which are in registers by then; it ends before the
// right-hand sides (binary64 keeps 9G of it, binary32 12G, the first three
// row arrays hold 3*G*mp).
template <class R, int M>
__host__ __device__ constexpr bool chunk_alias() { return M > 0 && (sizeof(R) == 8 ? 3 : 4) <= (M | 1); }
template <class R, int G, int TL = 1, int M = 0, bool ALIAS = false>
__device__ __forceinline__ void chunk_solve(R* line, int m, int mp, bool active) {
  const int k = threadIdx.x % G;
  constexpr bool HALF = sizeof(R) == 8;
  R* a = line + k * mp;
  R* b = a + (size_t)G * mp;
  R* c = b + (size_t)G * mp;
  R* d = c + (size_t)G * mp;
  static_assert(!ALIAS || chunk_alias<R, M>(), "the reduced system would reach the right-hand sides");
  R* red = line + (ALIAS ? (size_t)0 : (size_t)4 * G * mp);
  R x0, xl;
  if constexpr (M > 0) {
    Chunk<R, M> ch;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      ch.a[i] = R(0); ch.b[i] = R(1); ch.c[i] = R(0); ch.d[i] = R(0);
      if (active) { ch.a[i] = a[i]; ch.b[i] = b[i]; ch.c[i] = c[i]; ch.d[i] = d[i]; }
    }
    ch.eliminate();
    if constexpr (ALIAS) line_sync<G, TL>(false);  // every chunk is in registers
    reduced_pcr<R, HALF>(red, G, 1, G, k, k, active, ch.eA, ch.eC, ch.eD, ch.oA, ch.oC, ch.oD, x0, xl,
                         [](bool q) { return line_sync<G, TL>(q); });
    if (active) {
      ch.substitute(x0, xl);
#pragma unroll
      for (int i = 0; i < M; ++i) d[i] = ch.d[i];
    }
  } else {
    R eA = R(0), eC = R(0), eD = R(0), oA = R(0), oC = R(0), oD = R(0);
    if (active) {
      // forward: rows 1..m-1 -> x_k + a'_k x_0 + c'_k x_{k+1} = d'_k
      const R a0 = a[0], b0 = b[0], c0 = c[0], d0 = d[0];
      const R inv = fast_rcp(b[1]);
      R ap = a[1] * inv, cp = c[1] * inv, dp = d[1] * inv;
      a[1] = ap; c[1] = cp; d[1] = dp;
      for (int i = 2; i < m; ++i) {
        const R ai = a[i];
        const R r = fast_rcp(fmaT(-ai, cp, b[i]));
        ap = -ai * ap * r;
        dp = fmaT(-ai, dp, d[i]) * r;
        cp = c[i] * r;
        a[i] = ap; c[i] = cp; d[i] = dp;
      }
      // backward: rows m-3..1 -> x_i + a''_i x_0 + c''_i x_{m-1} = d''_i
      R an = a[m - 2], cn = c[m - 2], dn = d[m - 2];
      for (int i = m - 3; i >= 1; --i) {
        const R ci = c[i];
        dn = fmaT(-ci, dn, d[i]);
        an = fmaT(-ci, an, a[i]);
        cn = -ci * cn;
        a[i] = an; c[i] = cn; d[i] = dn;
      }
      // reduced rows 2k (chunk's first row) and 2k+1 (its last row), unit diagonal
      const R r0 = fast_rcp(fmaT(-c0, an, b0));
      eA = a0 * r0; eC = -c0 * cn * r0; eD = fmaT(-c0, dn, d0) * r0;
      oA = ap; oC = cp; oD = dp;
    }
    reduced_pcr<R, HALF>(red, G, 1, G, k, k, active, eA, eC, eD, oA, oC, oD, x0, xl, [](bool q) { return line_sync<G, TL>(q); });
    if (active) {
      d[0] = x0;
      for (int i = 1; i < m - 1; ++i) d[i] = fmaT(-c[i], xl, fmaT(-a[i], x0, d[i]));
      d[m - 1] = xl;
    }
  }
}

}  // namespace ixb
