// FP64 radial ODE solver of the FK hot path: one (omega, l) item per thread.
//
// The arithmetic of every step restates the reference (file:line cited per
// function) in the same operation order; the control structure is the
// GPU's own:
//   * system matrices are evaluated at each modified-midpoint sub-step instead
//     of being cached on the 1/48 grid (same values, no per-thread cache); the
//     fast build shares them between the two attempts of a pair;
//   * matrix-vector products skip the structural zeros of each system (adding
//     a zero product leaves a sum unchanged);
//   * results at nodes go to a per-thread scratch slot laid out
//     element-major across threads, so a warp's stores coalesce;
//   * a warp integrates its 32 items in lockstep (see fk_kernel.cu);
//   * the spheroidal adjoint is integrated only for the unit jumps whose
//     Green functions reach a stored component (jumps 2 and 4 without
//     stresses), and only as far as the last node it feeds.
#pragma once
#include "gem_device.cuh"
#include "fk_types.cuh"

// Compiled twice: GEM_NS = gem_plain (GEM_FAST 0, built with --fmad=false, the
// parity path) and GEM_NS = gem_fast (GEM_FAST 1, FMA contraction, division-free
// spline evaluation, reciprocal-based complex inverses).
#ifndef GEM_NS
#error "define GEM_NS and GEM_FAST before including fk_solver.cuh"
#endif

namespace GEM_NS {
namespace {   // one copy per translation unit
using namespace gem;

// Bulirsch-Stoer subdivision scheme (parametersBulirschStep.f90:28-48)
__device__ __constant__ const int SEQDIV[7] = {2, 4, 6, 8, 12, 16, 24};
__device__ __constant__ const int NXDIV[7] = {3, 2, 4, 4, 4, 8, 8};
// flop weights of one system-matrix evaluation (incl. spline) and of one
// midpoint matrix-vector update, per ODE system (minors, fluid, radial,
// toroidal, adjoint); identical to the oracle's accounting.
__device__ __constant__ const int FLOP_SYSMAT[5] = {230, 150, 175, 140, 215};
__device__ __constant__ const int FLOP_MV[5] = {8 * 19 + 4 * 5, 8 * 3 + 4 * 2, 8 * 4 + 4 * 2,
                                               8 * 4 + 4 * 2, 8 * 14 + 4 * 4};

// ------------------------------------------------------------------------
//  locate (locatePoint.f90:72-101), 1-based x in the parameter block
// ------------------------------------------------------------------------
__device__ __forceinline__ int locate(double xx, int n, const double* x) {
  int lidx = 0, ridx = n + 1;
  bool asc = x[n] > x[1];
  while (ridx - lidx > 1) {
    int midx = (lidx + ridx) >> 1;
    bool gt = xx > x[midx];
    if (asc) { if (gt) lidx = midx; else ridx = midx; }
    else { if (gt) ridx = midx; else lidx = midx; }
  }
  return lidx;
}

// getLayerIndexNodeEarthmodel (nodeEarthmodel.f90:599-607)
__device__ __forceinline__ void layer_index(const FKStatic& P, double r, int& nl, int& top) {
  nl = locate(r, P.nlay, P.rb) + 1;
  int nlc = nl < P.nlay ? nl : P.nlay;
  top = fabs(r / P.rb[nlc] - 1.0) < EPS_D ? 1 : 0;
}

// ------------------------------------------------------------------------
//  Spline evaluation (splineEarthmodelCoefficients.f90:118-162).
//  MASK selects the elastic constants (bit c -> constant c of A,C,F,L,N,K,M).
// ------------------------------------------------------------------------
#if GEM_FAST
// values at t of the cubics of one knot interval: density and the constants of MASK
template <unsigned MASK>
__device__ __forceinline__ void horner_spline(const double* __restrict__ q, double t, double& ro, dz* el) {
  auto horner = [&](int v) {
    double2 c32 = __ldg(reinterpret_cast<const double2*>(q + 4 * v));
    double2 c10 = __ldg(reinterpret_cast<const double2*>(q + 4 * v + 2));
    return fma(fma(fma(c32.x, t, c32.y), t, c10.x), t, c10.y);
  };
  ro = horner(0);
#pragma unroll
  for (int c = 0; c < 7; ++c)
    if (MASK & (1u << c)) el[c] = dz{horner(poly_value(c)), horner(poly_value(c) + 1)};
}
#endif
template <unsigned MASK>
__device__ __forceinline__ void eval_spline(const FKStatic& P, const Env& e, double r, int nl, double& ro,
                                            dz* el) {
  const Tab* __restrict__ T = e.tab;
#if GEM_FAST
  {
    // cubic in t = r - rk(j) per knot interval, Horner form (no divisions)
    int j;
    double t;
    if (nl == 1) {
      j = T->iktop[1];
      t = 0.0;
    } else {
      int j1 = T->iktop[nl - 1] + 1, j2 = T->iktop[nl];
      if (j2 - j1 == 1) {
        j = j1;
      } else if (P.equidis == 1) {
        j = (int)((r - T->rk[j1]) * T->rdrk[nl]) + j1;
        j = j < j1 ? j1 : (j > j2 - 1 ? j2 - 1 : j);
      } else {
        j = j1 - 1;
        int jr = j2 + 1;
        while (jr - j > 1) {
          int m = (j + jr) >> 1;
          if (r > T->rk[m]) j = m; else jr = m;
        }
        if (j == j1 - 1) j = j1;
      }
      j = j < 1 ? 1 : (j > P.nk - 1 ? P.nk - 1 : j);
      t = r - T->rk[j];
    }
    horner_spline<MASK>(e.poly + (long long)j * POLY_STRIDE, t, ro, el);
    return;
  }
#endif
  const double* __restrict__ spl = e.spl;
  // One code path for every layer, so lanes of a warp stay converged:
  //  * layer 1 (homogeneous sphere) reads knot iktop(1) with weights (1,0,0,0);
  //  * two-knot layers use the cubic formula with their zero second
  //    derivatives, which adds exact zeros to the linear interpolant.
  int j;
  double a, b, cc, dd;
  if (nl == 1) {
    j = T->iktop[1];
    a = 1.0; b = 0.0; cc = 0.0; dd = 0.0;
  } else {
    int j1 = T->iktop[nl - 1] + 1, j2 = T->iktop[nl];
    if (j2 - j1 == 1) {
      j = j1;
    } else if (P.equidis == 1) {
      j = (int)((r - T->rk[j1]) / T->drk[nl]) + j1;
      if (j == j2) j = j2 - 1;
    } else {
      j = j1 - 1;
      int jr = j2 + 1;
      while (jr - j > 1) {
        int m = (j + jr) >> 1;
        if (r > T->rk[m]) j = m; else jr = m;
      }
      if (j == j1 - 1) j = j1;
    }
    j = j < 1 ? 1 : (j > P.nk - 1 ? P.nk - 1 : j);   // memory guard (in-range inputs unaffected)
    double x1 = T->rk[j], x2 = T->rk[j + 1], h = x2 - x1;
    a = (x2 - r) / h;
    b = 1.0 - a;
    cc = h * h * a * (a * a - 1.0) / 6.0;
    dd = h * h * b * (b * b - 1.0) / 6.0;
  }
  const double* t1 = spl + j * SPL_STRIDE;
  const double* t2 = t1 + SPL_STRIDE;
  ro = a * __ldg(t1) + b * __ldg(t2) + cc * __ldg(t1 + 1) + dd * __ldg(t2 + 1);
#pragma unroll
  for (int c = 0; c < 7; ++c)
    if (MASK & (1u << c)) {
      double2 e1 = __ldg(reinterpret_cast<const double2*>(t1 + 2 + 2 * c));
      double2 e2 = __ldg(reinterpret_cast<const double2*>(t2 + 2 + 2 * c));
      double2 s1 = __ldg(reinterpret_cast<const double2*>(t1 + 16 + 2 * c));
      double2 s2 = __ldg(reinterpret_cast<const double2*>(t2 + 16 + 2 * c));
      el[c] = a * dz{e1.x, e1.y} + b * dz{e2.x, e2.y} + cc * dz{s1.x, s1.y} + dd * dz{s2.x, s2.y};
    }
}

#if GEM_FAST
// The environment of one Bulirsch-Stoer step (fast build): the knot intervals
// jlo..jhi of the step's two ends are looked up once per step.  A step is a
// fraction of a wavelength and mostly stays in one interval or crosses one
// knot, so a sub-step finds its interval by one comparison with the knot above
// jlo; a search runs only while a lane of the warp steps over several knots
// (wide).  The interval is the last one of jlo..jhi whose lower bound kb is not
// above r (kb: the knots, or with equidistant knots their regular grid, which
// gives the interval int((r - rk(j1)) / drk) of eval_spline).
struct EnvF : Env {
  int jlo, jhi;
  bool wide;               // a lane of the warp spans more than two intervals
  double kb1, rk0, rk1;    // kb(jlo+1) (infinite when jlo = jhi), rk(jlo), rk(jlo+1)
};
// last interval j of j1..j2 with kb(j) <= r (j1 when there is none), searched
// from j: a solve's steps move through the intervals one by one
__device__ __forceinline__ int knot_interval(const double* __restrict__ kb, int j1, int j2, double r, int j) {
  j = max(j1, min(j, j2));
  while (j < j2 && kb[j + 1] <= r) ++j;
  while (j > j1 && kb[j] > r) --j;
  return j;
}
// jknot: interval of the solve's last step (any value gives the same result).
// Lanes without a step (active false) may hold no layer yet (a lane that never
// took an item): they read the tables of layer 1 and evaluate nothing.
__device__ __forceinline__ EnvF make_envf(const FKStatic& P, const Env& e, bool active, double xa, double xb, int& jknot) {
  EnvF f;
  static_cast<Env&>(f) = e;
  const Tab* __restrict__ T = e.tab;
  const int nl = (active && e.nl >= 1 && e.nl <= P.nlay) ? e.nl : 1;
  if (nl == 1) {   // the homogeneous sphere: the constant cubic of its knot
    f.jlo = f.jhi = T->iktop[1];
  } else {
    const int j1 = min(max(T->iktop[nl - 1] + 1, 1), P.nk - 1), j2 = min(T->iktop[nl] - 1, P.nk - 1);
    f.jlo = knot_interval(T->kb, j1, max(j1, j2), fmin(xa, xb), jknot);
    f.jhi = knot_interval(T->kb, f.jlo, max(f.jlo, j2), fmax(xa, xb), f.jlo);
    jknot = f.jlo;
  }
  f.rk0 = T->rk[f.jlo];
  f.rk1 = T->rk[f.jlo + 1];
  f.kb1 = f.jhi > f.jlo ? T->kb[f.jlo + 1] : __longlong_as_double(0x7ff0000000000000LL);
  f.wide = __any_sync(0xffffffffu, active && f.jhi > f.jlo + 1);
  return f;
}
// cubics and argument of the spline at r
__device__ __forceinline__ const double* spline_at(const EnvF& e, double r, double& t) {
  const bool up = r >= e.kb1;
  int j = up ? e.jlo + 1 : e.jlo;
  double rk = up ? e.rk1 : e.rk0;
  if (e.wide) {
    const Tab* __restrict__ T = e.tab;
    while (j < e.jhi && r >= T->kb[j + 1]) ++j;
    rk = T->rk[j];
  }
  t = r - rk;
  return e.poly + j * POLY_STRIDE;
}
#endif

// ------------------------------------------------------------------------
//  ODE systems: y = A(x) z, nonzero entries only, column order as matmul
// ------------------------------------------------------------------------
enum { SYS_MINORS = 0, SYS_FLUID = 1, SYS_RADIAL = 2, SYS_TOROIDAL = 3, SYS_SOLIDT = 4 };
template <int SYS> struct SysNV;
template <> struct SysNV<SYS_MINORS> { static constexpr int NV = 5; };
template <> struct SysNV<SYS_FLUID> { static constexpr int NV = 2; };
template <> struct SysNV<SYS_RADIAL> { static constexpr int NV = 2; };
template <> struct SysNV<SYS_TOROIDAL> { static constexpr int NV = 2; };
template <> struct SysNV<SYS_SOLIDT> { static constexpr int NV = 4; };

// 1/x and 1/z: divisions (Smith's for z) on the parity path.  The fast path
// takes one reciprocal without a branch: the PTX approximation (20 bits, rel.
// error d) and one third-order Newton (Householder) update r (1 + d + d^2),
// whose error d^3 is below the rounding.  A correctly rounded reciprocal has a
// slow path behind a branch, which keeps the compiler from overlapping the
// evaluations of a step.
__device__ __forceinline__ double rinv(double x) {
#if GEM_FAST
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double d = fma(-x, r, 1.0);
  return fma(r, fma(d, d, d), r);
#else
  return 1.0 / x;
#endif
}
__device__ __forceinline__ dz zinv(dz z) {
#if GEM_FAST
  const double r = rinv(fma(z.re, z.re, __dmul_rn(z.im, z.im)));
  return {z.re * r, -z.im * r};
#else
  return 1.0 / z;
#endif
}

#if GEM_FAST
// acc + a b, four FMAs for a complex factor
__device__ __forceinline__ void cfma(dz& acc, dz a, dz b) {
  acc.re = fma(a.re, b.re, fma(-a.im, b.im, acc.re));
  acc.im = fma(a.re, b.im, fma(a.im, b.re, acc.im));
}
__device__ __forceinline__ void cfma(dz& acc, double a, dz b) {
  acc.re = fma(a, b.re, acc.re);
  acc.im = fma(a, b.im, acc.im);
}
__device__ __forceinline__ dz cmul(dz a, dz b) {
  return {fma(a.re, b.re, -__dmul_rn(a.im, b.im)), fma(a.re, b.im, __dmul_rn(a.im, b.re))};
}

// Matrix entries of the fast build.  Products and sums are written so that the
// compiler has no choice in contracting them (fma, or the _rn products): the
// thread form and the group form of a step give the same bits.
template <int SYS> struct SysE;
template <> struct SysE<SYS_MINORS> { dz a, m12, m14, m23, m24, m32, m42, z4; double m11, m13, m22, m33, m55; };
template <> struct SysE<SYS_FLUID> { dz m12, m21; double m11; };
template <> struct SysE<SYS_RADIAL> { dz m11, m12, m21, m22; };
template <> struct SysE<SYS_TOROIDAL> { dz m12, m21; double rr; };
template <> struct SysE<SYS_SOLIDT> { dz a11, a12, a14, z2, zrpc, a31, a32, a34, a43; double rr, a22, a42; };

// A(x) from the cubics q at t.  ISO (every knot of the model isotropic:
// A = C, N = L, F = C - 2 L): with m = L/C, A - F^2/C - N = L (3 - 4 m) and
// F/C = 1 - 2 m, so only the density, C and L are evaluated (5 cubics instead
// of 11).  zom2 = (omega - i sigma)^2.
template <int SYS, bool ISO>
__device__ __forceinline__ void sys_eval(const EnvF& e, dz zom2, const double* __restrict__ q, double t, double x,
                                         SysE<SYS>& E) {
  double ro;
  dz el[7];
  const double dll1 = e.dll1;
  auto scale = [](double a, dz z) { return dz{__dmul_rn(a, z.re), __dmul_rn(a, z.im)}; };
  if constexpr (SYS == SYS_MINORS || SYS == SYS_SOLIDT) {   // minorsOdeSystem.f90:77-126, solidtOdeSystem.f90:77-114
    horner_spline<ISO ? 0x0Au : 0x1Fu>(q, t, ro, el);
    const double rr = rinv(x), rr2 = __dmul_rn(rr, rr);
    const dz zrpc = zinv(el[1]), zom = scale(ro, zom2), rl = zinv(el[3]);
    dz z1, fc, n;   // A - F^2/C - N, F/C, N
    if constexpr (ISO) {
      const dz m = cmul(el[3], zrpc);
      n = el[3];
      z1 = cmul(n, dz{fma(-4.0, m.re, 3.0), -4.0 * m.im});
      fc = dz{fma(-2.0, m.re, 1.0), -2.0 * m.im};
    } else {
      n = el[4];
      fc = cmul(el[2], zrpc);
      z1 = el[0] - n;
      cfma(z1, -el[2], fc);
    }
    const dz z = scale(rr2, z1), c = scale(rr2, n);
    if constexpr (SYS == SYS_MINORS) {
      E.a = scale(2.0 * rr, fc);
      E.m11 = -2.0 * rr;
      E.m13 = __dmul_rn(dll1, rr);
      E.m12 = scale(-2.0 * dll1, z);
      E.m14 = scale(-0.5 * dll1, E.a);
      E.m22 = __dsub_rn(rr, E.a.re);     // the imaginary parts of m22, m33, m55 are -a, -a, +a
      E.m33 = fma(-3.0, rr, -E.a.re);
      E.m55 = fma(-5.0, rr, E.a.re);
      E.m23 = rl;
      E.m24 = zrpc;
      E.z4 = dz{4.0 * z.re, 4.0 * z.im};
      E.m42 = dz{__dsub_rn(E.z4.re, zom.re), __dsub_rn(E.z4.im, zom.im)};
      E.m32 = dz{fma(dll1, z.re, fma(dll1 - 2.0, c.re, -zom.re)), fma(dll1, z.im, fma(dll1 - 2.0, c.im, -zom.im))};
    } else {
      E.rr = rr;
      E.z2 = scale(rr, fc);
      E.zrpc = -zrpc;
      E.a43 = -rl;
      E.a11 = dz{2.0 * E.z2.re, 2.0 * E.z2.im};
      E.a12 = dz{fma(-4.0, z.re, zom.re), fma(-4.0, z.im, zom.im)};
      E.a14 = dz{2.0 * z.re, 2.0 * z.im};
      E.a22 = fma(2.0, rr, -E.a11.re);   // its imaginary part is -a11
      E.a31 = scale(-dll1, E.z2);
      E.a32 = scale(2.0 * dll1, z);
      E.a34 = dz{fma(-dll1, z.re, fma(2.0 - dll1, c.re, zom.re)), fma(-dll1, z.im, fma(2.0 - dll1, c.im, zom.im))};
      E.a42 = __dmul_rn(-dll1, rr);
    }
  } else if constexpr (SYS == SYS_FLUID) {   // fluidOdeSystem.f90:78-95
    horner_spline<0x02u>(q, t, ro, el);
    const dz zomro = scale(ro, zom2);
    const dz k = zinv(el[1]), g = zinv(scale(__dmul_rn(x, x), zomro));
    E.m11 = -2.0 * rinv(x);
    E.m12 = dz{fma(-dll1, g.re, k.re), fma(-dll1, g.im, k.im)};
    E.m21 = -zomro;
  } else if constexpr (SYS == SYS_RADIAL) {  // radialOdeSystem.f90:78-99
    horner_spline<ISO ? 0x0Au : 0x17u>(q, t, ro, el);
    if constexpr (ISO) {
      el[0] = el[1]; el[4] = el[3];
      el[2] = dz{fma(-2.0, el[3].re, el[1].re), fma(-2.0, el[3].im, el[1].im)};
    }
    const dz zomro = scale(ro, zom2);
    const double rr = rinv(x), rr2 = __dmul_rn(rr, rr);
    const dz rc = zinv(el[1]), fc = cmul(el[2], rc);
    dz z1 = el[0] - el[4];   // A - F^2/C - N
    cfma(z1, -el[2], fc);
    E.m11 = scale(-2.0 * rr, fc);
    E.m12 = rc;
    E.m21 = dz{fma(4.0 * rr2, z1.re, -zomro.re), fma(4.0 * rr2, z1.im, -zomro.im)};
    E.m22 = scale(2.0 * rr, dz{__dsub_rn(fc.re, 1.0), fc.im});
  } else {                                   // toroidalOdeSystem.f90:81-102
    horner_spline<ISO ? 0x08u : 0x18u>(q, t, ro, el);
    const dz zom = scale(ro, zom2);
    const double rr = rinv(x), k = __dmul_rn(dll1 - 2.0, __dmul_rn(rr, rr));
    const dz n = el[ISO ? 3 : 4];
    E.m12 = zinv(el[3]);
    E.m21 = dz{fma(n.re, k, -zom.re), fma(n.im, k, -zom.im)};
    E.rr = rr;
  }
}

// acc += E z
template <int SYS>
__device__ __forceinline__ void sys_mul(const SysE<SYS>& E, const dz* z, dz* acc) {
  if constexpr (SYS == SYS_MINORS) {
    const dz m22{E.m22, -E.a.im}, m33{E.m33, -E.a.im}, m55{E.m55, E.a.im};
    cfma(acc[0], E.m11, z[0]); cfma(acc[1], m22, z[1]); cfma(acc[2], -E.a, z[0]); cfma(acc[3], -E.m11, z[0]); cfma(acc[4], E.z4, z[0]);
    cfma(acc[0], E.m12, z[1]); cfma(acc[1], E.m23, z[2]); cfma(acc[2], E.m32, z[1]); cfma(acc[3], E.m42, z[1]); cfma(acc[4], E.m42, z[2]);
    cfma(acc[0], E.m13, z[2]); cfma(acc[1], E.m24, z[3]); cfma(acc[2], m33, z[2]); cfma(acc[3], -m22, z[3]); cfma(acc[4], E.m32, z[3]);
    cfma(acc[0], E.m14, z[3]); cfma(acc[2], E.m24, z[4]); cfma(acc[3], E.m23, z[4]); cfma(acc[4], m55, z[4]);
  } else if constexpr (SYS == SYS_FLUID) {
    cfma(acc[0], E.m11, z[0]); cfma(acc[1], E.m21, z[0]);
    cfma(acc[0], E.m12, z[1]);
  } else if constexpr (SYS == SYS_RADIAL) {
    cfma(acc[0], E.m11, z[0]); cfma(acc[1], E.m21, z[0]);
    cfma(acc[0], E.m12, z[1]); cfma(acc[1], E.m22, z[1]);
  } else if constexpr (SYS == SYS_TOROIDAL) {
    cfma(acc[0], E.rr, z[0]); cfma(acc[1], E.m21, z[0]);
    cfma(acc[0], E.m12, z[1]); cfma(acc[1], -3.0 * E.rr, z[1]);
  } else {
    const dz a22{E.a22, -E.a11.im};
    cfma(acc[0], E.a11, z[0]); cfma(acc[1], E.zrpc, z[0]); cfma(acc[2], E.a31, z[0]); cfma(acc[3], E.a42, z[1]);
    cfma(acc[0], E.a12, z[1]); cfma(acc[1], a22, z[1]); cfma(acc[2], E.a32, z[1]); cfma(acc[3], E.a43, z[2]);
    cfma(acc[0], E.rr, z[2]); cfma(acc[1], E.z2, z[3]); cfma(acc[2], -E.rr, z[2]); cfma(acc[3], 3.0 * E.rr, z[3]);
    cfma(acc[0], E.a14, z[3]); cfma(acc[2], E.a34, z[3]);
  }
}

template <int SYS, bool ISO>
__device__ __forceinline__ void sys_at(const EnvF& e, dz zom2, double x, SysE<SYS>& E) {
  double t;
  const double* q = spline_at(e, x, t);
  sys_eval<SYS, ISO>(e, zom2, q, t, x, E);
}
#else
template <int SYS>
__device__ __forceinline__ void apply_sys(const FKStatic& P, const Env& e, double x, const dz* z, dz* y) {
  double ro;
  dz el[7];
  dz zom{e.omre, e.omim};
  double dll1 = e.dll1;
  if (SYS == SYS_MINORS) {          // minorsOdeSystem.f90:77-126
    eval_spline<0x1Fu>(P, e, x, e.nl, ro, el);
    dz zomro = zom * zom * ro;
    double rr = rinv(x), rr2 = rr * rr;
    dz zrpc = zinv(el[1]);
    dz z1 = el[0] - (el[2] * el[2]) * zrpc - el[4];
    dz z2 = (2.0 * el[2]) * zrpc;
    dz z3 = (4.0 * z1) * rr2;
    double m11 = -2.0 * rr;
    dz m12 = ((-2.0 * dll1) * z1) * rr2;
    double m13 = dll1 * rr;
    dz m14 = (((-dll1) * el[2]) * zrpc) * rr;
    dz m22 = (1.0 - z2) * rr;
    dz m23 = zinv(el[3]);
    dz m24 = zrpc;
    dz m31 = (-z2) * rr;
    dz m32 = (-zomro) + ((dll1 * (z1 + el[4])) - 2.0 * el[4]) * rr2;
    dz m33 = (-(3.0 + z2)) * rr;
    double m41 = -m11;
    dz m42 = (-zomro) + z3;
    dz m55 = (z2 - 5.0) * rr;
    y[0] = m11 * z[0] + m12 * z[1] + m13 * z[2] + m14 * z[3];
    y[1] = m22 * z[1] + m23 * z[2] + m24 * z[3];
    y[2] = m31 * z[0] + m32 * z[1] + m33 * z[2] + m24 * z[4];
    y[3] = m41 * z[0] + m42 * z[1] + (-m22) * z[3] + m23 * z[4];
    y[4] = z3 * z[0] + m42 * z[2] + m32 * z[3] + m55 * z[4];
  } else if (SYS == SYS_FLUID) {    // fluidOdeSystem.f90:78-95
    eval_spline<0x02u>(P, e, x, e.nl, ro, el);
    dz zomro = zom * zom * ro;
    double m11 = -2.0 / x;
    dz m12 = 1.0 / el[1] - dll1 / ((zomro * x) * x);
    y[0] = m11 * z[0] + m12 * z[1];
    y[1] = (-zomro) * z[0];
  } else if (SYS == SYS_RADIAL) {   // radialOdeSystem.f90:78-99
    eval_spline<0x17u>(P, e, x, e.nl, ro, el);
    dz zomro = zom * zom * ro;
    double rr = rinv(x), rr2 = rr * rr;
    dz m11 = ((-2.0 * el[2]) * rr) / el[1];
    dz m12 = 1.0 / el[1];
    dz m21 = (-zomro) + (4.0 * rr2) * ((el[0] - (el[2] * el[2]) / el[1]) - el[4]);
    dz m22 = (2.0 * rr) * (el[2] / el[1] - 1.0);
    y[0] = m11 * z[0] + m12 * z[1];
    y[1] = m21 * z[0] + m22 * z[1];
  } else if (SYS == SYS_TOROIDAL) { // toroidalOdeSystem.f90:81-102
    eval_spline<0x18u>(P, e, x, e.nl, ro, el);
    dz zomro = zom * zom * ro;
    double rr = rinv(x), rr2 = rr * rr;
    dz m12 = zinv(el[3]);
    dz m21 = (-zomro) - (el[4] * rr2) * (2.0 - dll1);
    y[0] = rr * z[0] + m12 * z[1];
    y[1] = m21 * z[0] + (-3.0 * rr) * z[1];
  } else {                          // solidtOdeSystem.f90:77-114
    eval_spline<0x1Fu>(P, e, x, e.nl, ro, el);
    dz zomro = zom * zom * ro;
    double rr = rinv(x), rr2 = rr * rr;
    dz zrpc = zinv(el[1]);
    dz z1 = el[0] - (el[2] * el[2]) * zrpc - el[4];
    dz z2 = (el[2] * rr) * zrpc;
    dz zdlz1 = dll1 * z1;
    dz a11 = 2.0 * z2;
    dz a21 = -zrpc;
    dz a31 = (-dll1) * z2;
    dz a12 = zomro - (4.0 * z1) * rr2;
    dz a22 = (-a11) + 2.0 * rr;
    dz a32 = (2.0 * rr2) * zdlz1;
    double a42 = (-dll1) * rr;
    dz a43 = -zinv(el[3]);
    dz a14 = (2.0 * z1) * rr2;
    dz a34 = zomro - (zdlz1 + (dll1 - 2.0) * el[4]) * rr2;
    y[0] = a11 * z[0] + a12 * z[1] + rr * z[2] + a14 * z[3];
    y[1] = a21 * z[0] + a22 * z[1] + z2 * z[3];
    y[2] = a31 * z[0] + a32 * z[1] + (-rr) * z[2] + a34 * z[3];
    y[3] = a42 * z[1] + a43 * z[2] + (3.0 * rr) * z[3];
  }
}
#endif

// ------------------------------------------------------------------------
//  Bulirsch-Stoer full step (complexBulirschStep.f90:111-240,297-340)
// ------------------------------------------------------------------------
#if GEM_FAST
// Extrapolation of the attempts 1..j to step size 0 by the polynomial through
// (x_i = h / n_i, Y_i): its value is Y_j + sum_{i<j} w_i (Y_i - Y_j) with the
// Lagrange weights w_i = prod_{k != i} n_i / (n_i - n_k), in which h cancels, and
// the last correction of the Neville recursion (the polynomial through all
// attempts minus the one without the first) is sum_{i<j} e_i (Y_i - Y_j),
// e_i = w_i - w_i of the attempts 2..j.  |w_i| <= 39.
struct ExtrapTab {
  double w[8][7], e[8][7];
};
constexpr ExtrapTab make_extrap() {
  const int n[7] = {2, 4, 6, 8, 12, 16, 24};
  ExtrapTab t{};
  for (int j = 2; j <= 7; ++j)
    for (int i = 0; i < j; ++i) {
      double w = 1.0, w1 = 1.0;
      for (int k = 0; k < j; ++k) {
        if (k == i) continue;
        w *= (double)n[i] / (double)(n[i] - n[k]);
        if (k > 0) w1 *= (double)n[i] / (double)(n[i] - n[k]);
      }
      t.w[j][i] = w;
      t.e[j][i] = i == 0 ? w : w - w1;
    }
  return t;
}
__device__ __constant__ const ExtrapTab EXTRAP = make_extrap();

// Modified midpoint of n sub-steps, and with pair the one of n/2 sub-steps
// beside it: its grid is every second point of the finer one, so both share
// the system matrices.  t0 = A(xstart) y0 is given (in memory); the grid point g
// (in 48ths of the step) sits at xstart + g h48, h48 = h / 48 rounded once per step.
// A sub-step z2 = z0 + A (2 hf z1) accumulates into z0.  The last sub-step takes
// half the weight: z_{n-1} + A (hf z_n), whose mean with z_n is the result.
// One evaluation per loop trip: the loop stays small enough for the instruction
// caches (with two per trip, warps waited longer for instructions than for data).
template <int SYS, bool ISO>
__device__ __forceinline__ void midpoint(const EnvF& e, dz zom2, int n, bool pair, double h48, double xstart, const dz* y0,
                                         const Slot& t0, dz* fine, dz* coarse) {
  constexpr int NV = SysNV<SYS>::NV;
  const int dix = 48 / n;
  const double dg = (double)dix, hf = dg * h48;
  dz f0[NV], c0[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const dz y = y0[v], t = t0.get(v);
    f0[v] = c0[v] = fine[v] = coarse[v] = y;
    cfma(fine[v], hf, t);
    cfma(coarse[v], 2.0 * hf, t);
  }
  double g = 0.0;
#pragma unroll 1
  for (int m = 1; m <= n; ++m) {
    g += dg;
    SysE<SYS> E;
    const double w = m == n ? hf : 2.0 * hf;
    sys_at<SYS, ISO>(e, zom2, fma(g, h48, xstart), E);
    dz u[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = w * fine[v];
    sys_mul<SYS>(E, u, f0);
#pragma unroll
    for (int v = 0; v < NV; ++v) { const dz z = f0[v]; f0[v] = fine[v]; fine[v] = z; }
    if (pair && !(m & 1)) {
#pragma unroll
      for (int v = 0; v < NV; ++v) u[v] = (2.0 * w) * coarse[v];
      sys_mul<SYS>(E, u, c0);
#pragma unroll
      for (int v = 0; v < NV; ++v) { const dz z = c0[v]; c0[v] = coarse[v]; coarse[v] = z; }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    fine[v] = 0.5 * (f0[v] + fine[v]);
    coarse[v] = 0.5 * (c0[v] + coarse[v]);
  }
}
#else
template <int SYS>
__device__ __forceinline__ void midpoint(const FKStatic& P, const Env& e, int jtry, double h, double xstart,
                                         const dz* y0, dz* out) {
  constexpr int NV = SysNV<SYS>::NV;
  const int nstep = SEQDIV[jtry - 1];
  const double hdiv = h / (double)nstep;
  const int dix = 48 / nstep;
  dz z0[NV], z1[NV], t[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) z0[v] = y0[v];
  apply_sys<SYS>(P, e, xstart + (0.0 * h) / 48.0, z0, t);
#pragma unroll
  for (int v = 0; v < NV; ++v) z1[v] = z0[v] + hdiv * t[v];
  const double h2 = 2.0 * hdiv;
  for (int m = 1; m <= nstep - 1; ++m) {
    double x = xstart + ((double)(m * dix) * h) / 48.0;
    apply_sys<SYS>(P, e, x, z1, t);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      dz z2 = z0[v] + h2 * t[v];
      z0[v] = z1[v];
      z1[v] = z2;
    }
  }
  apply_sys<SYS>(P, e, xstart + (48.0 * h) / 48.0, z1, t);
#pragma unroll
  for (int v = 0; v < NV; ++v) out[v] = 0.5 * ((z1[v] + z0[v]) + hdiv * t[v]);
}
#endif

// ------------------------------------------------------------------------
//  Nodes and discontinuities inside an integration range
//  (geminiIntegrationEnvironment.f90:96-203); returns index bounds only.
// ------------------------------------------------------------------------
__device__ __forceinline__ void disco_range(const FKStatic& P, double x1, double x2, int& jl, int& jr) {
  double xl = x1, xr = x2;
  if (x1 > x2) { xl = x2; xr = x1; }
  int n = P.nlay;
  jl = locate(xl, n, P.rb) + 1;
  if (jl > n) { jr = jl - 1; return; }
  if (fabs(1.0 - xl / P.rb[jl]) < EPS_D) jl = jl + 1;
  if (jl >= n) { jr = jl - 1; return; }
  jr = locate(xr, n, P.rb);
  if (jr == 0) { jr = 0; jl = 1; }
}

__device__ __forceinline__ void node_range(const FKStatic& P, double x1, double x2, int& jl, int& jr) {
  double xl = x1, xr = x2;
  if (x1 > x2) { xl = x2; xr = x1; }
  int n = P.nnod;
  jl = locate(xl, n, P.rnod) + 1;
  if (jl > n) { jr = jl - 1; return; }
  jr = locate(xr, n, P.rnod);
  if (jr < n) { if (fabs(1.0 - xr / P.rnod[jr + 1]) < EPS_D) jr = jr + 1; }
  if (jr == 0) { jr = 0; jl = 1; }
}

// ------------------------------------------------------------------------
//  Start radius (initialValues.f90:71-192)
// ------------------------------------------------------------------------
__device__ __forceinline__ double velocity_at(const FKStatic& P, const Env& e, double r, int nl) {
  double ro; dz el[7];
  eval_spline<0x60u>(P, e, r, nl, ro, el);
  double v = sqrt(el[6].re / ro);
  if (P.iflso[nl] == 1) v = sqrt(el[5].re / ro);
  return v;
}
__device__ __forceinline__ double vslow(double om, double dll1, double r, double v) {
  return dll1 / (r * r) - (om / v) * (om / v);
}
// The search for the turning radius walks the same radii r_i, r_{i+1} =
// min(r_i + dr, rmax), for every degree of a frequency: start_table_kernel lists
// them with their velocities once per frequency and motion type.
struct StartGrid {
  double r0, dr, rmax, rbot;
  int nl0;
};
__device__ __forceinline__ StartGrid start_grid(const FKStatic& P, bool tor) {
  StartGrid g;
  if (tor && P.hascore) { g.r0 = P.roc; g.nl0 = P.noc + 1; } else { g.r0 = P.rhs; g.nl0 = 1; }
  g.dr = (P.rearth - g.r0) / 400.0;
  g.rmax = (tor && P.hasocean) ? P.ruc : P.rearth;
  g.rbot = (tor && P.hascore) ? P.roc : P.rhs - TENTH_F * g.dr;
  return g;
}
// entry i of the table; r_i is rmax from some i <= 402 on
__device__ __forceinline__ double2 start_entry(const FKStatic& P, const Env& e, const StartGrid& g, int i) {
  double r = g.r0;
  for (int j = 0; j < i; ++j) r = fmin(r + g.dr, g.rmax);
  int nl = g.nl0, top;
  if (i > 0) layer_index(P, r, nl, top);
  return make_double2(r, velocity_at(P, e, r, nl));
}
// integrate the vertical slowness downwards from rturn until its decay reaches
// 1e-5 or the bottom (initialValues.f90:158-192): one warp evaluates 32 radii at
// a time and adds their terms in order
__device__ __forceinline__ double integrate_slowness(const FKStatic& P, const Env& e, const StartGrid& g, double rturn,
                                                     int lane) {
  const double qmax = -log(1.e-5);
  double q = 0.0, r = rturn;
  for (;;) {
    double rl = r, prev = r;
    for (int j = 0; j < 32; ++j)
      if (j <= lane) { prev = rl; rl = rl - g.dr; }
    const bool bottom = prev - g.dr < g.rbot;
    double c = 0.0;
    if (!bottom) {
      int nl, top;
      layer_index(P, rl, nl, top);
      const double v = velocity_at(P, e, rl, nl);
      c = g.dr * sqrt(vslow(e.omre, e.dll1, rl, v));
    }
    const unsigned bm = __ballot_sync(0xffffffffu, bottom);
    for (int l = 0; l < 32; ++l) {
      if (!(q < qmax)) return r;
      if (bm >> l & 1u) return g.rbot;
      r = __shfl_sync(0xffffffffu, rl, l);
      q = q + __shfl_sync(0xffffffffu, c, l);
    }
  }
}
// Start radius of one (omega, l) and motion type, by one warp (initialValues.f90:71-150)
__device__ double start_radius(const FKStatic& P, const Env& e, const StartGrid& g, bool tor,
                               const double2* __restrict__ tab, int lane) {
  double plast = 0.0;   // the value before the current 32
  for (int base = 0; base < START_ENTRIES; base += 32) {
    const double2 rv = tab[base + lane];
    const double p = vslow(e.omre, e.dll1, rv.x, rv.y);
    const bool attop = fabs(1.0 - rv.x / g.rmax) < EPS_D;
    const unsigned m = __ballot_sync(0xffffffffu, !(p > 0.0) || attop);
    if (m) {
      const int l = __ffs(m) - 1;
      const double r = __shfl_sync(0xffffffffu, rv.x, l), pi = __shfl_sync(0xffffffffu, p, l);
      double pold = __shfl_sync(0xffffffffu, p, max(l - 1, 0));
      if (l == 0) pold = plast;
      if (base + l == 0 && !(pi > 0.0)) return (tor && P.hascore) ? P.roc : P.rhs - TENTH_F * g.dr;
      if (pi > 0.0) return integrate_slowness(P, e, g, g.rmax, lane);
      return integrate_slowness(P, e, g, r - g.dr * pi / (pi - pold), lane);
    }
    plast = __shfl_sync(0xffffffffu, p, 31);
  }
  return g.rmax;   // not reached: the table ends at rmax
}

// ------------------------------------------------------------------------
//  Continued fractions (initialValues.f90:487-574)
// ------------------------------------------------------------------------
__device__ int sphancf(dz zx, double el, int kindhf, dz& zf) {
  const double tiny = 1.e-30, eps = 1.e-6;
  zf = dz{tiny, 0.0};
  dz zc = zf, zd{0.0, 0.0};
  double elph2 = (el + 0.5) * (el + 0.5);
  int j;
  for (j = 1; j <= 10000; ++j) {
    dz zb = 2.0 * (zx + dz{0.0, (double)j});
    double za = ((double)j - 0.5) * ((double)j - 0.5) - elph2;
    zd = zb + za * zd;
    if (zabs(zd) < tiny) zd = dz{tiny, 0.0};
    zc = zb + za / zc;
    if (zabs(zc) < tiny) zc = dz{tiny, 0.0};
    zd = 1.0 / zd;
    dz zdelta = zc * zd;
    zf = zf * zdelta;
    if (zabs(zdelta - 1.0) < eps) break;
  }
  if (j > 10000) return ST_CF;
  const dz ci{0.0, 1.0};
  if (kindhf == 1) zf = ((el + 1.0) - ci * zx) - ci * zf;
  else zf = ((el + 1.0) + ci * zx) + ci * zf;
  return ST_OK;
}

__device__ int zetl(dz zx2, double el, dz& z) {
  const double tiny = 1.e-30, eps = 1.e-6;
  z = dz{tiny, 0.0};
  dz zd{2.0 * el + 3.0, 0.0};
  dz zc = zd + zx2 / z;
  zd = 1.0 / zd;
  dz zdelta = zc * zd;
  z = z * zdelta;
  for (int i = 2; i <= 10000; ++i) {
    zd = (2.0 * (el + (double)i) + 1.0) - zx2 * zd;
    if (zd.re == 0.0 && zd.im == 0.0) zd = dz{tiny, 0.0};
    zc = (2.0 * (el + (double)i) + 1.0) - zx2 / zc;
    if (zc.re == 0.0 && zc.im == 0.0) zc = dz{tiny, 0.0};
    zd = 1.0 / zd;
    zdelta = zc * zd;
    z = z * zdelta;
    if (fabs(zabs(zdelta) - 1.0) < eps) return ST_OK;
  }
  return ST_CF;
}

// minors start vector from the ratio functions (initialValues.f90:258-274, 329-346)
__device__ __forceinline__ void minors_from_ratios(bool liquid, double el, double elp1, double r, double ro,
                                                   dz zom, const dz* el7, dz zeta, dz zetb, dz zxb2, dz* ys) {
  if (el < EPS_D) {
    ys[0] = -zeta;
    ys[1] = (((-ro) * r) * zom) * zom + ((4.0 * el7[6]) / r) * zeta;
  } else if (liquid) {
    ys[0] = (-(1.0 - zeta / el)) / (((zom * zom) * ro) * r);
    ys[1] = dz{1.0 / el, 0.0};
  } else {
    dz za = zeta / el;
    dz zb = zetb / (el + 1.0);
    ys[1] = ((-za) + zb * (za - 1.0)) / el;
    dz mr = el7[6] / r;
    ys[0] = mr * (zxb2 / el + (2.0 * elp1) * ys[1]);
    ys[2] = mr * ((-2.0) * ys[1] + (zxb2 / elp1) * (za - 1.0));
    ys[3] = (-mr) * ((zxb2 / (el * el)) * (1.0 - zb) + 4.0 * ys[1]);
    ys[4] = ((el7[6] * el7[6]) / (r * r)) *
            ((((-4.0) * (el - 1.0)) * (el + 2.0)) * ys[1] +
             (zxb2 / el) * ((((zxb2 / elp1) - ((2.0 * (el - 1.0)) * (2.0 * el + 1.0)) / elp1) -
                             (4.0 / (el + 1.0)) * za) - (2.0 / el) * zb));
  }
}

// minorsBottomInitialValues (initialValues.f90:202-275)
__device__ int minors_bottom_iv(const FKStatic& P, const Env& e, double rstart, dz* ys, double& htry) {
  double ro; dz el7[7];
  eval_spline<0x7Fu>(P, e, rstart, e.nl, ro, el7);
  bool liquid = P.iflso[e.nl] == 1;
  double el = -0.5 + sqrt(0.25 + e.dll1);
  double elp1 = e.dll1;
  dz zom{e.omre, e.omim};
  double rsq = rstart * rstart;
  double v = sqrt(el7[6].re / ro);
  if (liquid) v = sqrt(el7[5].re / ro);
  htry = ((0.25 * v) * TWO_PI_F) / e.omre;
  dz zxa2 = (((ro * zom) * zom) * rsq) / (el7[5] + (4.0 * el7[6]) / 3.0);
  dz zeta{0, 0}, zetb{0, 0}, zxb2{0, 0};
  int rc;
  if (el < EPS_D) {
    rc = zetl(zxa2, el, zeta); if (rc) return rc;
  } else {
    if (zabs(zxa2 / elp1) <= 1.0) rc = zetl(zxa2, el, zeta);
    else rc = sphancf(zsqrt(zxa2), el, 1, zeta);
    if (rc) return rc;
    if (!liquid) {
      zxb2 = (((ro * zom) * zom) * rsq) / el7[6];
      if (zabs(zxb2 / elp1) <= 1.0) rc = zetl(zxb2, el, zetb);
      else rc = sphancf(zsqrt(zxb2), el, 1, zetb);
      if (rc) return rc;
    }
  }
  minors_from_ratios(liquid, el, elp1, rstart, ro, zom, el7, zeta, zetb, zxb2, ys);
  return ST_OK;
}

// minorsSurfaceInitialValues (initialValues.f90:287-367)
__device__ int minors_surface_iv(const FKStatic& P, const Env& e, dz* ys, double& htry) {
  int nlay = P.nlay;
  double elp1 = e.dll1;
  double el = -0.5 + sqrt(0.25 + elp1);
  double rearth = P.rearth;
  dz zom{e.omre, e.omim};
  bool liquid = P.iflso[nlay] == 1;
  double ro; dz el7[7];
  eval_spline<0x7Fu>(P, e, rearth, nlay, ro, el7);
  double v = sqrt(el7[6].re / ro);
  if (liquid) v = sqrt(el7[5].re / ro);
  htry = ((0.25 * v) * TWO_PI_F) / e.omre;
  if (P.fsflag == 1) {
    double rsq = rearth * rearth;
    dz zxa2 = (((ro * zom) * zom) * rsq) / (el7[5] + (4.0 * el7[6]) / 3.0);
    dz zeta, zetb{0, 0}, zxb2{0, 0};
    int rc = sphancf(zsqrt(zxa2), el, 2, zeta); if (rc) return rc;
    if (!liquid) {
      zxb2 = (((ro * zom) * zom) * rsq) / el7[6];
      rc = sphancf(zsqrt(zxb2), el, 2, zetb); if (rc) return rc;
    }
    minors_from_ratios(liquid, el, elp1, rearth, ro, zom, el7, zeta, zetb, zxb2, ys);
  } else {
    if (el < EPS_F || liquid) { ys[0] = dz{1.0, 0.0}; ys[1] = dz{0.0, 0.0}; }
    else { ys[0] = dz{0, 0}; ys[1] = dz{1.0, 0.0}; ys[2] = dz{0, 0}; ys[3] = dz{0, 0}; ys[4] = dz{0, 0}; }
  }
  return ST_OK;
}

// toroidalBottomInitialValues (initialValues.f90:376-418)
__device__ int toroidal_bottom_iv(const FKStatic& P, const Env& e, double rstart, dz* ys, double& htry) {
  double ro; dz el7[7];
  eval_spline<0x40u>(P, e, rstart, e.nl, ro, el7);
  double el = -0.5 + sqrt(0.25 + e.dll1);
  double elp1 = e.dll1;
  dz zom{e.omre, e.omim};
  double rsq = rstart * rstart;
  double v = sqrt(el7[6].re / ro);
  htry = ((0.25 * v) * TWO_PI_F) / e.omre;
  if (rstart > P.roc) {
    dz zxb2 = (((ro * zom) * zom) * rsq) / el7[6], zetb;
    int rc;
    if (zabs(zxb2 / elp1) < 1.0) rc = zetl(zxb2, el, zetb);
    else rc = sphancf(zsqrt(zxb2), el, 1, zetb);
    if (rc) return rc;
    ys[0] = dz{1.0 / el, 0.0};
    ys[1] = (el7[6] / (rstart * el)) * ((el - 1.0) - zetb);
  } else {
    ys[0] = dz{1.0 / el, 0.0};
    ys[1] = dz{0.0, 0.0};
  }
  return ST_OK;
}

// toroidalSurfaceInitialValues (initialValues.f90:434-469)
__device__ int toroidal_surface_iv(const FKStatic& P, const Env& e, dz* ys, double& htry, double& rsurf,
                                   int& nl) {
  if (P.hasocean) { nl = P.nlay - 1; rsurf = P.ruc; } else { nl = P.nlay; rsurf = P.rearth; }
  double el = -0.5 + sqrt(0.25 + e.dll1);
  dz zom{e.omre, e.omim};
  double ro; dz el7[7];
  eval_spline<0x40u>(P, e, rsurf, nl, ro, el7);
  double v = sqrt(el7[6].re / ro);
  htry = ((0.25 * v) * TWO_PI_F) / e.omre;
  if (P.fsflag == 1) {
    double rsq = rsurf * rsurf;
    dz zxb2 = (((ro * zom) * zom) * rsq) / el7[6], zetb;
    int rc = sphancf(zsqrt(zxb2), el, 2, zetb); if (rc) return rc;
    ys[0] = dz{1.0 / el, 0.0};
    ys[1] = (el7[6] / (rsurf * el)) * ((el - 1.0) - zetb);
  } else {
    ys[0] = dz{1.0, 0.0}; ys[1] = dz{0.0, 0.0};
  }
  return ST_OK;
}

}  // namespace
}  // namespace GEM_NS
