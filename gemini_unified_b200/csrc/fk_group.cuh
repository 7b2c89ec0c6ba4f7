// Group form of the phase kernels (fast build): a group of lanes per solve.
//
// The thread form (fk_phases.cuh) walks one solve per lane, so a slab's time is
// the longest solve's serial chain of some hundred Bulirsch-Stoer steps, each of
// 32 matrix evaluations and 54 matrix-vector products one after another: about
// 60,000 cycles a step, whatever the number of solves below the 37,888 lanes.
// Here 16 lanes (8 in the toroidal phase) share one step:
//   * the attempts' sub-steps use 24 grid positions of the step besides its
//     start; their system matrices do not depend on the solution, so the
//     group's lanes evaluate them side by side into shared memory;
//   * the six attempts run as three chains of 16 sub-steps (n = 16; 12 and 4;
//     8, 6 and 2), one lane per chain and component of the solution: a lane
//     makes one row of the matrix-vector product, the vector passes through
//     shared memory;
//   * the convergence tests of attempts 3 to 6 run beside each other; the step
//     is accepted at the first that converges, as in the thread form.
// A seventh attempt (a few per cent of the steps) evaluates its 24 positions and
// runs alone.  The arithmetic of every entry, sub-step and test is that of the
// thread form in the same order, so both give the same bits.
// Bookkeeping (advance) is done by the group's first lane; its loops over the
// nodes are shared by the group.
#pragma once
#include "fk_phases.cuh"

namespace GEM_NS {
namespace {

constexpr int GP_PTS = 25;       // grid positions of a step: 0 and the multiples of 3 and 4 up to 48
constexpr int GP_WARPS = 12;     // warps per block, one block per SM

template <int PH> struct GroupShape {
  static constexpr int NV = PhaseNV<PH>::NV;
  static constexpr int GL = PH == PH_TOR ? 8 : 16;    // lanes per solve
  static constexpr int QS = PH == PH_TOR ? 5 : 17;    // double2 per matrix (odd: no bank conflicts)
};
template <int PH> struct GroupItem {
  Lane L;
  double2 E[GP_PTS * GroupShape<PH>::QS];
  double2 w[8 * PhaseNV<PH>::NV];   // vectors of the sub-steps, two buffers; correction and value of the tests
  double2 Y[6 * PhaseNV<PH>::NV];   // results of the attempts 1..6
};
template <int PH> constexpr size_t group_smem() { return sizeof(GroupItem<PH>) * (32 / GroupShape<PH>::GL) * GP_WARPS; }

// Matrix entries as complex numbers and, per row, the entries of the product in
// the order of sys_mul: entry | column << 5; rows are filled up with a zero entry.
template <int SYS> __device__ __forceinline__ void put_entries(const SysE<SYS>& E, double2* q) {
  auto put = [&](int i, dz z) { q[i] = make_double2(z.re, z.im); };
  auto real = [&](int i, double x) { q[i] = make_double2(x, 0.0); };
  if constexpr (SYS == SYS_MINORS) {
    const dz m22{E.m22, -E.a.im};
    put(0, E.a); put(1, E.m12); put(2, E.m14); put(3, E.m23); put(4, E.m24); put(5, E.m32); put(6, E.m42); put(7, E.z4);
    real(8, E.m11); real(9, E.m13); put(10, m22); put(11, dz{E.m33, -E.a.im}); put(12, dz{E.m55, E.a.im});
    put(13, -E.a); real(14, -E.m11); put(15, -m22); real(16, 0.0);
  } else if constexpr (SYS == SYS_SOLIDT) {
    put(0, E.a11); put(1, E.a12); put(2, E.a14); put(3, dz{E.a22, -E.a11.im}); put(4, E.z2); put(5, E.zrpc); put(6, E.a31);
    put(7, E.a32); put(8, E.a34); put(9, E.a43); real(10, E.rr); real(11, E.a42); real(12, 3.0 * E.rr); real(13, -E.rr);
    real(14, 0.0);
  } else if constexpr (SYS == SYS_TOROIDAL) {
    real(0, E.rr); put(1, E.m12); put(2, E.m21); real(3, -3.0 * E.rr);
  } else if constexpr (SYS == SYS_FLUID) {
    real(0, E.m11); put(1, E.m12); put(2, E.m21); real(3, 0.0);
  } else {
    put(0, E.m11); put(1, E.m12); put(2, E.m21); put(3, E.m22);
  }
}
#define GP_T(entry, col) ((entry) | (col) << 5)
struct GroupRows {
  unsigned char t[5][5][4];   // [system][row][term]
};
constexpr GroupRows make_rows() {
  GroupRows r{};
  constexpr unsigned char m[5][4] = {{GP_T(8, 0), GP_T(1, 1), GP_T(9, 2), GP_T(2, 3)},
                                     {GP_T(10, 1), GP_T(3, 2), GP_T(4, 3), GP_T(16, 0)},
                                     {GP_T(13, 0), GP_T(5, 1), GP_T(11, 2), GP_T(4, 4)},
                                     {GP_T(14, 0), GP_T(6, 1), GP_T(15, 3), GP_T(3, 4)},
                                     {GP_T(7, 0), GP_T(6, 2), GP_T(5, 3), GP_T(12, 4)}};
  constexpr unsigned char s[4][4] = {{GP_T(0, 0), GP_T(1, 1), GP_T(10, 2), GP_T(2, 3)},
                                     {GP_T(5, 0), GP_T(3, 1), GP_T(4, 3), GP_T(14, 0)},
                                     {GP_T(6, 0), GP_T(7, 1), GP_T(13, 2), GP_T(8, 3)},
                                     {GP_T(11, 1), GP_T(9, 2), GP_T(12, 3), GP_T(14, 0)}};
  for (int i = 0; i < 5; ++i) for (int k = 0; k < 4; ++k) r.t[SYS_MINORS][i][k] = m[i][k];
  for (int i = 0; i < 4; ++i) for (int k = 0; k < 4; ++k) r.t[SYS_SOLIDT][i][k] = s[i][k];
  for (int y : {(int)SYS_TOROIDAL, (int)SYS_FLUID, (int)SYS_RADIAL}) {
    r.t[y][0][0] = GP_T(0, 0); r.t[y][0][1] = GP_T(1, 1); r.t[y][1][0] = GP_T(2, 0); r.t[y][1][1] = GP_T(3, 1);
  }
  return r;
}
__device__ __constant__ const GroupRows GP_ROWS = make_rows();
#undef GP_T

struct GroupTab {   // in shared memory: lanes index them divergently
  double2 ext[4][5];   // extrapolation weights (w, e) of attempt 6, 5, 4 (chains 0, 1, 2) and 3 on attempts 1, 2, 3, 5, 4
  unsigned char grid[GP_PTS + 3], index[52];
};
__device__ __forceinline__ void group_tab(GroupTab& T) {
  int np = 0;
  for (int g = 0; g <= 48; ++g) {
    T.index[g] = (unsigned char)np;
    if (g % 3 == 0 || g % 4 == 0) T.grid[np++] = (unsigned char)g;
  }
  for (int q = 0; q < 4; ++q)
    for (int l = 0; l < 5; ++l) {
      const int j = 6 - q, i = l < 3 ? l + 1 : (l == 3 ? 5 : 4);
      T.ext[q][l] = i < j ? make_double2(EXTRAP.w[j][i - 1], EXTRAP.e[j][i - 1]) : make_double2(0.0, 0.0);
    }
}

// One step of the groups with act set (all lanes of the warp call); the result
// (attempts, 0 for a failed step) is returned to every lane of the group and an
// accepted solution is written to L.y.
template <int PH, int SYS, bool ISO>
__device__ __noinline__ int group_step(const FKStatic& P, GroupItem<PH>& G, const GroupTab& T, bool act, int lane) {
  constexpr int NV = SysNV<SYS>::NV, GL = GroupShape<PH>::GL, QS = GroupShape<PH>::QS;
  constexpr int NT = NV == 2 ? 2 : 4;   // terms per row
  const unsigned FULL = 0xffffffffu;
  const int sub = lane & (GL - 1), base = lane & ~(GL - 1);
  const double x = G.L.x, h48 = G.L.h / 48.0;
  int jknot = G.L.jknot;
  const EnvF e = make_envf(P, G.L.e, act, x, fma(48.0, h48, x), jknot);
  const dz zom2 = cmul(dz{e.omre, e.omim}, dz{e.omre, e.omim});
#pragma unroll 1
  for (int p = sub; p < GP_PTS; p += GL) {
    if (!act) break;
    SysE<SYS> E;
    sys_at<SYS, ISO>(e, zom2, fma((double)T.grid[p], h48, x), E);
    put_entries<SYS>(E, G.E + p * QS);
  }
  // chain and component of the lane, its row's terms
  const int ch = sub / NV, c = sub - ch * NV;
  const bool on = act && sub < 3 * NV;
  int eo[NT], zo[NT];
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    const int t = GP_ROWS.t[SYS][c][k];
    eo[k] = t & 31;
    zo[k] = t >> 5;
  }
  __syncwarp();
  if (act && sub == 0) G.L.jknot = jknot;
  dz y0{0.0, 0.0}, t0{0.0, 0.0};
  if (on) {
    y0 = G.L.y[c];
#pragma unroll
    for (int k = 0; k < NT; ++k) { const double2 a = G.E[eo[k]]; cfma(t0, dz{a.x, a.y}, G.L.y[zo[k]]); }
  }
  // z += row of the matrix times the weighted vector of the chain; mask: the lanes that do so
  auto mulrow = [&](unsigned mask, dz& z, const double2* row, double2* u, double wt, dz v) {
    double2 a[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) a[k] = row[eo[k]];
    u[c] = make_double2(wt * v.re, wt * v.im);
    __syncwarp(mask);
#pragma unroll
    for (int k = 0; k < NT; ++k) { const double2 q = u[zo[k]]; cfma(z, dz{a[k].x, a[k].y}, dz{q.x, q.y}); }
  };
  // chains: 16; 12 then 4; 8, 6 then 2 sub-steps (attempts 6; 5, 2; 4, 3, 1), two sub-steps per trip
  const unsigned onm = __ballot_sync(FULL, on);
  if (on) {
    int n = ch == 0 ? 16 : (ch == 1 ? 12 : 8), att = 6 - ch, m = 0, dg = 48 / n;
    double hf = (double)dg * h48;
    dz f0 = y0, f = y0;
    cfma(f, hf, t0);
    double2* u = G.w + ch * NV;
#pragma unroll 1
    for (int s = 0; s < 8; ++s) {
      const double2 *ra = G.E + T.index[(m + 1) * dg] * QS, *rb = G.E + T.index[(m + 2) * dg] * QS;
      m += 2;
      mulrow(onm, f0, ra, u, 2.0 * hf, f);
      mulrow(onm, f, rb, u + 3 * NV, m == n ? hf : 2.0 * hf, f0);
      if (m == n) {
        G.Y[(att - 1) * NV + c] = make_double2(0.5 * (f0.re + f.re), 0.5 * (f0.im + f.im));
        if (ch == 1) { n = 4; att = 2; }
        else if (n == 8) { n = 6; att = 3; }
        else { n = 2; att = 1; }
        m = 0; dg = 48 / n;
        hf = (double)dg * h48;
        f0 = f = y0;
        cfma(f, hf, t0);
      }
    }
  }
  __syncwarp();
  // extrapolation to the attempt with result yj (component c) from the first NL of the results of
  // the attempts 1, 2, 3, 5, 4, as in bs_step.  5 and 4 have weight 0 where the thread form has not
  // made them yet: left out, because they may have overflowed.
  auto extrapolate = [&](auto NL, const double2* wt, dz yj, dz& yy, dz& dy) {
    yy = yj;
    dy = dz{0.0, 0.0};
#pragma unroll
    for (int l = 0; l < decltype(NL)::value; ++l) {
      const double2 q = G.Y[(l < 3 ? l : (l == 3 ? 4 : 3)) * NV + c], k = wt[l];
      if (l < 3 || k.x != 0.0) {
        const dz d = dz{q.x, q.y} - yj;
        cfma(yy, k.x, d);
        cfma(dy, k.y, d);
      }
    }
  };
  auto put_test = [&](int q, dz yy, dz dy) {
    G.w[2 * (q * NV + c)] = make_double2(dy.re, dy.im);
    G.w[2 * (q * NV + c) + 1] = make_double2(yy.re, yy.im);
  };
  auto passes = [&](int q) {
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double2 d = G.w[2 * (q * NV + v)], y = G.w[2 * (q * NV + v) + 1];
      s1 = fma(d.x, d.x, fma(d.y, d.y, s1));
      s2 = fma(y.x, y.x, fma(y.y, y.y, s2));
    }
    return s1 < (P.eps * P.eps) * s2;
  };
  // attempts 6, 5, 4 on the chains 0, 1, 2, and 3 besides on the last
  dz yy{0.0, 0.0}, dy{0.0, 0.0}, y3{0.0, 0.0};
  if (on) {
    const double2 q = G.Y[(5 - ch) * NV + c];
    extrapolate(std::integral_constant<int, 5>(), T.ext[ch], dz{q.x, q.y}, yy, dy);
    put_test(ch, yy, dy);
    if (ch == 2) {
      const double2 r = G.Y[2 * NV + c];
      extrapolate(std::integral_constant<int, 2>(), T.ext[3], dz{r.x, r.y}, y3, dy);
      put_test(3, y3, dy);
    }
  }
  __syncwarp();
  const unsigned b1 = __ballot_sync(FULL, on && passes(ch));
  const unsigned b2 = __ballot_sync(FULL, on && ch == 2 && passes(3));
  int res = 0;
  if (act) res = b2 >> (base + 2 * NV) & 1 ? 3 : (b1 >> (base + 2 * NV) & 1 ? 4 : (b1 >> (base + NV) & 1 ? 5 : (b1 >> base & 1 ? 6 : 0)));
  if (on && res == 3 && ch == 2) G.L.y[c] = y3;
  if (on && res > 3 && ch == 6 - res) G.L.y[c] = yy;
  const bool seventh = act && res == 0;
  if (__any_sync(FULL, seventh)) {
    const bool on7 = seventh && sub < NV;
#pragma unroll 1
    for (int p = sub; p < 24; p += GL) {
      if (!seventh) break;
      SysE<SYS> E;
      sys_at<SYS, ISO>(e, zom2, fma((double)(2 * (p + 1)), h48, x), E);
      put_entries<SYS>(E, G.E + p * QS);
    }
    __syncwarp();   // the rows are other lanes' stores, and a vote orders no memory
    const unsigned onm7 = __ballot_sync(FULL, on7);
    if (on7) {
      const double hf = 2.0 * h48;
      dz f0 = y0, f = y0;
      cfma(f, hf, t0);
#pragma unroll 1
      for (int s = 0; s < 24; s += 2) {
        mulrow(onm7, f0, G.E + s * QS, G.w, 2.0 * hf, f);
        mulrow(onm7, f, G.E + (s + 1) * QS, G.w + 3 * NV, s == 22 ? hf : 2.0 * hf, f0);
      }
      const dz yj{0.5 * (f0.re + f.re), 0.5 * (f0.im + f.im)};
      yy = yj;
      dy = dz{0.0, 0.0};
#pragma unroll 1
      for (int l = 0; l < 6; ++l) {   // attempts 1, 2, 3, 5, 4, 6
        const int i = l < 3 ? l + 1 : (l == 3 ? 5 : (l == 4 ? 4 : 6));
        const double2 q = G.Y[(i - 1) * NV + c];
        const dz d = dz{q.x, q.y} - yj;
        cfma(yy, EXTRAP.w[7][i - 1], d);
        cfma(dy, EXTRAP.e[7][i - 1], d);
      }
    }
    __syncwarp();
    if (on7) put_test(0, yy, dy);
    __syncwarp();
    const unsigned b7 = __ballot_sync(FULL, on7 && passes(0));
    if (seventh && (b7 >> base & 1)) {
      res = 7;
      if (on7) G.L.y[c] = yy;
    }
  }
  __syncwarp();
  return res;
}

template <int PH>
__global__ void __launch_bounds__(GP_WARPS * 32, 1) fk_group_kernel(const __grid_constant__ FKStatic P, FKLaunch LL) {
  constexpr int GL = GroupShape<PH>::GL, IPW = 32 / GL;
  extern __shared__ __align__(16) unsigned char gp_raw[];
  __shared__ Tab tab;
  __shared__ GroupTab T;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & (GL - 1);
  if (threadIdx.x == 0) group_tab(T);
  load_tab(P, tab);
  load_bounds(P, tab);
  GroupItem<PH>& G = reinterpret_cast<GroupItem<PH>*>(gp_raw)[warp * IPW + lane / GL];
  Lane& L = G.L;
  LaneLayout lay{P.nnod + 1};
  const int slot_n = LaneLayout::PER_NODE * lay.NN + FK_LANE_STEP_SLOTS;
  const Slot s{LL.scratch + (long long)((blockIdx.x * GP_WARPS + warp) * IPW + lane / GL) * slot_n, 1};
  const bool lead = sub == 0;
  unsigned* queue = LL.queue + PH;
  Counters cnt{0, 0, 0, 0, 0, 0, 0, 0};
  if (lead) {
    L.st = S_FETCH;
    L.e.tab = &tab;
    L.jknot = 1;
  }
  __syncwarp();
  for (;;) {
    if (lead) {
      if (L.st == S_FETCH) {
        unsigned pos = atomicAdd(queue, 1u);
        if (pos < LL.nqueue) {
          if (PH == PH_ADJ && LL.nsrc > 0) {
            L.src = (int)(pos / (unsigned)LL.nitems);
            pos -= (unsigned)L.src * (unsigned)LL.nitems;
          }
          L.k = LL.order[pos];
          L.st = S_ITEM_NEW;
        } else {
          L.st = S_IDLE;
        }
      } else if (L.st != S_INTEG && L.st != S_IDLE) {
        advance<PH, true>(P, LL, s, lay, L);
      }
    }
    __syncwarp();
    const int st = L.st;
    __syncwarp();
    if (st == S_ITEM_NEW) {
      if (PH == PH_TOR)
        for (int el = sub; el < 4 * lay.NN; el += GL) s.put(el, dz{0.0, 0.0});
      if (PH == PH_ADJ)
        for (int el = sub; el < LaneLayout::PER_NODE * lay.NN; el += GL) s.put(el, dz{0.0, 0.0});
      if (lead) L.st = S_ITEM_INIT;
    } else if (PH == PH_TOR && st == S_TOR_OUT) {
      tor_output<PH>(P, LL, s, lay, L, sub, GL);
      if (lead) L.st = S_ITEM_END;
    } else if (PH == PH_SPH && st == S_SPH_NORM) {
      sph_normalise(P, LL, s, lay, L, sub, GL);
      if (lead) L.st = S_SPH_NORMED;
    } else if (PH == PH_ADJ && st == S_OUTPUT) {
      for (int n = 1 + sub; n <= P.nnod; n += GL) output_sph_node(P, s, lay, n, LL, L);
      if (lead) L.st = S_ITEM_END;
    }
    __syncwarp();
    const bool integ = st == S_INTEG;
    if (__any_sync(FULL, !integ && st != S_IDLE)) continue;
    if (!__any_sync(FULL, integ)) break;
    // overshoot clamp (integrationStep.f90:136-139)
    if (lead && integ && (L.x + L.h - L.xe) * (L.x + L.h - L.xa) > 0.0) L.h = L.xe - L.x;
    __syncwarp();
    int res = 0, sys = 0;
    auto step = [&](auto S) {
      constexpr int Y = decltype(S)::value;
      const bool act = integ && L.sys == Y;
      if (!__any_sync(FULL, act)) return;
      const int r = P.iso ? group_step<PH, Y, true>(P, G, T, act, lane) : group_step<PH, Y, false>(P, G, T, act, lane);
      if (act) { res = r; sys = Y; }
    };
    if constexpr (PH == PH_TOR) step(std::integral_constant<int, SYS_TOROIDAL>());
    else if constexpr (PH == PH_ADJ) step(std::integral_constant<int, SYS_SOLIDT>());
    else {
      step(std::integral_constant<int, SYS_MINORS>());
      step(std::integral_constant<int, SYS_FLUID>());
      step(std::integral_constant<int, SYS_RADIAL>());
    }
    // step-size control (integrationStep.f90:140-185) and the reference's work counts
    if (lead && integ) {
      const int jd = res ? res : 7, nv = sys == SYS_MINORS ? 5 : (sys == SYS_SOLIDT ? 4 : 2);
      const int mv = STEPWORK.mv[jd], sm = STEPWORK.sm[jd];
      cnt.attempts += jd;
      cnt.matvecs += mv;
      cnt.sysmats += sm;
      cnt.flops += (long long)sm * FLOP_SYSMAT[sys] + (long long)mv * FLOP_MV[sys] + STEPWORK.ext[nv][jd];
      L.nstep++;
      if (res > 0) {
        cnt.steps_ok++;
        L.x = L.x + L.h;
        if (fabs(L.x - L.xe) < MINSIZE_IS) {
          L.st = S_SUB_END;
        } else {
          if (res > L.kopt) L.h = L.h * SHRINK_BS;
          else if (res < L.kopt) L.h = L.h * GROW_BS;
          L.hdid = L.h;
        }
      } else {
        cnt.steps_rej++;
        L.h = 0.5 * L.h / 1.0;
        if (fabs(L.h) < MINSIZE_IS) { L.status = ST_MINSTEP; L.st = S_ITEM_END; }
      }
      if (L.st == S_INTEG && L.nstep >= MAXNUM_IS) { L.status = ST_MAXSTEPS; L.st = S_ITEM_END; }
    }
    __syncwarp();
  }
  long long v[6] = {cnt.steps_ok, cnt.steps_rej, cnt.attempts, cnt.sysmats, cnt.matvecs, cnt.flops};
  for (int kk = 0; kk < 6; ++kk) {
    long long t = v[kk];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(FULL, t, o);
    if (lane == 0) atomicAdd(LL.stats + kk, (unsigned long long)t);
  }
}

}  // namespace
}  // namespace GEM_NS
