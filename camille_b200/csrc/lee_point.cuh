// Pointwise part of the fused RK stage, shared by every stage kernel: the LEE
// right-hand side from the physical gradients (compute_RHS_linearized_Euler,
// camille src/solver/spatial_discretization.cpp:2053-2130), the monopole source and
// the Freund sponges (src/solver/source.cpp:10-18, :174-201), then the Runge-Kutta
// stage update with the hole bypass (RungeKutta::integrate,
// src/solver/temporal_discretization.cpp:205-229).
#pragma once

#include "lee_internal.h"

namespace lee {

// a b + c with one rounding: the kernels that share this file's terms give the same bits whatever
// the compiler would have contracted around them
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

template <typename T, typename I>
__device__ __forceinline__ T cval(const Coef<T>& c, I l) {
  return c.p ? __ldg(c.p + l) : c.c;
}

// The stage's kind: from the traits when they fix it, else from p.stage and p.last.
template <int TR>
struct Kind {
  static constexpr int K = (TR >> kKindShift) & 7;
  template <typename T>
  __device__ __forceinline__ static bool rhs(const StageParams<T>& p) {
    return K == kKindRuntime ? p.stage < 0 : K == kKindRhs;
  }
  template <typename T>
  __device__ __forceinline__ static bool first(const StageParams<T>& p) {
    return K == kKindRuntime ? p.stage == 0 : K == kKindFirst;
  }
  template <typename T>
  __device__ __forceinline__ static bool last(const StageParams<T>& p) {
    return K == kKindRuntime ? p.last != 0 : (K == kKindLast || K == kKindLastIncrement);
  }
  // the last stage writes the increment alone (compile-time kinds only)
  static constexpr bool increment = K == kKindLastIncrement;
};

// Per-point inputs read from global memory, gathered before the arithmetic so that
// every load of the point is in flight at once.
template <typename T, int DIM>
struct PointIn {
  T jm[DIM][DIM];     // J * metrics[d][x]
  T yn[DIM + 2];      // y_n (stages after the first)
  T av[DIM + 2];      // accumulator (stages after the first) or carried error (compensated, first stage)
  T sg;               // sponge strength (kTrSponge)
};

template <typename T, int DIM, bool COMP, int TR, typename I>
__device__ __forceinline__ void gather(const StageParams<T>& p, I l, PointIn<T, DIM>& in) {
  constexpr int V = DIM + 2;
  using K = Kind<TR>;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      const Coef<T>& c = p.jm[d * 3 + x];
      // TMA kernels: every entry is a field when any is
      in.jm[d][x] = (TR & kTrJmField) ? ((TR & kTrTma) ? __ldg(c.p + l) : cval(c, l)) : c.c;
    }
  const bool mid = !K::rhs(p) && !K::first(p);
  const bool need_yn = mid && (COMP || !K::last(p)) && !K::increment;
  const bool need_av = mid || (COMP && K::first(p));
#pragma unroll
  for (int v = 0; v < V; ++v) {
    in.yn[v] = need_yn ? p.yn[v][l] : T(0);
    in.av[v] = need_av ? (K::first(p) ? p.comp[v][l] : p.acc[v][l]) : T(0);
  }
  in.sg = (TR & kTrSponge) ? __ldg(p.sigma + l) : T(0);
}

template <typename T, int TR>
__device__ __forceinline__ bool reads_rho_prev(const StageParams<T>& p) {
  return (Kind<TR>::first(p) || Kind<TR>::rhs(p)) && p.rho_prev;
}

// The mean flow at a point of a non-uniform block, in one of two forms with the same values: read
// into registers ahead, every component of a gradient that is not identically zero (PointMean, where
// registers are to spare: the 11-point and direct 2-D kernels, the pairs of lee_pair.cuh), or read
// where it is used, component by component (MeanAt: k_stage and k_stage_tma, whose registers are
// full). k_stage_tma, 96^3, per launch: FP64 with one gradient component 80 us, read ahead 105; with
// all fifteen 130 and 129. FP32 51 and 67, 81 and 90. k_stage, FP32, 65^3 with two components: 56 and
// 76. The 11-point kernel, FP32: read ahead 78 and 85, where used 83 and 109.
template <typename T, int DIM>
struct PointMean {
  T ub_[DIM], rbi_, pb_, gs_[DIM], gu_[DIM][DIM], gp_[DIM];
  T rr_;  // rho'/rho_bar of the previous step (stages that read it), else 1 / p_bar
  __device__ __forceinline__ T ub(int x) const { return ub_[x]; }
  __device__ __forceinline__ T rbi() const { return rbi_; }
  __device__ __forceinline__ T pb() const { return pb_; }
  __device__ __forceinline__ T gs(int x) const { return gs_[x]; }
  __device__ __forceinline__ T gp(int x) const { return gp_[x]; }
  __device__ __forceinline__ T gu(int a, int x) const { return gu_[a][x]; }
  __device__ __forceinline__ T rho_prev() const { return rr_; }
  __device__ __forceinline__ T ipb() const { return rr_; }
  static __device__ __forceinline__ bool has(int terms, int field, int) { return (terms & field) != 0; }
};

template <typename T, int DIM, int TR, typename I>
__device__ __forceinline__ void gather_mean(const StageParams<T>& p, I l, PointMean<T, DIM>& m) {
  auto at = [&](int k) { return __ldg(p.mean[k] + (l & (I)p.mean_mask[k])); };
#pragma unroll
  for (int x = 0; x < DIM; ++x) m.ub_[x] = at(kMeanUb + x);
  m.rbi_ = at(kMeanRbi);
  m.pb_ = at(kMeanPb);
#pragma unroll
  for (int x = 0; x < DIM; ++x) {
    m.gs_[x] = (p.mean_terms & kMeanHasGs) ? at(kMeanGs + x) : T(0);
    m.gp_[x] = (p.mean_terms & kMeanHasGp) ? at(kMeanGp + x) : T(0);
#pragma unroll
    for (int a = 0; a < DIM; ++a) m.gu_[a][x] = (p.mean_terms & kMeanHasGu) ? at(kMeanGu + a * 3 + x) : T(0);
  }
  m.rr_ = !(p.mean_terms & kMeanHasGu) ? T(0) : (reads_rho_prev<T, TR>(p) ? p.rho_prev[l] : at(kMeanIpb));
}

template <typename T, typename I>
struct MeanAt {
  const StageParams<T>& p;
  I l;
  __device__ __forceinline__ T at(int k) const { return __ldg(p.mean[k] + (l & (I)p.mean_mask[k])); }
  __device__ __forceinline__ T ub(int x) const { return at(kMeanUb + x); }
  __device__ __forceinline__ T rbi() const { return at(kMeanRbi); }
  __device__ __forceinline__ T pb() const { return at(kMeanPb); }
  __device__ __forceinline__ T gs(int x) const { return at(kMeanGs + x); }
  __device__ __forceinline__ T gp(int x) const { return at(kMeanGp + x); }
  __device__ __forceinline__ T gu(int a, int x) const { return at(kMeanGu + a * 3 + x); }
  __device__ __forceinline__ T rho_prev() const { return p.rho_prev[l]; }
  __device__ __forceinline__ T ipb() const { return at(kMeanIpb); }
  static __device__ __forceinline__ bool has(int terms, int, int component) { return (terms & component) != 0; }
};

template <typename T, int DIM, int TR, typename M>
__device__ __forceinline__ void rhs_mean_terms(const StageParams<T>& p, const T (&g)[DIM + 2][DIM],
                                               const T (&q)[DIM + 2], const M& m, T (&r)[DIM + 2]);
template <typename T, int DIM, bool COMP, int TR, typename I>
__device__ __forceinline__ void rk_update(const StageParams<T>& p, I l, const T (&q)[DIM + 2],
                                          const PointIn<T, DIM>& in, const T (&r)[DIM + 2]);

// D[v][d]: computational-space derivative of field v along direction d; q[v]: the
// stage input at the point; in: the gathered inputs, mean: the mean flow of a non-uniform block.
// r receives the right-hand side.
template <typename T, int DIM, int TR, typename I, typename M>
__device__ __forceinline__ void rhs_point(const StageParams<T>& p, I l, int i, int j, int k,
                                          const T (&D)[DIM + 2][DIM], const T (&q)[DIM + 2],
                                          const PointIn<T, DIM>& in, const M& mean, T (&r)[DIM + 2]) {
  constexpr int V = DIM + 2;
  constexpr int P = DIM + 1;
  // physical gradients g[v][x] = sum_d JM[d][x] D_d f_v (take_derivative_xyz, :1802-1826)
  T g[V][DIM];
#pragma unroll
  for (int x = 0; x < DIM; ++x) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      T s = T(0);
#pragma unroll
      for (int d = 0; d < DIM; ++d) s = fma_t(in.jm[d][x], D[v][d], s);
      g[v][x] = s;
    }
  }
  constexpr bool UNI = (TR & kTrUniform) != 0;
  if (UNI) {
    T ub[DIM];
#pragma unroll
    for (int x = 0; x < DIM; ++x) ub[x] = p.ubar[x].c;
    // uniform mean flow: every mean-gradient term vanishes
    T rs = T(0);
#pragma unroll
    for (int x = 0; x < DIM; ++x) rs = fma_t(-ub[x], g[0][x], rs);
    r[0] = rs;
    const T rbi = p.rhobar_inv.c;
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      T ru = T(0);
#pragma unroll
      for (int x = 0; x < DIM; ++x) ru = fma_t(-ub[x], g[1 + a][x], ru);
      ru = fma_t(-g[P][a], rbi, ru);
      r[1 + a] = ru;
    }
    T rp = T(0);
    const T gpb = p.gamma * p.pbar.c;
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      rp = fma_t(-ub[x], g[P][x], rp);
      rp = fma_t(-gpb, g[1 + x][x], rp);
    }
    r[P] = rp;
  } else {
    rhs_mean_terms<T, DIM, TR>(p, g, q, mean, r);
  }
  if constexpr (DIM == 2 && !(TR & kTrTma)) {
    if (p.axisym) {
      // -gamma (p_bar u_r' + p' u_r_bar) / (r + DUMMY_SMALL), in FP64 in the reference's order
      // (src/solver/spatial_discretization.cpp:2118-2126)
      const double pb = (double)cval(p.pbar, l), ur = (double)cval(p.ubar[1], l);
      const double num = __dadd_rn(__dmul_rn(pb, (double)q[2]), __dmul_rn((double)q[P], ur));
      r[P] -= (T)__ddiv_rn(__dmul_rn((double)p.gamma, num), __dadd_rn(p.ry[l], 1e-99));
    }
  }
  if (p.has_src && i >= p.src_lo[0] && i <= p.src_hi[0] && j >= p.src_lo[1] && j <= p.src_hi[1] &&
      k >= p.src_lo[2] && k <= p.src_hi[2]) {
    int b0 = p.src_hi[0] - p.src_lo[0] + 1, b1 = p.src_hi[1] - p.src_lo[1] + 1;
    long long lb = (i - p.src_lo[0]) + (long long)b0 * ((j - p.src_lo[1]) + (long long)b1 * (k - p.src_lo[2]));
    const T amp = p.amp_tab ? p.amp_tab[*p.step_ctr * p.nstages + p.stage] : p.src_amp;
    r[P] = fma_t(amp, p.src_g[lb], r[P]);
  }
  if (TR & kTrSponge) {
#pragma unroll
    for (int v = 0; v < V; ++v) r[v] = fma_t(-in.sg, q[v], r[v]);
  } else {
    for (int z = 0; z < p.nzones; ++z) {
      const Zone<T>& zn = p.zones[z];
      if (i < zn.lo[0] || i > zn.hi[0] || j < zn.lo[1] || j > zn.hi[1] || k < zn.lo[2] || k > zn.hi[2]) continue;
      int b0 = zn.hi[0] - zn.lo[0] + 1, b1 = zn.hi[1] - zn.lo[1] + 1;
      long long lb = (i - zn.lo[0]) + (long long)b0 * ((j - zn.lo[1]) + (long long)b1 * (k - zn.lo[2]));
      T sg = zn.sig[lb];
      if (zn.ref) {
        // source::apply_bufferZone_Freund_harmonicWave (src/solver/source.cpp:264-320): the
        // reference state is the wave at the stage time
        const long long nbz = (long long)b0 * b1 * (zn.hi[2] - zn.lo[2] + 1);
#pragma unroll
        for (int v = 0; v < V; ++v) r[v] += -sg * (q[v] - zn.ref[v * nbz + lb]);
        continue;
      }
#pragma unroll
      for (int v = 0; v < V; ++v) r[v] += -sg * (q[v] - T(0));
    }
  }
}

// The right-hand side at a point, then the stage update: writes the next stage input and the
// accumulator.
template <typename T, int DIM, bool COMP, int TR, typename I, typename M>
__device__ __forceinline__ void rhs_update(const StageParams<T>& p, I l, int i, int j, int k,
                                           const T (&D)[DIM + 2][DIM], const T (&q)[DIM + 2],
                                           const PointIn<T, DIM>& in, const M& mean) {
  T r[DIM + 2];
  rhs_point<T, DIM, TR>(p, l, i, j, k, D, q, in, mean, r);
  rk_update<T, DIM, COMP, TR>(p, l, q, in, r);
}

// The LEE right-hand side of a non-uniform mean flow; gradients that are identically zero are
// skipped, by the field or component that M tells apart.
template <typename T, int DIM, int TR, typename M>
__device__ __forceinline__ void rhs_mean_terms(const StageParams<T>& p, const T (&g)[DIM + 2][DIM],
                                               const T (&q)[DIM + 2], const M& m, T (&r)[DIM + 2]) {
  constexpr int P = DIM + 1;
  const int has = p.mean_terms;
  T ub[DIM];
#pragma unroll
  for (int x = 0; x < DIM; ++x) ub[x] = m.ub(x);
  {
    T rs = T(0);
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      rs = fma_t(-ub[x], g[0][x], rs);
      if (M::has(has, kMeanHasGs, mean_gs(x))) rs = fma_t(-q[1 + x], m.gs(x), rs);
    }
    r[0] = rs;
  }
  T rr = T(0);
  if (has & kMeanHasGu) rr = reads_rho_prev<T, TR>(p) ? m.rho_prev() : fma_t(q[P] * p.inv_gamma, m.ipb(), -q[0]);
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    T ru = T(0);
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      ru = fma_t(-ub[x], g[1 + a][x], ru);
      if (M::has(has, kMeanHasGu, mean_gu(a, x))) ru = fma_t(-fma_t(rr, ub[x], q[1 + x]), m.gu(a, x), ru);
    }
    r[1 + a] = fma_t(-g[P][a], m.rbi(), ru);
  }
  {
    T rp = T(0);
    const T gpb = p.gamma * m.pb(), gq = p.gamma * q[P];
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      rp = fma_t(-ub[x], g[P][x], rp);
      if (M::has(has, kMeanHasGp, mean_gp(x))) rp = fma_t(-q[1 + x], m.gp(x), rp);
      rp = fma_t(-gpb, g[1 + x][x], rp);
      if (M::has(has, kMeanHasGu, mean_gu(x, x))) rp = fma_t(-gq, m.gu(x, x), rp);
    }
    r[P] = rp;
  }
}

// The Runge-Kutta stage update of one point from its right-hand side r.
template <typename T, int DIM, bool COMP, int TR, typename I>
__device__ __forceinline__ void rk_update(const StageParams<T>& p, I l, const T (&q)[DIM + 2],
                                          const PointIn<T, DIM>& in, const T (&r)[DIM + 2]) {
  constexpr int V = DIM + 2;
  using K = Kind<TR>;
  if (K::rhs(p)) {  // right-hand side only (spatial::compute_RHS)
#pragma unroll
    for (int v = 0; v < V; ++v) p.zout[v][l] = r[v];
    return;
  }
  const bool first = K::first(p), last = K::last(p);
  const bool hole = p.iblank && p.iblank[l] == 1;  // null on blocks without holes
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (hole) {
      p.acc[v][l] = T(0);
      if (!last || COMP) p.zout[v][l] = T(0);
      continue;
    }
    const T hk = r[v] * p.h;
    if (!COMP) {
      // y_next = y_n + sum b_i h k_i; the next stage input y_n + a h k_i
      const T yv = first ? q[v] : in.yn[v];
      const T prev = first ? q[v] : in.av[v];
      p.acc[v][l] = fma_t(p.b, hk, prev);
      if (!last) p.zout[v][l] = fma_t(p.a, hk, yv);
    } else {
      // compensated form: acc carries the increment of y since y_n plus the carried
      // rounding error of y; the last stage forms y_pre = y_n + increment as an exact
      // two-float sum (y_pre in zout, its rounding error in acc)
      const T yv = first ? q[v] : in.yn[v];
      const T inc = fma_t(p.b, hk, in.av[v]);
      if (!last) {
        p.acc[v][l] = inc;
        p.zout[v][l] = fma_t(p.a, hk, yv);
      } else if (K::increment) {
        p.acc[v][l] = inc;  // the filter forms y_pre and its rounding error
      } else {
        const T s = yv + inc;
        const T bb = s - yv;
        const T e = (yv - (s - bb)) + (inc - bb);
        p.zout[v][l] = s;
        p.acc[v][l] = e;
      }
    }
  }
}

}  // namespace lee
