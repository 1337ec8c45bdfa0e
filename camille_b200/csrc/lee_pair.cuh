// Two neighbouring points in packed FP32 (sm_100's __ffma2_rn, __fadd2_rn,
// __fmul2_rn): the pointwise part of the compensated RK stage, shared by the two-point kernels of
// 3-D and 2-D blocks (lee_stage_pair.cu, lee_plane.cu), so that both give the same bits.
#pragma once

#include "lee_point.cuh"

namespace lee {
namespace {

using F2 = float2;

__device__ __forceinline__ F2 f2(float x) { return make_float2(x, x); }
__device__ __forceinline__ F2 add(F2 a, F2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ F2 mul(F2 a, F2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
// a - b, exactly one rounding
__device__ __forceinline__ F2 sub(F2 a, F2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ F2 ld2(const float* p) { return *reinterpret_cast<const F2*>(p); }
__device__ __forceinline__ F2 ldg2(const float* p) { return __ldg(reinterpret_cast<const F2*>(p)); }
__device__ __forceinline__ void st2(float* p, F2 v) { *reinterpret_cast<F2*>(p) = v; }

// Pointwise inputs of a pair, gathered one plane ahead.
template <int DIM>
struct PairIn {
  F2 jm[DIM][DIM];  // J * metrics[d][x]
  F2 yn[DIM + 2];   // y_n (stages after the first)
  F2 av[DIM + 2];   // accumulator, or the carried rounding error (first stage)
  F2 sg;            // sponge strength
};

template <int DIM, int TR>
__device__ __forceinline__ void gather_pair(const StageParams<float>& p, unsigned l, PairIn<DIM>& in) {
  constexpr int V = DIM + 2;
  using K = Kind<TR>;
#pragma unroll
  for (int d = 0; d < DIM; ++d)
#pragma unroll
    for (int x = 0; x < DIM; ++x) in.jm[d][x] = (TR & kTrJmField) ? ldg2(p.jm[d * 3 + x].p + l) : f2(p.jm[d * 3 + x].c);
  const bool mid = !K::rhs(p) && !K::first(p);
  const bool need_av = mid || K::first(p);
#pragma unroll
  for (int v = 0; v < V; ++v) {
    in.yn[v] = (mid && !K::increment) ? ld2(p.yn[v] + l) : f2(0.f);
    in.av[v] = need_av ? (K::first(p) ? ld2(p.comp[v] + l) : ld2(p.acc[v] + l)) : f2(0.f);
  }
  in.sg = (TR & kTrSponge) ? ldg2(p.sigma + l) : f2(0.f);
}

// The mean flow at a pair of points of a non-uniform block (PointMean, lee_point.cuh).
template <int DIM>
struct PairField {
  F2 ub[DIM], rbi, pb, gs[DIM], gu[DIM][DIM], gp[DIM], rr;
};

template <int DIM, int TR>
__device__ __forceinline__ void gather_mean_pair(const StageParams<float>& p, unsigned l, PairField<DIM>& m) {
  auto at = [&](int k) { return ldg2(p.mean[k] + (l & (unsigned)p.mean_mask[k])); };
#pragma unroll
  for (int x = 0; x < DIM; ++x) m.ub[x] = at(kMeanUb + x);
  m.rbi = at(kMeanRbi);
  m.pb = at(kMeanPb);
#pragma unroll
  for (int x = 0; x < DIM; ++x) {
    m.gs[x] = (p.mean_terms & kMeanHasGs) ? at(kMeanGs + x) : f2(0.f);
    m.gp[x] = (p.mean_terms & kMeanHasGp) ? at(kMeanGp + x) : f2(0.f);
#pragma unroll
    for (int a = 0; a < DIM; ++a) m.gu[a][x] = (p.mean_terms & kMeanHasGu) ? at(kMeanGu + a * 3 + x) : f2(0.f);
  }
  m.rr = !(p.mean_terms & kMeanHasGu) ? f2(0.f) : (reads_rho_prev<float, TR>(p) ? ld2(p.rho_prev + l) : at(kMeanIpb));
}

// rhs_mean_terms (lee_point.cuh) of a pair
template <int DIM, int TR>
__device__ __forceinline__ void pair_mean_terms(const StageParams<float>& p, const F2 (&g)[DIM + 2][DIM],
                                                const F2 (&q)[DIM + 2], const PairField<DIM>& m, F2 (&r)[DIM + 2]) {
  constexpr int P = DIM + 1;
  const F2 neg = f2(-1.f);
  F2 nub[DIM], nu[DIM];
#pragma unroll
  for (int x = 0; x < DIM; ++x) {
    nub[x] = mul(m.ub[x], neg);
    nu[x] = mul(q[1 + x], neg);
  }
  F2 rr = f2(0.f);
  if (p.mean_terms & kMeanHasGu) {
    rr = m.rr;
    if (!reads_rho_prev<float, TR>(p)) rr = fma2(mul(q[P], f2(p.inv_gamma)), m.rr, mul(q[0], neg));
  }
  {
    F2 t = mul(nub[0], g[0][0]);
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      if (x) t = fma2(nub[x], g[0][x], t);
      if (p.mean_terms & kMeanHasGs) t = fma2(nu[x], m.gs[x], t);
    }
    r[0] = t;
  }
  const F2 ngpb = mul(m.pb, f2(-p.gamma)), ngq = mul(q[P], f2(-p.gamma));
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    F2 t = mul(nub[0], g[1 + a][0]);
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      if (x) t = fma2(nub[x], g[1 + a][x], t);
      if (p.mean_terms & kMeanHasGu) t = fma2(fma2(rr, nub[x], nu[x]), m.gu[a][x], t);
    }
    r[1 + a] = fma2(mul(g[P][a], neg), m.rbi, t);
  }
  {
    F2 t = mul(nub[0], g[P][0]);
#pragma unroll
    for (int x = 0; x < DIM; ++x) {
      if (x) t = fma2(nub[x], g[P][x], t);
      if (p.mean_terms & kMeanHasGp) t = fma2(nu[x], m.gp[x], t);
      t = fma2(ngpb, g[1 + x][x], t);
      if (p.mean_terms & kMeanHasGu) t = fma2(ngq, m.gu[x][x], t);
    }
    r[P] = t;
  }
}

// A block's uniform mean flow, negated where the right-hand side subtracts, and the stage's factors.
template <int DIM>
struct PairMean {
  F2 nub[DIM], nrbi, ngpb, h, b, a;
  __device__ __forceinline__ explicit PairMean(const StageParams<float>& s) {
#pragma unroll
    for (int x = 0; x < DIM; ++x) nub[x] = f2(-s.ubar[x].c);
    nrbi = f2(-s.rhobar_inv.c);
    ngpb = f2(-(s.gamma * s.pbar.c));
    h = f2(s.h);
    b = f2(s.b);
    a = f2(s.a);
  }
};

// From the pair's derivatives D[v][d], values q and gathered inputs to the next stage input and the
// accumulator at offset l (points (i, j, k) and (i + 1, j, k); src_ij0: the pair's (i, j) may lie in
// the source's box). STRIP: the pressure terms in the order of rhs_point (lee_point.cuh). A row's pad as the second point has D = q = 0 and zero inputs and stays zero.
template <int DIM, int TR, bool STRIP = false>
__device__ __forceinline__ void pair_update(const StageParams<float>& s, const PairMean<DIM>& M, unsigned l, int i,
                                            int j, int k, bool src_ij0, const F2 (&D)[DIM + 2][DIM],
                                            const F2 (&q)[DIM + 2], const PairIn<DIM>& in,
                                            const PairField<DIM>& mean) {
  using T = float;
  using K = Kind<TR>;
  constexpr int V = DIM + 2, PV = DIM + 1;
  // physical gradients g[v][x] = sum_d JM[d][x] D_d f_v (take_derivative_xyz, :1802-1826)
  F2 g[V][DIM];
#pragma unroll
  for (int x = 0; x < DIM; ++x)
#pragma unroll
    for (int v = 0; v < V; ++v) {
      F2 t = mul(in.jm[0][x], D[v][0]);
#pragma unroll
      for (int d = 1; d < DIM; ++d) t = fma2(in.jm[d][x], D[v][d], t);
      g[v][x] = t;
    }
  // uniform mean flow: r_s = -u.grad s', r_u = -u.grad u' - grad p' / rho, r_p = -u.grad p' - gamma p div u'
  F2 r[V];
  if (!(TR & kTrUniform)) {
    pair_mean_terms<DIM, TR>(s, g, q, mean, r);
  } else {
    F2 t = mul(M.nub[0], g[0][0]);
#pragma unroll
    for (int x = 1; x < DIM; ++x) t = fma2(M.nub[x], g[0][x], t);
    r[0] = t;
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      t = mul(M.nub[0], g[1 + a][0]);
#pragma unroll
      for (int x = 1; x < DIM; ++x) t = fma2(M.nub[x], g[1 + a][x], t);
      r[1 + a] = fma2(g[PV][a], M.nrbi, t);
    }
    t = mul(M.nub[0], g[PV][0]);
    if (STRIP) t = fma2(M.ngpb, g[1][0], t);
#pragma unroll
    for (int x = 1; x < DIM; ++x) {
      t = fma2(M.nub[x], g[PV][x], t);
      if (STRIP) t = fma2(M.ngpb, g[1 + x][x], t);
    }
    if (!STRIP) {
#pragma unroll
      for (int x = 0; x < DIM; ++x) t = fma2(M.ngpb, g[1 + x][x], t);
    }
    r[PV] = t;
  }
  // monopole: per point of the pair
  if (src_ij0 && k >= s.src_lo[2] && k <= s.src_hi[2]) {
    const T amp = s.amp_tab ? s.amp_tab[*s.step_ctr * s.nstages + s.stage] : s.src_amp;
    const int b0 = s.src_hi[0] - s.src_lo[0] + 1, b1 = s.src_hi[1] - s.src_lo[1] + 1;
    const long long row = (long long)b0 * ((j - s.src_lo[1]) + (long long)b1 * (k - s.src_lo[2]));
    if (i >= s.src_lo[0] && i <= s.src_hi[0]) r[PV].x += amp * s.src_g[row + (i - s.src_lo[0])];
    if (i + 1 >= s.src_lo[0] && i + 1 <= s.src_hi[0]) r[PV].y += amp * s.src_g[row + (i + 1 - s.src_lo[0])];
  }
  if (TR & kTrSponge) {
    const F2 nsg = mul(in.sg, f2(-1.f));
#pragma unroll
    for (int v = 0; v < V; ++v) r[v] = fma2(nsg, q[v], r[v]);
  } else {
    for (int zz = 0; zz < s.nzones; ++zz) {
      const Zone<T>& zn = s.zones[zz];
      if (j < zn.lo[1] || j > zn.hi[1] || k < zn.lo[2] || k > zn.hi[2]) continue;
      const int b0 = zn.hi[0] - zn.lo[0] + 1, b1 = zn.hi[1] - zn.lo[1] + 1;
      const long long row = (long long)b0 * ((j - zn.lo[1]) + (long long)b1 * (k - zn.lo[2]));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int ii = i + e;
        if (ii < zn.lo[0] || ii > zn.hi[0]) continue;
        const T sg = zn.sig[row + (ii - zn.lo[0])];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (e == 0) r[v].x += -sg * q[v].x;
          else r[v].y += -sg * q[v].y;
        }
      }
    }
  }
  // the compensated RK stage update (rk_update, lee_point.cuh)
  if (K::rhs(s)) {
#pragma unroll
    for (int v = 0; v < V; ++v) st2(s.zout[v] + l, r[v]);
  } else {
    const bool first = K::first(s), last = K::last(s);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const F2 hk = mul(r[v], M.h);
      const F2 yv = first ? q[v] : in.yn[v];
      const F2 inc = fma2(M.b, hk, in.av[v]);
      if (!last) {
        st2(s.acc[v] + l, inc);
        st2(s.zout[v] + l, fma2(M.a, hk, yv));
      } else if (K::increment) {
        st2(s.acc[v] + l, inc);  // the filter forms y_pre and its rounding error
      } else {
        const F2 sm = add(yv, inc);
        const F2 bv = sub(sm, yv);
        const F2 e = add(sub(yv, sub(sm, bv)), sub(inc, bv));
        st2(s.zout[v] + l, sm);
        st2(s.acc[v] + l, e);
      }
    }
  }
}

}  // namespace
}  // namespace lee
