// Stage and filter kernels of 2-D blocks: no shared memory, no barriers, no copies in flight.
//
// A 2-D block is one plane: the TMA-staged kernels (lee_tma.cu, lee_stage_pair.cu) load one box per
// CTA, wait for it, compute and leave, so a launch is a chain of latencies (3.4 us per stage at
// 256 x 256, where the bytes take 0.5), and the strip kernels of a batch (lee_batch.cu) pay a CTA
// barrier per row. Here every thread owns two neighbouring points along xi and reads its stencil
// straight from global memory: the pair's word and its left and right neighbours' (one 8- or
// 16-byte load each; a row's words are shared by the warp through L1), and the rows above and
// below. All loads of a point pair are in flight at once and nothing waits for another thread.
// Rows start on 16 bytes (the row pitch px), so every pair is aligned; taps beyond the block carry
// zero weight and are read from the pair itself.
//
// The stage kernel computes the same terms in the same order as the kernels it stands for
// (k_stage_pair or k_stage_tma for a block, batch_stage_run for a batch, whose right closure rows
// are summed from the edge inwards), then the pointwise right-hand side and RK update of
// lee_point.cuh or lee_pair.cuh. The filter kernel (k_filter_tma_row's arithmetic) filters a tile
// and its halo rows along xi into shared memory and takes F_eta from there after its one barrier.
#include <algorithm>
#include <cstddef>

#include "lee_plane.h"
#include "lee_pair.cuh"
#include "lee_tma_util.cuh"

namespace lee {
namespace {

template <typename T>
struct Vec2;
template <>
struct Vec2<float> {
  using V = float2;
};
template <>
struct Vec2<double> {
  using V = double2;
};

template <typename T>
struct Two {
  T a, b;
};

template <typename T>
__device__ __forceinline__ Two<T> ldp(const T* p) {  // coefficients: written by no kernel of the time loop
  const typename Vec2<T>::V v = __ldg(reinterpret_cast<const typename Vec2<T>::V*>(p));
  return Two<T>{v.x, v.y};
}
template <typename T>
__device__ __forceinline__ Two<T> ldw(const T* p) {
  const typename Vec2<T>::V v = *reinterpret_cast<const typename Vec2<T>::V*>(p);
  return Two<T>{v.x, v.y};
}
// the pair, or its first point alone where the second is the row's pad
template <typename T>
__device__ __forceinline__ void stp(T* p, T a, T b, bool both) {
  typename Vec2<T>::V v;
  v.x = a;
  v.y = b;
  if (both) *reinterpret_cast<typename Vec2<T>::V*>(p) = v;
  else *p = a;
}

constexpr int kH = kPlaneFdHalf;
constexpr int kNW = 2 * kH + 1;

// sum of w[o] f[o] in ascending order, or descending (the strip kernels' right closure rows)
template <typename T, int N>
__device__ __forceinline__ T taps(const T (&w)[N], const T (&f)[N], bool rev) {
  T s = T(0);
  if (!rev) {
#pragma unroll
    for (int o = 0; o < N; ++o) s = fma_t(w[o], f[o], s);
  } else {
#pragma unroll
    for (int o = N - 1; o >= 0; --o) s = fma_t(w[o], f[o], s);
  }
  return s;
}

// The words of a pair's xi neighbours and the pointwise inputs.
template <typename T, bool COMP, int TR>
__device__ __forceinline__ void load_inputs(const StageParams<T>& s, unsigned l, PointIn<T, 2> (&in)[2]) {
  constexpr int V = 4;
  using K = Kind<TR>;
#pragma unroll
  for (int d = 0; d < 2; ++d)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const Coef<T>& q = s.jm[d * 3 + x];
      Two<T> t{q.c, q.c};
      if ((TR & kTrJmField) && q.p) t = ldp(q.p + l);
      in[0].jm[d][x] = t.a;
      in[1].jm[d][x] = t.b;
    }
  const bool mid = !K::rhs(s) && !K::first(s);
  const bool need_yn = mid && (COMP || !K::last(s));
  const bool need_av = mid || (COMP && K::first(s));
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const Two<T> y = need_yn ? ldw(s.yn[v] + l) : Two<T>{T(0), T(0)};
    const Two<T> a = need_av ? ldw((K::first(s) ? s.comp[v] : s.acc[v]) + l) : Two<T>{T(0), T(0)};
    in[0].yn[v] = y.a;
    in[1].yn[v] = y.b;
    in[0].av[v] = a.a;
    in[1].av[v] = a.b;
  }
  const Two<T> g = s.sigma ? ldp(s.sigma + l) : Two<T>{T(0), T(0)};
  in[0].sg = g.a;
  in[1].sg = g.b;
}

// One pair of points (i, i + 1) of row j: derivatives, right-hand side, RK update. REV: a batch's
// order of terms (the strip kernels'). Uniform compensated blocks without holes take the packed
// arithmetic of lee_pair.cuh; a single block's xi taps then come in k_stage_pair's order.
template <typename T, bool COMP, int TR, bool HOLES, bool REV>
__device__ __forceinline__ void stage_point(const StageParams<T>& s, const T (&W)[6][5], int i, int j) {
  constexpr int V = 4;
  using K = Kind<TR>;
  const int nx = s.nx, ny = s.ny;
  const unsigned px = (unsigned)s.px;
  const bool both = i + 1 < nx;  // else the second point is the row's pad
  const unsigned l = (unsigned)i + px * (unsigned)j;
  const bool xin = i >= kH && i + 1 <= nx - 1 - kH, yin = j >= kH && j <= ny - 1 - kH;
  // offsets of the pair's left and right neighbours and of rows j - 2 .. j + 2; taps beyond the block
  // carry zero weight: the pair itself, or the nearest row, stands in
  const unsigned ll = i >= kH ? l - kH : l, lr = i + kH < nx ? l + kH : l;
  unsigned lo[kNW];
#pragma unroll
  for (int o = 0; o < kNW; ++o) lo[o] = (unsigned)i + px * (unsigned)min(max(j + o - kH, 0), ny - 1);
  if constexpr (COMP && (TR & kTrUniform) && !HOLES) {
    F2 D[V][2], q[V];
    // the stencil's words of one field
    struct Field {
      F2 m2, p2, y[kNW];
    };
    auto words = [&](int v) {
      const float* z = s.zin[v];
      Field w;
      w.m2 = ld2(z + ll);
      w.p2 = ld2(z + lr);
#pragma unroll
      for (int o = 0; o < kNW; ++o) w.y[o] = ld2(z + lo[o]);
      return w;
    };
    F2 wx[kNW], wy[kNW];
    const int c0 = cls_of(i, nx, kH), c1 = both ? cls_of(i + 1, nx, kH) : 1 + 2 * kH, cy = cls_of(j, ny, kH);
    if (xin && yin) {
#pragma unroll
      for (int o = 0; o < kNW; ++o) wx[o] = wy[o] = f2(W[0][o]);
    } else {
#pragma unroll
      for (int o = 0; o < kNW; ++o) {
        wx[o] = make_float2(W[c0][o], W[c1][o]);
        wy[o] = f2(W[cy][o]);
      }
    }
    auto right = [&](int cls) { return REV && cls > kH && cls <= 2 * kH; };
    const bool rx0 = right(c0), rx1 = right(c1), ry = right(cy);
    auto deriv = [&](int v, const Field& w) {
      const F2 m2 = w.m2, z0 = w.y[kH], p2 = w.p2;
      q[v] = z0;
      F2 dx = mul(wx[0], m2);
      if (!REV) {
        dx = fma2(wx[2], z0, dx);
        dx = fma2(wx[4], p2, dx);
        dx.x = fmaf(wx[1].x, m2.y, dx.x);
        dx.y = fmaf(wx[1].y, z0.x, dx.y);
        dx.x = fmaf(wx[3].x, z0.y, dx.x);
        dx.y = fmaf(wx[3].y, p2.x, dx.y);
      } else {
        dx.x = fmaf(wx[1].x, m2.y, dx.x);
        dx.y = fmaf(wx[1].y, z0.x, dx.y);
        dx = fma2(wx[2], z0, dx);
        dx.x = fmaf(wx[3].x, z0.y, dx.x);
        dx.y = fmaf(wx[3].y, p2.x, dx.y);
        dx = fma2(wx[4], p2, dx);
        if (rx0) {
          const float u[kNW] = {wx[0].x, wx[1].x, wx[2].x, wx[3].x, wx[4].x}, f[kNW] = {m2.x, m2.y, z0.x, z0.y, p2.x};
          dx.x = taps(u, f, true);
        }
        if (rx1) {
          const float u[kNW] = {wx[0].y, wx[1].y, wx[2].y, wx[3].y, wx[4].y}, f[kNW] = {m2.y, z0.x, z0.y, p2.x, p2.y};
          dx.y = taps(u, f, true);
        }
      }
      F2 dy;
      if (!ry) {
        dy = mul(wy[0], w.y[0]);
#pragma unroll
        for (int o = 1; o < kNW; ++o) dy = fma2(wy[o], w.y[o], dy);
      } else {
        dy = mul(wy[kNW - 1], w.y[kNW - 1]);
#pragma unroll
        for (int o = kNW - 2; o >= 0; --o) dy = fma2(wy[o], w.y[o], dy);
      }
      D[v][0] = dx;
      D[v][1] = dy;
    };
    // two fields' words in flight, then the next two and the pointwise inputs while they are used
    PairIn<2> pin;
    auto inputs = [&] {
      PointIn<T, 2> in[2];
      load_inputs<T, COMP, TR>(s, l, in);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        pin.yn[v] = make_float2(in[0].yn[v], in[1].yn[v]);
        pin.av[v] = make_float2(in[0].av[v], in[1].av[v]);
      }
#pragma unroll
      for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int x = 0; x < 2; ++x) pin.jm[d][x] = make_float2(in[0].jm[d][x], in[1].jm[d][x]);
      pin.sg = make_float2(in[0].sg, in[1].sg);
    };
    // a single block (few warps): every load before any arithmetic. A batch (many warps, so fewer
    // registers): two fields' words in flight, then the others and the pointwise inputs
    const Field a0 = words(0), a1 = words(1);
    const Field a2 = words(2);
    if (REV) deriv(0, a0);
    const Field a3 = words(3);
    if (REV) deriv(1, a1);
    inputs();
    if (!REV) {
      deriv(0, a0);
      deriv(1, a1);
    }
    deriv(2, a2);
    deriv(3, a3);
    const bool src = s.has_src && j >= s.src_lo[1] && j <= s.src_hi[1] && i + 1 >= s.src_lo[0] && i <= s.src_hi[0];
    pair_update<2, TR, REV>(s, PairMean<2>(s), l, i, j, 0, src, D, q, pin, PairField<2>{});
    return;
  }
  struct Field {
    Two<T> L, R, c[kNW];
  };
  auto words = [&](int v) {
    const T* z = s.zin[v];
    Field w;
    w.L = ldw(z + ll);
    w.R = ldw(z + lr);
#pragma unroll
    for (int o = 0; o < kNW; ++o) w.c[o] = ldw(z + lo[o]);
    return w;
  };
  T D[2][V][2], q[2][V];
  const bool inner = !HOLES && xin && yin;
  int cx[2] = {0, 0}, cy[2] = {0, 0};
  if (HOLES) {
    cx[0] = cls_of_code(s.code[0][l], kH);
    cx[1] = both ? cls_of_code(s.code[0][l + 1], kH) : 1 + 2 * kH;
    cy[0] = cls_of_code(s.code[1][l], kH);
    cy[1] = both ? cls_of_code(s.code[1][l + 1], kH) : 1 + 2 * kH;
  } else if (!inner) {
    cx[0] = cls_of(i, nx, kH);
    cx[1] = both ? cls_of(i + 1, nx, kH) : 1 + 2 * kH;
    cy[0] = cy[1] = cls_of(j, ny, kH);
  }
  auto right = [&](int cls) { return REV && cls > kH && cls <= 2 * kH; };
  auto deriv = [&](int v, const Field& w) {
    const T f[6] = {w.L.a, w.L.b, w.c[kH].a, w.c[kH].b, w.R.a, w.R.b};
    q[0][v] = w.c[kH].a;
    q[1][v] = w.c[kH].b;
    if (inner) {
      T x0 = T(0), x1 = T(0), y0 = T(0), y1 = T(0);
#pragma unroll
      for (int o = 0; o < kNW; ++o) {
        if (o == kH) continue;  // (the interior stencil's centre weight is zero)
        x0 = fma_t(W[0][o], f[o], x0);
        x1 = fma_t(W[0][o], f[o + 1], x1);
        y0 = fma_t(W[0][o], w.c[o].a, y0);
        y1 = fma_t(W[0][o], w.c[o].b, y1);
      }
      D[0][v][0] = x0;
      D[1][v][0] = x1;
      D[0][v][1] = y0;
      D[1][v][1] = y1;
      return;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      T wx[kNW], wy[kNW], fx[kNW], fy[kNW];
#pragma unroll
      for (int o = 0; o < kNW; ++o) {
        wx[o] = W[cx[e]][o];
        wy[o] = W[cy[e]][o];
        fx[o] = f[o + e];
        fy[o] = e ? w.c[o].b : w.c[o].a;
      }
      D[e][v][0] = taps(wx, fx, right(cx[e]));
      D[e][v][1] = taps(wy, fy, right(cy[e]));
    }
  };
  const Field a0 = words(0), a1 = words(1);
  const Field a2 = words(2);
  if (REV) deriv(0, a0);
  const Field a3 = words(3);
  if (REV) deriv(1, a1);
  PointIn<T, 2> in[2];
  load_inputs<T, COMP, TR>(s, l, in);
  PointMean<T, 2> mean[2];
  if (!(TR & kTrUniform)) {
    gather_mean<T, 2, TR>(s, l, mean[0]);
    gather_mean<T, 2, TR>(s, both ? l + 1 : l, mean[1]);
  }
  if (!REV) {
    deriv(0, a0);
    deriv(1, a1);
  }
  deriv(2, a2);
  deriv(3, a3);
  T r[2][V];
#pragma unroll
  for (int e = 0; e < 2; ++e) rhs_point<T, 2, TR>(s, both ? l + e : l, both ? i + e : i, j, 0, D[e], q[e], in[e], mean[e], r[e]);
  if (K::rhs(s)) {
#pragma unroll
    for (int v = 0; v < V; ++v) stp(s.zout[v] + l, r[0][v], r[1][v], both);
    return;
  }
  const bool first = K::first(s), last = K::last(s);
  bool hole[2] = {false, false};
  if (HOLES) {
    hole[0] = s.iblank[l] == 1;
    hole[1] = both && s.iblank[l + 1] == 1;
  }
  // the stage update (rk_update of lee_point.cuh) with the hole bypass
#pragma unroll
  for (int v = 0; v < V; ++v) {
    T ac[2], zo[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const T hk = r[e][v] * s.h;
      const T yv = first ? q[e][v] : in[e].yn[v];
      if (!COMP) {
        const T prev = first ? q[e][v] : in[e].av[v];
        ac[e] = fma_t(s.b, hk, prev);
        zo[e] = fma_t(s.a, hk, yv);
      } else {
        const T inc = fma_t(s.b, hk, in[e].av[v]);
        if (!last) {
          ac[e] = inc;
          zo[e] = fma_t(s.a, hk, yv);
        } else {
          const T sm = yv + inc;
          const T bb = sm - yv;
          zo[e] = sm;
          ac[e] = (yv - (sm - bb)) + (inc - bb);
        }
      }
      if (HOLES && hole[e]) ac[e] = zo[e] = T(0);
    }
    stp(s.acc[v] + l, ac[0], ac[1], both);
    if (COMP || !last) stp(s.zout[v] + l, zo[0], zo[1], both);
  }
}

// A kernel launched while its predecessor's last CTAs run waits here for the predecessor's end and
// for its writes: every thread, before it reads or writes a field, and also one that has no point.
// (Fields are read with plain loads, which stay behind the wait.) The predecessor gives no sign of
// its own, so a kernel's CTAs start as the predecessor's leave: per step of 64 x 48 FP64 12.3 us,
// 256 x 256 FP64 16.2, 513 x 385 FP32 21.5; with the sign at the predecessor's start, when waiting
// CTAs take room and issue slots from it, 14.6, 16.7 and 21.8; without early launches 13.1, 18.3
// and 23.5.
__device__ __forceinline__ void after_predecessor() { cudaGridDependencySynchronize(); }

template <typename P>
cudaError_t launch(void (*kernel)(P), dim3 grid, dim3 blk, const P& p, cudaStream_t s) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = blk;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = p.overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

// A warp owns 64 columns of one row; a CTA kPlaneRows rows.
template <typename T, bool COMP, int TR, bool HOLES>
__global__ void __launch_bounds__(32 * kPlaneRows, sizeof(T) == 4 ? 4 : 2)
    k_plane_stage(const __grid_constant__ PlaneStage<T> P) {
  const int i = (int)blockIdx.x * kPlaneCols + 2 * (int)threadIdx.x;
  const int j = (int)blockIdx.y * kPlaneRows + (int)threadIdx.y;
  after_predecessor();
  if (i >= P.s.nx || j >= P.s.ny) return;
  stage_point<T, COMP, TR, HOLES, false>(P.s, P.w, i, j);
}

// The tiles (block, x0, y0) of many blocks, 64 x kPlaneBatchTall points each; a CTA copies its block's
// parameters from global to shared memory.
template <typename T, bool COMP, int TR>
__global__ void __launch_bounds__(32 * kPlaneRows, sizeof(T) == 4 ? 4 : 2)
    k_plane_stage_batch(const StageParams<T>* __restrict__ prm, const int4* __restrict__ tiles,
                        const __grid_constant__ PlaneWeights<T> W) {
  __shared__ __align__(16) StageParams<T> s;
  const int4 t = __ldg(tiles + blockIdx.x);
  {
    const int* from = reinterpret_cast<const int*>(prm + t.x);
    int* to = reinterpret_cast<int*>(&s);
    for (int q = (int)threadIdx.y * 32 + (int)threadIdx.x; q < (int)(offsetof(StageParams<T>, fd) / 4);
         q += 32 * kPlaneRows)
      to[q] = __ldg(from + q);
  }
  __syncthreads();
  const int i = t.y + 2 * (int)threadIdx.x, j0 = t.z + (int)threadIdx.y, j1 = min(t.z + kPlaneBatchTall, s.ny);
  if (i >= s.nx) return;
  for (int j = j0; j < j1; j += kPlaneRows) stage_point<T, COMP, TR, false, true>(s, W.w, i, j);
}

// Offsets of the pair words of a row window of half-width HF around the pair, from 2 HP points
// before it, kept inside the row (a tap beyond it carries zero weight).
template <int HF>
struct Window {
  static constexpr int HP = (HF + 1) / 2, NP = 2 * HP + 1, NQ = 2 * HF + 1;
  static constexpr int E = 2 * HP - HF;  // window entries before the first point's first tap
  int xo[NP];
  __device__ __forceinline__ Window(int i, int nx) {
#pragma unroll
    for (int m = 0; m < NP; ++m) {
      const int o = 2 * (m - HP);
      xo[m] = (i + o >= 0 && i + o < nx) ? o : 0;
    }
  }
};

// The window of a tile row r (0: the first halo row) around the pair: from global memory (rows
// beyond the block feed zero-weight taps only: any row of it stands in), or from a TMA box (`at`:
// the pair's first point in the box's first row).
template <typename T, int HF>
struct GlobalRows {
  using Wn = Window<HF>;
  const T* x;
  int i, j0, ny;
  unsigned px;
  Wn win;
  __device__ __forceinline__ GlobalRows(const T* x_, int i_, int j0_, int nx, int ny_, int px_)
      : x(x_), i(i_ < nx ? i_ : 0), j0(j0_), ny(ny_), px((unsigned)px_), win(i_ < nx ? i_ : 0, nx) {}
  __device__ __forceinline__ void operator()(int r, Two<T> (&f)[Wn::NP]) const {
    const T* row = x + ((unsigned)min(max(j0 - HF + r, 0), ny - 1) * px + (unsigned)i);
#pragma unroll
    for (int m = 0; m < Wn::NP; ++m) f[m] = ldw(row + win.xo[m]);
  }
};
template <typename T, int HF>
struct BoxRows {
  using Wn = Window<HF>;
  const T* at;
  __device__ __forceinline__ void operator()(int r, Two<T> (&f)[Wn::NP]) const {
#pragma unroll
    for (int m = 0; m < Wn::NP; ++m) f[m] = ldw(at + r * PlaneFilterBox<T>::BX + 2 * (m - Wn::HP));
  }
};

// Pairs: w * a + c, a + b, a - b lane by lane (packed instructions in FP32, the same bits).
__device__ __forceinline__ void fma2p(Two<float> w, Two<float> a, Two<float>& c) {
  const F2 r = fma2(make_float2(w.a, w.b), make_float2(a.a, a.b), make_float2(c.a, c.b));
  c = Two<float>{r.x, r.y};
}
__device__ __forceinline__ void fma2p(Two<double> w, Two<double> a, Two<double>& c) {
  c = Two<double>{fma(w.a, a.a, c.a), fma(w.b, a.b, c.b)};
}
__device__ __forceinline__ Two<float> add2p(Two<float> a, Two<float> b) {
  const F2 r = add(make_float2(a.a, a.b), make_float2(b.a, b.b));
  return Two<float>{r.x, r.y};
}
__device__ __forceinline__ Two<double> add2p(Two<double> a, Two<double> b) { return Two<double>{a.a + b.a, a.b + b.b}; }
template <typename T>
__device__ __forceinline__ Two<T> sub2p(Two<T> a, Two<T> b) {
  return Two<T>{a.a - b.a, a.b - b.b};
}
template <typename T>
__device__ __forceinline__ void sts2(T* p, Two<T> v) {
  typename Vec2<T>::V x;
  x.x = v.a;
  x.y = v.b;
  *reinterpret_cast<typename Vec2<T>::V*>(p) = x;
}
// d += the o-th tap of both points from the window f, whose entry E + o is the first point's
template <int E, typename T, int NP>
__device__ __forceinline__ void tap_row(Two<T> w, const Two<T> (&f)[NP], int o, Two<T>& d) {
  const int t = E + o;
  if (t % 2 == 0) {
    fma2p(w, f[t / 2], d);
  } else {
    d.a = fma_t(w.a, f[t / 2].b, d.a);
    d.b = fma_t(w.b, f[t / 2 + 1].a, d.b);
  }
}

// The carried errors of the thread's pairs of a tile.
template <typename T, int RT>
__device__ __forceinline__ void tile_errors(const T* err, int nx, int ny, int px, int i, int j0, Two<T> (&e0)[RT]) {
#pragma unroll
  for (int q = 0; q < RT; ++q) {
    const int j = j0 + (int)threadIdx.y + kPlaneWarps * q;
    e0[q] = i < nx && j < ny ? ldw(err + ((unsigned)j * (unsigned)px + (unsigned)i)) : Two<T>{T(0), T(0)};
  }
}

// The filter of one field on a tile of kPlaneCols x kPlaneWarps * RT points at (i0, j0) (thread:
// columns i, i + 1): every warp filters its RT rows and its share of the 2 HF rows above and below
// along xi, straight from global memory, into shared memory (u1); after one barrier each warp
// takes F_eta of its rows from there. W: the class table (interior, left rows, right rows, zero).
template <typename T, bool COMP, int HF, int RT, bool HOLES, bool REV, typename Rows, typename Barrier>
__device__ __forceinline__ void filter_tile(const PlaneFilterField<T>& F, const Rows& rows,
                                            const T (&W)[1 + 2 * kPlaneFilterNb + 1][11], int nb, const int8_t* code0,
                                            const int8_t* code1, const int* iblank, T blend, int nx, int ny, int px,
                                            int i, int j0, T (*u1)[kPlaneCols], const Two<T> (&e0)[RT],
                                            Barrier&& barrier) {
  using Wn = Window<HF>;
  constexpr int NQ = Wn::NQ, NP = Wn::NP, NWP = kPlaneWarps, TYF = NWP * RT;
  constexpr int NH = (2 * HF + NWP - 1) / NWP;  // halo rows per warp
  constexpr int NR = RT + NH;                    // rows a warp filters along xi: its own, then its halo rows
  const int w = threadIdx.y, tc = 2 * (int)threadIdx.x;
  const bool col = i < nx, both = i + 1 < nx;
  // row of the tile (with its halo: 0 .. TYF + 2 HF - 1) of the warp's q-th xi row, -1 for none
  auto tile_row = [&](int q) -> int {
    if (q < RT) return HF + w + NWP * q;
    const int h = w + NWP * (q - RT);
    return h < HF ? h : (h < 2 * HF ? h + TYF : -1);
  };
  auto right = [&](int cls) { return REV && cls > nb && cls <= 2 * nb; };
  Two<T> f[NR][NP];
#pragma unroll
  for (int q = 0; q < NR; ++q) rows(max(tile_row(q), 0), f[q]);
  const int cxa = col ? cls_of(i, nx, nb) : 0, cxb = both ? cls_of(i + 1, nx, nb) : 0;
  const bool ra = right(cxa), rb = right(cxb), rx = REV && __any_sync(0xffffffffu, ra || rb);
  Two<T> wx[NQ];  // the pair's classes' weights (a row's pad stays zero)
  if (!HOLES) {
#pragma unroll
    for (int o = 0; o < NQ; ++o) wx[o] = Two<T>{W[cxa][o], both ? W[cxb][o] : T(0)};
  }
  Two<T> d1[RT];
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const int tr = tile_row(q);
    if (HOLES) {
      const unsigned l = (unsigned)min(max(j0 - HF + max(tr, 0), 0), ny - 1) * (unsigned)px + (unsigned)i;
      const int ca = col ? cls_of_code(code0[l], nb) : 0, cb = both ? cls_of_code(code0[l + 1], nb) : 0;
#pragma unroll
      for (int o = 0; o < NQ; ++o) wx[o] = Two<T>{W[ca][o], both ? W[cb][o] : T(0)};
    }
    Two<T> d{T(0), T(0)};
#pragma unroll
    for (int o = 0; o < NQ; ++o) tap_row<Wn::E>(wx[o], f[q], o, d);
    if (rx) {
      // (lanes of the last columns alone sum in descending order)
      T fa[NQ], fb[NQ], va[NQ], vb[NQ];
#pragma unroll
      for (int o = 0; o < NQ; ++o) {
        const int t = Wn::E + o;
        fa[o] = t % 2 ? f[q][t / 2].b : f[q][t / 2].a;
        fb[o] = t % 2 ? f[q][t / 2 + 1].a : f[q][t / 2].b;
        va[o] = wx[o].a;
        vb[o] = wx[o].b;
      }
      if (ra) d.a = taps(va, fa, true);
      if (rb) d.b = taps(vb, fb, true);
    }
    if (q < RT) d1[q] = d;
    if (tr >= 0) {
      const Two<T> x = f[q][Wn::HP];
      sts2(&u1[tr][tc], COMP ? add2p(x, d) : d);
    }
  }
  if (!barrier()) return;
  if (!col) return;
#pragma unroll
  for (int q = 0; q < RT; ++q) {
    const int j = j0 + w + NWP * q, tr = HF + w + NWP * q;
    if (j >= ny) continue;
    const unsigned l = (unsigned)j * (unsigned)px + (unsigned)i;
    Two<T> u[NQ];
#pragma unroll
    for (int o = 0; o < NQ; ++o) u[o] = ldw(&u1[tr - HF + o][tc]);
    int ca = cls_of(j, ny, nb), cb = ca;
    if (HOLES) {
      ca = cls_of_code(code1[l], nb);
      cb = both ? cls_of_code(code1[l + 1], nb) : 0;
    }
    Two<T> y{T(0), T(0)};
    if (ca == 0 && cb == 0) {
#pragma unroll
      for (int o = 0; o < NQ; ++o) fma2p(Two<T>{W[0][o], W[0][o]}, u[o], y);
    } else if (right(ca)) {
#pragma unroll
      for (int o = NQ - 1; o >= 0; --o) fma2p(Two<T>{W[ca][o], W[ca][o]}, u[o], y);
    } else {
#pragma unroll
      for (int o = 0; o < NQ; ++o) fma2p(Two<T>{W[ca][o], W[cb][o]}, u[o], y);
    }
    bool ha = false, hb = false;
    if (HOLES) {
      ha = iblank[l] == 1;
      hb = both && iblank[l + 1] == 1;
    }
    const Two<T> x = f[q][Wn::HP];
    if (!COMP) {
      const T a = fma_t(blend, y.a, (T(1) - blend) * x.a), b = fma_t(blend, y.b, (T(1) - blend) * x.b);
      stp(F.y + l, ha ? T(0) : a, hb ? T(0) : b, both);
    } else {
      // the exact two-float sum of the pre-filter value and blend * increment + carried error
      Two<T> t = e0[q];
      fma2p(Two<T>{blend, blend}, add2p(d1[q], y), t);
      const Two<T> sm = add2p(x, t), bb = sub2p(sm, x);
      const Two<T> ce = add2p(sub2p(x, sub2p(sm, bb)), sub2p(t, bb));
      stp(F.y + l, ha ? T(0) : sm.a, hb ? T(0) : sm.b, both);
      stp(F.comp + l, ha ? T(0) : ce.a, hb ? T(0) : ce.b, both);
    }
  }
}

template <typename T, bool COMP, int HF, int RT, bool HOLES>
__global__ void __launch_bounds__(32 * kPlaneWarps) k_plane_filter(const __grid_constant__ PlaneFilter<T> P) {
  __shared__ __align__(16) T u1[kPlaneWarps * RT + 2 * HF][kPlaneCols];
  const int i = (int)blockIdx.x * kPlaneCols + 2 * (int)threadIdx.x, j0 = (int)blockIdx.y * kPlaneWarps * RT;
  const PlaneFilterField<T>& F = P.f[blockIdx.z];
  Two<T> e0[RT];
  after_predecessor();
  if (COMP) tile_errors<T, RT>(F.err, P.nx, P.ny, P.px, i, j0, e0);
  filter_tile<T, COMP, HF, RT, HOLES, false>(F, GlobalRows<T, HF>(F.x, i, j0, P.nx, P.ny, P.px), P.w, P.nb, P.code[0],
                                             P.code[1], P.iblank, P.blend, P.nx, P.ny, P.px, i, j0, u1, e0, [] {
                                               __syncthreads();
                                               return true;
                                             });
}

// The tiles of many blocks, field blockIdx.y of each: a CTA takes `per` consecutive tiles, whose boxes
// (with their halos) come by TMA through a ring of kPlaneSlots slots. One barrier per tile: u1
// alternates between two buffers, and a box is free for the tile kPlaneSlots ahead once every
// thread is past the barrier of its tile.
template <typename T, bool COMP, int RT>
__global__ void __launch_bounds__(32 * kPlaneWarps, sizeof(T) == 4 ? 3 : 2)
    k_plane_filter_batch(const BatchFilterInst<T>* __restrict__ inst, const CUtensorMap* __restrict__ maps,
                         const int4* __restrict__ tiles, int ntiles, int per, const __grid_constant__ PlaneFilter<T> P,
                         int* err, unsigned long long wait_ns) {
  using B = PlaneFilterBox<T>;
  constexpr int NS = kPlaneSlots;
  constexpr int U1 = (kPlaneWarps * RT + 8) * kPlaneCols;
  extern __shared__ __align__(128) unsigned char smem[];
  T* ring = reinterpret_cast<T*>(smem);
  T* u1s = ring + NS * B::FB;
  __shared__ uint64_t bar[NS];
  const int v = blockIdx.y, tid = (int)threadIdx.y * 32 + (int)threadIdx.x;
  const int t0 = (int)blockIdx.x * per, t1 = min(t0 + per, ntiles);
  int issued = t0;  // thread 0: tiles whose copies are under way
  int acquired = -1;  // ... and the block whose map it has acquired
  auto issue_upto = [&](int last) {
    for (; issued < min(t1, last); ++issued) {
      const int4 t = __ldg(tiles + issued);
      const int q = (issued - t0) % NS;
      const CUtensorMap* map = maps + t.x * 4 + v;
      if (t.x != acquired) {
        acquire_map(map);
        acquired = t.x;
      }
      mbar_expect_tx(&bar[q], (unsigned)(sizeof(T) * B::FB));
      tma_load_3d(ring + q * B::FB, map, t.y - B::HX, t.z - 4, 0, &bar[q]);
    }
  };
  if (tid == 0) {
    for (int q = 0; q < NS; ++q) mbar_init(&bar[q], 1);
    fence_mbar_init();
    issue_upto(t0 + NS);
  }
  __syncthreads();
  for (int k = t0; k < t1; ++k) {
    const int4 t = __ldg(tiles + k);
    const BatchFilterInst<T>& b = inst[t.x];
    const PlaneFilterField<T> F{nullptr, b.err[v], b.y[v], b.comp[v]};
    const int nx = b.nx, ny = b.ny, px = b.px, i = t.y + 2 * (int)threadIdx.x;
    Two<T> e0[RT];
    if (COMP) tile_errors<T, RT>(F.err, nx, ny, px, i, t.z, e0);
    const int q = (k - t0) % NS;
    const bool ok = mbar_wait(&bar[q], (unsigned)(((k - t0) / NS) & 1), wait_ns);
    // (a thread whose wait gave up reads a box in flight: values only, never used)
    bool failed = false;
    T(*u1)[kPlaneCols] = reinterpret_cast<T(*)[kPlaneCols]>(u1s + ((k - t0) & 1) * U1);
    filter_tile<T, COMP, 4, RT, false, true>(F, BoxRows<T, 4>{ring + q * B::FB + B::HX + 2 * (int)threadIdx.x}, P.w, P.nb,
                                             nullptr, nullptr, nullptr, P.blend, nx, ny, px, i, t.z, u1, e0, [&] {
                                               failed = __syncthreads_or(!ok) != 0;
                                               if (!failed && tid == 0) issue_upto(k + 1 + NS);
                                               return !failed;
                                             });
    if (failed) {
      if (tid == 0) {
        atomicExch(err, 1);
        for (int w = k; w < issued; ++w) mbar_wait(&bar[(w - t0) % NS], (unsigned)(((w - t0) / NS) & 1));
      }
      return;
    }
  }
}

template <typename T, bool COMP, int TR>
cudaError_t go_stage(const PlaneStage<T>& p, cudaStream_t s) {
  const dim3 grid((p.s.nx + kPlaneCols - 1) / kPlaneCols, (p.s.ny + kPlaneRows - 1) / kPlaneRows);
  const dim3 blk(32, kPlaneRows);
  if (p.s.code[0]) return launch<PlaneStage<T>>(k_plane_stage<T, COMP, TR, true>, grid, blk, p, s);
  // (a varying mean flow without holes runs the TMA kernels)
  if constexpr ((TR & kTrUniform) != 0) return launch<PlaneStage<T>>(k_plane_stage<T, COMP, TR, false>, grid, blk, p, s);
  return cudaErrorInvalidValue;
}

constexpr int kBase = kTrTma | kTrSponge;

template <typename T, bool COMP, int KIND>
cudaError_t go_stage_layout(const PlaneStage<T>& p, int traits, cudaStream_t s) {
  constexpr int B = kBase | (KIND << kKindShift);
  switch (traits & (kTrJmField | kTrUniform)) {
    case 0: return go_stage<T, COMP, B>(p, s);
    case kTrJmField: return go_stage<T, COMP, B | kTrJmField>(p, s);
    case kTrUniform: return go_stage<T, COMP, B | kTrUniform>(p, s);
    default: return go_stage<T, COMP, B | kTrJmField | kTrUniform>(p, s);
  }
}

// CTAs of `threads` threads and `smem` bytes of a kernel that the device holds at once (its shared
// memory limit is raised first)
template <typename K>
int resident_ctas(int dev, K kernel, int threads, size_t smem) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  int sms = 0, per = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess) return 0;
  return sms * per;
}

template <typename T, bool COMP, int JM>
cudaError_t go_batch(const StageParams<T>* prm, const int4* tiles, int n, const PlaneWeights<T>& w, int kind,
                     cudaStream_t s) {
  constexpr int B = kBase | kTrUniform | JM;
  const dim3 blk(32, kPlaneRows);
  switch (kind) {
    case kKindFirst: k_plane_stage_batch<T, COMP, B | (kKindFirst << kKindShift)><<<n, blk, 0, s>>>(prm, tiles, w); break;
    case kKindMid: k_plane_stage_batch<T, COMP, B | (kKindMid << kKindShift)><<<n, blk, 0, s>>>(prm, tiles, w); break;
    case kKindLast: k_plane_stage_batch<T, COMP, B | (kKindLast << kKindShift)><<<n, blk, 0, s>>>(prm, tiles, w); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <typename T, int HF, int RT>
cudaError_t go_filter(const PlaneFilter<T>& p, int V, cudaStream_t s) {
  constexpr bool COMP = sizeof(T) == 4;
  constexpr int TYF = kPlaneWarps * RT;
  const dim3 grid((p.nx + kPlaneCols - 1) / kPlaneCols, (p.ny + TYF - 1) / TYF, V), blk(32, kPlaneWarps);
  return launch<PlaneFilter<T>>(p.code[0] ? k_plane_filter<T, COMP, HF, RT, true> : k_plane_filter<T, COMP, HF, RT, false>,
                                grid, blk, p, s);
}

template <typename T, int HF>
cudaError_t go_filter_rows(const PlaneFilter<T>& p, int V, cudaStream_t s) {
  return p.rows == 1 ? go_filter<T, HF, 1>(p, V, s) : go_filter<T, HF, 2>(p, V, s);
}

}  // namespace

template <typename T>
cudaError_t launch_plane_stage(const PlaneStage<T>& p, int traits, cudaStream_t s) {
  constexpr bool COMP = sizeof(T) == 4;
  switch ((traits >> kKindShift) & 7) {
    case kKindRhs: return go_stage_layout<T, COMP, kKindRhs>(p, traits, s);
    case kKindFirst: return go_stage_layout<T, COMP, kKindFirst>(p, traits, s);
    case kKindMid: return go_stage_layout<T, COMP, kKindMid>(p, traits, s);
    case kKindLast: return go_stage_layout<T, COMP, kKindLast>(p, traits, s);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t launch_plane_stage_batch(const StageParams<T>* prm, const int4* tiles, int n, const PlaneWeights<T>& w,
                                     int kind, bool jm_fields, cudaStream_t s) {
  constexpr bool COMP = sizeof(T) == 4;
  return jm_fields ? go_batch<T, COMP, kTrJmField>(prm, tiles, n, w, kind, s)
                   : go_batch<T, COMP, 0>(prm, tiles, n, w, kind, s);
}

template <typename T>
cudaError_t launch_plane_filter(const PlaneFilter<T>& p, int hf, int V, cudaStream_t s) {
  if (hf == 2) return go_filter_rows<T, 2>(p, V, s);
  if (hf == 4) return go_filter_rows<T, 4>(p, V, s);
  if (hf == 5) return go_filter_rows<T, 5>(p, V, s);
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_plane_filter_batch(const BatchFilterInst<T>* inst, const CUtensorMap* maps, const int4* tiles, int n,
                                      const PlaneFilter<T>& p, int* err, unsigned long long wait_ns, cudaStream_t s) {
  constexpr bool COMP = sizeof(T) == 4;
  const size_t smem = sizeof(T) * (kPlaneSlots * PlaneFilterBox<T>::FB +
                                   2 * (kPlaneWarps * kPlaneBatchRows + 8) * kPlaneCols);
  static PerDevice held;
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  const int resident = held.get(
      dev, [&] { return resident_ctas(dev, k_plane_filter_batch<T, COMP, kPlaneBatchRows>, 32 * kPlaneWarps, smem); });
  if (resident <= 0) return cudaErrorInvalidConfiguration;
  const int runs = std::max(1, resident / 4), per = (n + runs - 1) / runs;  // four fields
  k_plane_filter_batch<T, COMP, kPlaneBatchRows><<<dim3((n + per - 1) / per, 4), dim3(32, kPlaneWarps), smem, s>>>(
      inst, maps, tiles, n, per, p, err, wait_ns);
  return cudaGetLastError();
}

void plane_filter_box(int* bx, int* by) {
  *bx = PlaneFilterBox<float>::BX;
  *by = PlaneFilterBox<float>::BY;
}

#define LEE_PLANE_INST(T)                                                                                          \
  template cudaError_t launch_plane_stage<T>(const PlaneStage<T>&, int, cudaStream_t);                             \
  template cudaError_t launch_plane_stage_batch<T>(const StageParams<T>*, const int4*, int, const PlaneWeights<T>&, \
                                                   int, bool, cudaStream_t);                                       \
  template cudaError_t launch_plane_filter<T>(const PlaneFilter<T>&, int, int, cudaStream_t);                      \
  template cudaError_t launch_plane_filter_batch<T>(const BatchFilterInst<T>*, const CUtensorMap*, const int4*, int, \
                                                    const PlaneFilter<T>&, int*, unsigned long long, cudaStream_t);
LEE_PLANE_INST(float)
LEE_PLANE_INST(double)
#undef LEE_PLANE_INST

}  // namespace lee
