// Fused three-direction filter of 3-D blocks without holes, two rows per thread (sm_100a): two points
// of each row in FP32, one in FP64.
//
// spatial::apply_filter (src/solver/spatial_discretization.cpp:2191-2246) filters line by line in
// xi, then eta, then zeta, and the blend with the pre-filter state follows. This kernel fuses the
// three passes as k_filter_tma_row (lee_tma.cu) does, with each point's arithmetic in the same
// order (the same bits), but every thread owns two neighbouring points along xi:
//   - the pair's xi taps come from 8-byte shared-memory words, and the xi taps whose two values
//     lie in one word run as packed FP32 instructions (__ffma2_rn, with the pair's two weights
//     held in a register pair), as do the sums of pairs (__fadd2_rn);
//   - the per-plane work (the wait on the plane's copy, the barrier, addressing) is shared by the
//     two points, and the output moves in 8-byte words.
//
// A CTA owns 64 x 16 points in (i, j) (FP64: 32 x 16), two neighbouring rows per thread, and marches along k through
// a chunk of planes. Per incoming plane p (one TMA box: the tile plus its halos, in a ring of h + 4
// slots):
//   xi:   F_xi - I at the thread's own rows and at one eta halo row, from the box, into one of two
//         shared row buffers (u1, alternating by plane, so one barrier per plane suffices);
//   eta:  F_eta - I at the own rows, from one window of u1 for both;
//   zeta: a register queue of the last 2h + 1 planes' F_eta F_xi values and a per-thread shared
//         ring of the last h + 1 planes' summed xi and eta increments finish plane p - h: F_zeta,
//         then the blend as the exact
//         two-float sum of the pre-filter value, blend * (sum of the increments) and the carried
//         rounding error. The pre-filter value comes from the ring, whose slot of plane p - h is
//         re-issued only after every thread has finished that plane.
// Each thread keeps its pair's xi weights (one closure class per point) in registers; rows near an
// eta end (one warp each) and planes near a zeta end take their class rows.
//
// Bound by the latencies that 16 warps per SM leave open (192^3 FP32: 60 % of the issue slots, the
// shared-memory pipe 53 %, DRAM 40 %; the bytes take 208 us at 256^3): one row per thread took 78 %
// of the issue slots for 292 instructions per pair and plane. Two rows share the wait, the barrier,
// the addresses, the classes and the eta window, and a tile of 16 rows filters half a halo row per
// own row instead of one: 90 instructions per point and field instead of 152, 429 -> 355 us at
// 256^3, 49 -> 37 at 128 x 112 x 96; the zeta queue shifted every third plane (its entries are
// addressed statically in between): 350 and 36. Small and very narrow blocks have too few of the
// 64 x 16 tiles (20^3 FP32 14.8 us, one row and one point 12.7; 16 x 400 x 300 takes that form too):
// lee_prepare times the forms. FP64 (one point of each row, no increments; 47 % of the issue slots,
// shared memory 64 %) against k_filter_tma with two rows per thread, whose weights along eta and queues of
// pre-filter values and increments shift every plane: 189 -> 129 us at 160 x 144 x 128.
//
// Every mbarrier wait is bounded (about one second, or the context's limit); on expiry the CTA
// records the failure in the device flag, waits (bounded) for its own copies in flight and
// returns.
#include "lee_tma.h"
#include "lee_tma_util.cuh"

namespace lee {
namespace {

using F2 = float2;

__device__ __forceinline__ F2 add2(F2 a, F2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
// w * a + c and a - b lane by lane (scalar instructions)
__device__ __forceinline__ F2 fmas(float w, F2 a, F2 c) { return make_float2(fmaf(w, a.x, c.x), fmaf(w, a.y, c.y)); }
__device__ __forceinline__ F2 subs(F2 a, F2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double add2(double a, double b) { return a + b; }
__device__ __forceinline__ double fmas(double w, double a, double c) { return fma(w, a, c); }
__device__ __forceinline__ double subs(double a, double b) { return a - b; }

// What a thread owns of a row: two points in FP32, one in FP64.
template <typename T>
struct Own;
template <>
struct Own<float> {
  using W = float2;
  static constexpr int N = 2;
  static __device__ __forceinline__ W zero() { return make_float2(0.f, 0.f); }
  // (1 - b) x + b f with the roundings of the other forms (lee_tma.cu)
  static __device__ __forceinline__ W blend(float b, W x, W f) {
    return make_float2(fmaf(b, f.x, (1.f - b) * x.x), fmaf(b, f.y, (1.f - b) * x.y));
  }
};
template <>
struct Own<double> {
  using W = double;
  static constexpr int N = 1;
  static __device__ __forceinline__ W zero() { return 0.0; }
  static __device__ __forceinline__ W blend(double b, W x, W f) { return fma(b, f, (1.0 - b) * x); }
};
template <typename T>
__device__ __forceinline__ typename Own<T>::W ld2(const T* p) {
  return *reinterpret_cast<const typename Own<T>::W*>(p);
}
template <typename T>
__device__ __forceinline__ void st2(T* p, typename Own<T>::W v) {
  *reinterpret_cast<typename Own<T>::W*>(p) = v;
}

constexpr int kPairLX = 32;           // threads per tile row (one warp)
constexpr int kPairWarps = 8;         // warps of a CTA
constexpr int kPairRY = 2;            // rows a thread owns
constexpr int kPairUnroll = 3;        // planes between shifts of the zeta queue
constexpr int kPairTY = kPairWarps * kPairRY;

// Geometry of the kernel for half-width HF.
template <typename T, int HF>
struct PairGeo {
  static constexpr int A = 16 / (int)sizeof(T), TX = kPairLX * Own<T>::N;  // points along i per CTA
  static constexpr int HX = ((HF + A - 1) / A) * A;  // xi halo of the box: every TMA row starts on 16 bytes
  static constexpr int BX = TX + 2 * HX;
  static constexpr int BY = kPairTY + 2 * HF;
  static constexpr int FB = BX * BY;
  static constexpr int FBP = ((FB * (int)sizeof(T) + 127) / 128) * 128 / (int)sizeof(T);  // box stride: 128-byte multiple
  static constexpr int PF = 3;                                   // planes of prefetch
  static constexpr int NS = HF + 1 + PF;                          // ring slots
  static constexpr int HP = (HF + 1) / 2;  // a pair's row window starts 2 HP points before it
  static constexpr int NW = 1 + 2 * HP;    // 8-byte words of the window
  static constexpr int U1 = BY * TX;  // elements of one row buffer
  static constexpr int ND = HF + 1;        // planes of summed increments kept per point
  static constexpr int DP = kPairTY * TX;  // elements of one plane of them
  // (the compensated form alone keeps increments)
  static constexpr size_t bytes(bool comp) {
    return ((size_t)NS * FBP + 2 * U1 + (comp ? ND * DP : 0)) * sizeof(T) + NS * sizeof(uint64_t);
  }
  static_assert(HX % 2 == 0 && BX % 2 == 0, "pairs start on 8 bytes");
  // the window of the last pair (column HX + kPairTX - 2) ends inside the box row
  static_assert(Own<T>::N == 1 || (2 * HP <= HX && HX + TX - 2 + 2 * HP + 1 < BX), "row window inside the box");
  static_assert(BX <= 256 && BY <= 256, "TMA box dimensions are at most 256");
  static_assert(((size_t)NS * FBP + 2 * U1 + ND * DP) * sizeof(T) % 8 == 0, "mbarriers need 8-byte alignment");
};

// COMP: the compensated form (the increments F - I, the carried rounding error in and out);
// otherwise the plain filter and blend (out = (1 - blend) x + blend F x, the adjoint's transposed
// filter, whose class rows are the transposed operator's).
template <typename T, int HF, bool COMP>
__global__ void __launch_bounds__(32 * kPairWarps, 2) k_filter_pair(const __grid_constant__ FieldMaps ym,
                                                     const __grid_constant__ TmaFilterParams<T> P) {
  using G = PairGeo<T, HF>;
  using O = Own<T>;
  using W = typename O::W;
  constexpr int N = O::N, TX = G::TX;
  constexpr int U = kPairUnroll, RY = kPairRY, TY = kPairTY, NQ = 2 * HF + 1, NS = G::NS, BX = G::BX, FBP = G::FBP, HP = G::HP, NW = G::NW;
  extern __shared__ __align__(128) unsigned char smem[];
  T* ring = reinterpret_cast<T*>(smem);
  T* u1s = ring + NS * FBP;  // [2][BY][TX]
  // [ND][TY][TX]: the summed xi and eta increments of the last h + 1 planes, each point's
  // own (written and read by its thread only)
  T* dsm = u1s + 2 * G::U1;
  uint64_t* bar = reinterpret_cast<uint64_t*>(dsm + (COMP ? G::ND * G::DP : 0));

  const int v = blockIdx.z;
  const int i0 = (int)(blockIdx.x % P.tiles_x) * TX, j0 = (int)(blockIdx.x / P.tiles_x) * TY;
  const int k0 = (int)blockIdx.y * P.k_chunk;
  const int k1 = min(P.nz, k0 + P.k_chunk);
  const int tid = threadIdx.x, tx = tid % kPairLX, ty = tid / kPairLX;
  const int i = i0 + N * tx, j = j0 + RY * ty;  // the pair's first row: rows j .. j + RY - 1
  // with an odd nx the last pair's second point is the row's pad (the pitch px is even): its xi
  // weights are zero and the copies fill beyond nx with zeros, so its pad values stay zero
  const bool active = i < P.nx && j < P.ny;  // (a further row is checked when it is stored)
  const int plo = max(0, k0 - HF), phi = min(P.nz - 1, k1 - 1 + HF);

  if (tid == 0) {
    for (int q = 0; q < NS; ++q) mbar_init(&bar[q], 1);
    fence_mbar_init();
  }
  __syncthreads();
  int next_issue = plo;  // meaningful in thread 0 only
  auto issue_upto = [&](int last) {
    for (; next_issue <= min(phi, last); ++next_issue) {
      const int slot = (next_issue - plo) % NS;
      mbar_expect_tx(&bar[slot], (unsigned)(sizeof(T) * G::FB));
      tma_load_3d(ring + slot * FBP, &ym.m[v], i0 - G::HX, j0 - HF, next_issue, &bar[slot]);
    }
  };
  if (tid == 0) issue_upto(plo + NS - 1);

  // closure classes: along xi per point of the pair (its weights kept in registers, one pair of
  // weights per tap), along eta per row (the warp's), along zeta per plane
  W wx[NQ];
  {
    const int cxa = cls_of(min(i, P.nx - 1), P.nx, P.nb);
    if constexpr (N == 2) {
      const int cxb = cls_of(min(i + 1, P.nx - 1), P.nx, P.nb);
#pragma unroll
      for (int o = 0; o < NQ; ++o) wx[o] = make_float2(P.w[cxa][o], i + 1 < P.nx ? P.w[cxb][o] : 0.f);
    } else {
#pragma unroll
      for (int o = 0; o < NQ; ++o) wx[o] = P.w[cxa][o];
    }
  }
  int cy[RY];
  bool inner = true;
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    cy[r] = cls_of(min(j + r, P.ny - 1), P.ny, P.nb);
    inner &= cy[r] == 0;
  }
  const int c = G::HX + N * tx;  // column of the pair's first point in a box row

  // F_xi - I of the pair on one box row (brow: the row's first element); x receives the pair's values
  auto xi = [&](const T* brow, W& x) -> W {
    if constexpr (N == 2) {
      F2 win[NW];
#pragma unroll
      for (int m = 0; m < NW; ++m) win[m] = ld2(brow + c - 2 * HP + 2 * m);
      x = win[HP];
      F2 d = make_float2(0.f, 0.f);
#pragma unroll
      for (int o = -HF; o <= HF; ++o) {
        const int t = o + 2 * HP;  // window position of the first point's tap
        if ((t & 1) == 0) {
          d = fma2(wx[o + HF], win[t >> 1], d);
        } else {
          d.x = fmaf(wx[o + HF].x, win[t >> 1].y, d.x);
          d.y = fmaf(wx[o + HF].y, win[(t >> 1) + 1].x, d.y);
        }
      }
      return d;
    } else {
      x = brow[c];
      T d = T(0);
#pragma unroll
      for (int o = -HF; o <= HF; ++o) d = fmas(wx[o + HF], o == 0 ? x : brow[c + o], d);
      return d;
    }
  };

  // point offsets fit 32 bits (the host checks the block size)
  const unsigned nxy = (unsigned)P.px * (unsigned)P.ny;
  const unsigned lij = (unsigned)i + (unsigned)P.px * (unsigned)j;
  // (the carried error may be read from and written to the same buffer: each point's error is
  // read by its owner before the owner writes the new one)
  const T* errp = P.err[v];
  T* outp = P.out[v];
  T* cmpp = P.comp[v];

  W uq[RY][NQ + U - 1];
#pragma unroll
  for (int r = 0; r < RY; ++r)
#pragma unroll
    for (int q = 0; q < NQ + U - 1; ++q) uq[r][q] = O::zero();
  T* const dme = dsm + RY * ty * TX + N * tx;
  const int pstart = k0 - HF, pend = k1 - 1 + HF;
  int ds = 0;  // ring slot of plane p; advanced below, the slot of plane kf = p - h (h + 1 slots)
  auto plane = [&](const int p, auto S_) -> bool {
    constexpr int S = decltype(S_)::value;  // queue entries S .. S + NQ - 1 hold planes p - 2h .. p
    const int rel = p - plo;  // negative for the planes before the block
    const int kf = p - HF;    // the plane finished at the end of this iteration
    const bool fin = active && kf >= k0 && kf < k1;
    const unsigned lf = lij + nxy * (unsigned)kf;
    W e0[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r)
      e0[r] = COMP && fin && j + r < P.ny ? ld2(errp + lf + r * P.px) : O::zero();
    W u2[RY], d12[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) u2[r] = d12[r] = O::zero();
    if (p >= plo && p <= phi) {
      const int slot = (int)((unsigned)rel % NS);
      const bool ok = mbar_wait(&bar[slot], ((unsigned)rel / NS) & 1u, P.wait_ns);
      // (a thread whose wait gave up reads a box in flight: values only, never used below)
      const T* box = ring + slot * FBP;
      T* u1 = u1s + (rel & 1) * G::U1;
      W d1[RY], u1c[RY];
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        W xc;
        d1[r] = xi(box + (RY * ty + r + HF) * BX, xc);
        u1c[r] = COMP ? add2(xc, d1[r]) : d1[r];
        st2(u1 + (RY * ty + r + HF) * TX + N * tx, u1c[r]);
      }
      // the eta halo rows, one per warp (more than one for half-widths above 4)
#pragma unroll
      for (int r0 = 0; r0 < 2 * HF; r0 += kPairWarps) {
        const int r = r0 + ty;
        if (r < 2 * HF) {
          const int row = r < HF ? r : r + TY;
          W xh;
          const W dh = xi(box + row * BX, xh);
          st2(u1 + row * TX + N * tx, COMP ? add2(xh, dh) : dh);
        }
      }
      // every thread is past plane p - 1 (so the ring slot of plane p - 1 - h, finished there, is
      // free) and has written its part of this plane's u1; the other buffer, read by plane p - 1,
      // is next written at plane p + 1, after the next barrier
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {
          atomicExch(P.errflag, 1);
          // every copy still in flight, the one whose wait gave up included
          for (int w = p; w < next_issue; ++w) mbar_wait(&bar[(w - plo) % NS], (unsigned)(((w - plo) / NS) & 1));
        }
        return false;
      }
      if (tid == 0) issue_upto(p + G::PF);
      // the rows' common window of u1 (their own entries from registers)
      W col[2 * HF + RY];
#pragma unroll
      for (int m = 0; m < 2 * HF + RY; ++m)
        col[m] = m >= HF && m < HF + RY ? u1c[m - HF] : ld2(u1 + (RY * ty + m) * TX + N * tx);
      // (eta and zeta taps as two scalar FMAs whose weight is an operand from the constant bank:
      // a packed FMA would first need the weight copied into both halves of a register pair)
      W dy[RY];
#pragma unroll
      for (int r = 0; r < RY; ++r) dy[r] = O::zero();
      if (inner) {
#pragma unroll
        for (int r = 0; r < RY; ++r)
#pragma unroll
          for (int o = 0; o < NQ; ++o) dy[r] = fmas(P.w[0][o], col[r + o], dy[r]);
      } else {
#pragma unroll
        for (int r = 0; r < RY; ++r)
#pragma unroll
          for (int o = 0; o < NQ; ++o) dy[r] = fmas(P.w[cy[r]][o], col[r + o], dy[r]);
      }
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        u2[r] = COMP ? add2(u1c[r], dy[r]) : dy[r];
        if (COMP) d12[r] = add2(d1[r], dy[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < RY; ++r) uq[r][NQ - 1 + S] = u2[r];
    if (COMP) {
#pragma unroll
      for (int r = 0; r < RY; ++r) st2(dme + ds * G::DP + r * TX, d12[r]);
      ds = ds == HF ? 0 : ds + 1;
    }
    if (!fin) return true;
    const int cz = cls_of(kf, P.nz, P.nb);
    W fz[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) fz[r] = O::zero();
    if (cz == 0) {
#pragma unroll
      for (int r = 0; r < RY; ++r)
#pragma unroll
        for (int o = 0; o < NQ; ++o) fz[r] = fmas(P.w[0][o], uq[r][o + S], fz[r]);
    } else {
#pragma unroll
      for (int r = 0; r < RY; ++r)
#pragma unroll
        for (int o = 0; o < NQ; ++o) fz[r] = fmas(P.w[cz][o], uq[r][o + S], fz[r]);
    }
    // the pre-filter pairs of plane kf, still in its ring slot (kf >= plo)
    const T* xbox = ring + (int)((unsigned)(rel - HF) % NS) * FBP + (RY * ty + HF) * BX + c;
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      if (r > 0 && j + r >= P.ny) break;
      const W x0 = ld2(xbox + r * BX);
      const unsigned lr = lf + (unsigned)(r * P.px);
      if (!COMP) {
        // the one-row kernel's expression, lane by lane
        st2(outp + lr, O::blend(P.blend, x0, fz[r]));
        continue;
      }
      const W D = add2(ld2(dme + ds * G::DP + r * TX), fz[r]);
      const W t = fmas(P.blend, D, e0[r]);
      const W sm = add2(x0, t);
      const W bb = subs(sm, x0);
      const W cm = add2(subs(x0, subs(sm, bb)), subs(t, bb));
      st2(outp + lr, sm);
      st2(cmpp + lr, cm);
    }
    return true;
  };
  for (int p = pstart; p <= pend; p += U) {
    bool ok = true;
    static_for<U>([&](auto S) {
      if (ok && (decltype(S)::value == 0 || p + decltype(S)::value <= pend)) ok = plane(p + decltype(S)::value, S);
    });
    if (!ok) return;
#pragma unroll
    for (int r = 0; r < RY; ++r)
#pragma unroll
      for (int q = 0; q < NQ - 1; ++q) uq[r][q] = uq[r][q + U];
  }
}

template <typename T, int HF, bool COMP>
cudaError_t go_filter_pair(const FieldMaps& in, const TmaFilterParams<T>& p, int tiles, int chunks,
                           cudaStream_t s) {
  const size_t bytes = PairGeo<T, HF>::bytes(COMP);
  static PerDevice smem;
  if (const cudaError_t e = allow_smem(smem, k_filter_pair<T, HF, COMP>, bytes); e != cudaSuccess) return e;
  k_filter_pair<T, HF, COMP><<<dim3(tiles, chunks, p.V), 32 * kPairWarps, bytes, s>>>(in, p);
  return cudaGetLastError();
}

}  // namespace

bool filter_pair_half_width(int hf) { return hf == 2 || hf == 4 || hf == 5; }

void filter_pair_box(size_t esz, int hf, int* bx, int* by, int* tx, int* ty) {
  const int a = 16 / (int)esz;
  *tx = kPairLX * (esz == 4 ? 2 : 1);
  *ty = kPairTY;
  *bx = *tx + 2 * (((hf + a - 1) / a) * a);
  *by = kPairTY + 2 * hf;
}

cudaError_t launch_filter_pair(const FieldMaps& in, const TmaFilterParams<float>& p, int hf, int comp, int tiles,
                               int chunks, cudaStream_t s) {
  if (p.px % 2 != 0 || p.code[0] || (comp && (!p.err[0] || !p.comp[0]))) return cudaErrorInvalidValue;
#define LEE_PAIR_CASE(HF)                                                               \
  if (hf == HF)                                                                         \
    return comp ? go_filter_pair<float, HF, true>(in, p, tiles, chunks, s)              \
                : go_filter_pair<float, HF, false>(in, p, tiles, chunks, s);
  LEE_PAIR_CASE(2)
  LEE_PAIR_CASE(4)
  LEE_PAIR_CASE(5)
#undef LEE_PAIR_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_filter_pair(const FieldMaps& in, const TmaFilterParams<double>& p, int hf, int comp, int tiles,
                               int chunks, cudaStream_t s) {
  if (p.code[0] || comp) return cudaErrorInvalidValue;
  if (hf == 2) return go_filter_pair<double, 2, false>(in, p, tiles, chunks, s);
  if (hf == 4) return go_filter_pair<double, 4, false>(in, p, tiles, chunks, s);
  if (hf == 5) return go_filter_pair<double, 5, false>(in, p, tiles, chunks, s);
  return cudaErrorInvalidValue;
}

}  // namespace lee
