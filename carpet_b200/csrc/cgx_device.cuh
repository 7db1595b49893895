// cgx_device.cuh -- device side of the grid-transfer kernels (sm_100a, FP64).
//
// One descriptor describes one box-pair: a destination region and where its
// sources lie.  A descriptor is cut into tiles; one CTA runs one tile at a
// time.  The same tile routines serve the plain per-box kernel (a grid of the
// pair's tiles) and the persistent batched kernel (tiles taken from a device
// work queue across many pairs).
//
// Arithmetic follows CarpetLib's operation order exactly (see the operator
// families below); FMA selects whether each multiply-add is fused
// (__fma_rn) or rounded twice (__dmul_rn then __dadd_rn).  The intrinsics
// are never contracted by the compiler, so the exact mode is bit-identical
// to the reference built without contraction.
#pragma once
#include <cstddef>
#include <cstdint>
#include <type_traits>
#include <utility>

namespace cgx {

enum Kind : int {
  K_COPY = 0,        // copy_3d (+ time interpolation when ntl > 1)
  K_RESTRICT_VC = 1, // restrict_3d_rf2 (injection)
  K_RESTRICT_CC = 2, // restrict_3d_cc_rf2 (8-point average)
  K_PROLONG_VC = 3,  // prolongate_3d_rf2<ORDER>
  K_PROLONG_CC = 4,  // prolongate_3d_cc_rf2<ORDER>
  K_PROLONG_ENO = 5, // prolongate_3d_real8_eno
  K_RESTRICT_CC3 = 6, // restrict_3d_cc_o3_rf2 (4x4x4 cells)
  K_RESTRICT_CC5 = 7, // restrict_3d_cc_o5_rf2 (6x6x6 cells, separable)
  K_PROLONG_CC_ENO = 8, // prolongate_3d_cc_eno_rf2<ORDER>, ORDER (d.order) 2 or 3
  K_TIME = 9,           // time_interpolate of per-timelevel temporaries
  K_PROLONG_MONO = 10,  // prolongate_3d_o5_monotone_rf2
  K_NKINDS = 11
};

// T_LAG: interpolate_3d_4tl / interpolate_3d_5tl (ntl 4 or 5)
enum TKind : int { T_NONE = 0, T_LIN = 1, T_QUAD = 2, T_ENO = 3, T_LAG = 4 };

// Tile geometry.
constexpr int NTHREADS = 256;
constexpr int NWARPS = NTHREADS / 32;
// prolongation: a tile is ptx fine x (at most PTXMAX) by ptyc coarse rows
// (2*ptyc fine y) by pz fine z, which the CTA marches in stages of bz coarse
// planes.  The shape is chosen per descriptor (prolong_tiles in cgx.cu).
constexpr int PTXMAX = 16;

// 224 bytes: as a kernel parameter with a pointer beside it, a descriptor of 8
// bytes more costs each per-box launch 0.35 us of the host's time (2.30 against
// 2.67 us a launch, parameters of up to 232 bytes and of more).
struct Desc {
  unsigned char kind, order, ntl, tkind;
  int n[3];     // destination region extent (points)
  int soff[3];  // source offset of the region start (meaning per kind)
  int doff[3];  // destination index of the region start
  int sext[3];  // logical extent of the source arrays (load clamp)
  int tiles[2]; // tile grid over the region, x and y
  unsigned char ptx, ptyc; // prolongation tile shape (fine x, coarse y rows)
  unsigned char bx, by, bz; // staged coarse box of a stage: points, rows, planes
  unsigned char tma; // the stages are tensor copies (cgx_tma.cuh)
  // x tile t: fine points t * xw - xo .. (t + 1) * xw - xo - 1; with xs2, two
  // points further in the rows of the other sector alignment (prolong_tiles)
  unsigned char xo, xw;
  short pz; // fine z points of a tile (even)
  unsigned char xs2;
  unsigned char ahead; // copies: fetch the destination with the sources
  int rpx; // ceil(65536 / ptx): t / ptx = t * rpx >> 16 for t < 256
  int ns;  // copies: units per row (Sector), 0: point by point; monotone prolongation: coarse bases per row
  // division magic (div_magic) for ns or n[0], n[1]; prolongation: tiles[0],
  // tiles[1].  Four words on 16 bytes: one load from a descriptor in shared
  // memory.  With the shifts as bytes elsewhere a batch of 64 injections took
  // 7.0 instead of 6.6 us
  unsigned mg[2];
  int sh[2];
  long long ssy, ssz; // source strides (elements) in y and z
  long long dsy, dsz; // destination strides
  const double *src[3];
  double *dst;
  double w[8]; // time weights (layout of the oracle's cgxo_time_weights)
};
static_assert(sizeof(Desc) == 224 && offsetof(Desc, mg) % 16 == 0, "descriptor layout");

// compile-time loop: f(std::integral_constant<int, 0>()) ... f(<N-1>)
template <class Fn, int... I>
__device__ __forceinline__ void static_for_impl(Fn &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>()), ...);
}
template <int N, class Fn> __device__ __forceinline__ void static_for(Fn &&f) {
  static_for_impl(f, std::make_integer_sequence<int, N>());
}

// ---------------------------------------------------------------- arithmetic
template <int FMA> __device__ __forceinline__ double madd(double a, double b, double c) {
  if (FMA)
    return __fma_rn(a, b, c);
  return __dadd_rn(__dmul_rn(a, b), c);
}
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
// madd(a, b, c) for a caller that holds the product ab = mul(a, b)
template <int FMA> __device__ __forceinline__ double term(double a, double b, double ab, double c) {
  return FMA ? __fma_rn(a, b, c) : __dadd_rn(ab, c);
}

// Coefficients as exact dyadic rationals (numerator / 2^k).
// prolongate_3d_rf2.cc:92-124
__device__ __forceinline__ double vc_coeff(int order, int m) {
  switch (order) {
  case 1: return 0.5;
  case 3: { const double c[4] = {-1, 9, 9, -1}; return c[m] * 0.0625; }
  case 5: { const double c[6] = {3, -25, 150, 150, -25, 3}; return c[m] * (1.0 / 256); }
  case 7: { const double c[8] = {-5, 49, -245, 1225, 1225, -245, 49, -5}; return c[m] * (1.0 / 2048); }
  case 9: { const double c[10] = {35, -405, 2268, -8820, 39690, 39690, -8820, 2268, -405, 35};
            return c[m] * (1.0 / 65536); }
  default: { const double c[12] = {-63, 847, -5445, 22869, -76230, 320166,
                                    320166, -76230, 22869, -5445, 847, -63};
             return c[m] * (1.0 / 524288); }
  }
}
// prolongate_3d_cc_rf2.cc:116-139; di == 1 reverses the stencil (:67)
__device__ __forceinline__ double cc_coeff(int order, int di, int m) {
  int n = order + 1;
  int j = di ? n - 1 - m : m;
  switch (order) {
  case 0: return 1.0;
  case 1: { const double c[2] = {1, 3}; return c[j] * 0.25; }
  case 2: { const double c[3] = {5, 30, -3}; return c[j] * (1.0 / 32); }
  case 3: { const double c[4] = {-5, 35, 105, -7}; return c[j] * (1.0 / 128); }
  case 4: { const double c[5] = {-45, 420, 1890, -252, 35}; return c[j] * (1.0 / 2048); }
  default: { const double c[6] = {63, -495, 2310, 6930, -693, 77}; return c[j] * (1.0 / 8192); }
  }
}

// ---------------------------------------------------------------- families
// A family is a separable 1-D rule: the fine point with source position s
// (fine units) has coarse base c = s >> 1 and parity p = s & 1; its value on
// one axis is a function of the coarse values around c.  [LO, HI] is the
// union of the windows of both parities relative to c.  CarpetLib nests the
// axes as interp3(z) of interp2(y) of interp1(x), so the separable passes
// x -> y -> z reproduce its arithmetic exactly.

// A family evaluates its rule in two forms.  first/next take the window of
// one fine point at once (get(m): the coarse value at base + m).  Line takes
// the coarse values of a line one after another: push(v) hands it the value
// at index j and returns the parity-0 fine value of base j - D0 and the
// parity-1 value of base j - D1.  The linear families hold no window for it
// but the partial sums of the N - 1 fine points still open: each new value
// adds its term to every one of them, which is the reference's own
// left-to-right order of every sum.  The terms of one push are independent
// of each other (a window form chains them), a coefficient that stands twice
// in the stencil costs one product per coarse value instead of two per fine
// point (in the two-rounding mode, 9 instead of 12 operations of order 5).
// A sum stays in its register from its first term to its last: push<U> is
// the push of phase U = (values pushed before) % PHASES.  Values of a sum opened before the
// line's first point are never read; a caller that knows which of a line's
// sums it will read gives them as Open, and the others are not formed.
// FIRST selects the x pass's form of the sum (first).

// The push of value j of a line adds to the sum opened at value j - k its
// term k; sums opened at values lo .. hi-1 are wanted.
struct Open {
  int j = 1 << 20, lo = 0, hi = 1 << 30;
  __device__ constexpr bool has(int k) const { return j - k >= lo && j - k < hi; }
};

// vertex-centred Lagrange, prolongate_3d_rf2.cc:151-295
template <int ORDER> struct VC {
  static constexpr int N = ORDER + 1;
  static constexpr int LO = -(N / 2) + 1; // coeffs1d::imin
  static constexpr int HI = LO + N - 1;
  // x pass (interp1, :157-259, scalar Vectors order): vres = c0*p0;
  // vres = madd(c_m, p_m, vres); res = 0 + vres.  p points at coarse c.
  template <int FMA, class G> __device__ __forceinline__ static double first(int par, G get) {
    if (!par) return get(0); // interp0: no arithmetic
    double v = mul(vc_coeff(ORDER, 0), get(LO));
#pragma unroll
    for (int m = 1; m < N; ++m) v = madd<FMA>(vc_coeff(ORDER, m), get(LO + m), v);
    return add(0.0, v);
  }
  // y and z passes (interp2/interp3, :262-295): res = 0; res += c_m*v_m
  template <int FMA, class G> __device__ __forceinline__ static double next(int par, G get) {
    if (!par) return get(0);
    double r = 0.0;
#pragma unroll
    for (int m = 0; m < N; ++m) r = madd<FMA>(vc_coeff(ORDER, m), get(LO + m), r);
    return r;
  }
  static constexpr int D0 = 0, D1 = HI, PHASES = N - 1;
  template <int FMA, bool FIRST> struct Line {
    double a[N - 1] = {};
    template <int U>
    __device__ __forceinline__ void push(double v, double &o0, double &o1, Open w = {}) {
      double p[N]; // the stencil is symmetric
#pragma unroll
      for (int k = 0; k < N; ++k) p[k] = k < N / 2 ? mul(vc_coeff(ORDER, k), v) : p[N - 1 - k];
      o0 = v;
      if (w.has(N - 1)) {
        const double r = term<FMA>(vc_coeff(ORDER, N - 1), v, p[N - 1], a[U]);
        o1 = FIRST ? add(0.0, r) : r;
      }
#pragma unroll
      for (int k = N - 2; k >= 1; --k)
        if (w.has(k)) {
          double &s = a[(U + N - 1 - k) % (N - 1)];
          s = term<FMA>(vc_coeff(ORDER, k), v, p[k], s);
        }
      if (w.has(0)) a[U] = FIRST ? p[0] : term<FMA>(vc_coeff(ORDER, 0), v, p[0], 0.0);
    }
  };
};

// cell-centred Lagrange, prolongate_3d_cc_rf2.cc:150-195: every axis is
// interpolated, res = 0; res += c_m*v_m, with a parity-dependent window
template <int ORDER> struct CC {
  static constexpr int N = ORDER + 1;
  static constexpr int LO0 = -N / 2;
  static constexpr int LO1 = -N / 2 + (ORDER % 2 != 0 ? 1 : 0);
  static constexpr int LO = LO0;
  static constexpr int HI = LO1 + N - 1;
  template <int FMA, class G> __device__ __forceinline__ static double next(int par, G get) {
    double r = 0.0;
    if (!par) {
#pragma unroll
      for (int m = 0; m < N; ++m) r = madd<FMA>(cc_coeff(ORDER, 0, m), get(LO0 + m), r);
    } else {
#pragma unroll
      for (int m = 0; m < N; ++m) r = madd<FMA>(cc_coeff(ORDER, 1, m), get(LO1 + m), r);
    }
    return r;
  }
  template <int FMA, class G> __device__ __forceinline__ static double first(int par, G get) {
    return next<FMA>(par, get);
  }
  static constexpr int D0 = LO0 + N - 1, D1 = HI, PHASES = N > 1 ? N - 1 : 1;
  template <int FMA, bool FIRST> struct Line {
    double a[2][PHASES] = {};
    template <int U>
    __device__ __forceinline__ void push(double v, double &o0, double &o1, Open w = {}) {
      double p[2][N], o[2] = {0.0, 0.0}; // the two parities' stencils mirror each other
#pragma unroll
      for (int k = 0; k < N; ++k) p[0][k] = p[1][N - 1 - k] = mul(cc_coeff(ORDER, 0, k), v);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (q) w.j -= LO1 - LO0; // parity 1's windows start that much further
        if (w.has(N - 1)) o[q] = term<FMA>(cc_coeff(ORDER, q, N - 1), v, p[q][N - 1], N > 1 ? a[q][U] : 0.0);
#pragma unroll
        for (int k = N - 2; k >= 1; --k)
          if (w.has(k)) {
            double &s = a[q][(U + N - 1 - k) % PHASES];
            s = term<FMA>(cc_coeff(ORDER, q, k), v, p[q][k], s);
          }
        if (N > 1 && w.has(0)) a[q][U] = term<FMA>(cc_coeff(ORDER, q, 0), v, p[q][0], 0.0);
      }
      o0 = o[0];
      o1 = o[1];
    }
  };
};

// The limited families are not sums: their Line holds the window's earlier
// values and evaluates both parities of base j - HI.
template <class F, int FMA> struct WindowLine {
  static constexpr int M = F::HI - F::LO;
  double a[M] = {};
  template <int U> __device__ __forceinline__ void push(double v, double &o0, double &o1, Open = {}) {
    auto get = [&](int m) { return m == F::HI ? v : a[m - F::LO]; };
    o0 = F::template next<FMA>(0, get);
    o1 = F::template next<FMA>(1, get);
#pragma unroll
    for (int k = 0; k + 1 < M; ++k) a[k] = a[k + 1];
    a[M - 1] = v;
  }
};

// vertex-centred ENO, prolongate_3d_real8_eno.F90:23-76 (eno1d) and the
// x -> y -> z nesting of :195-285
struct ENO {
  static constexpr int LO = -1, HI = 2;
  template <int FMA>
  __device__ __forceinline__ static double eno1d(double q1, double q2, double q3, double q4) {
    double dl = __dsub_rn(__dadd_rn(q1, q3), __dmul_rn(2.0, q2));
    double dr = __dsub_rn(__dadd_rn(q2, q4), __dmul_rn(2.0, q3));
    double r;
    if (fabs(dl) < fabs(dr)) {
      // eighth * (-q(1) + six * q(2) + three * q(3))
      double t = FMA ? __fma_rn(6.0, q2, -q1) : __dadd_rn(-q1, __dmul_rn(6.0, q2));
      t = madd<FMA>(3.0, q3, t);
      r = __dmul_rn(0.125, t);
    } else {
      // eighth * (three * q(2) + six * q(3) - q(4))
      double t = madd<FMA>(3.0, q2, __dmul_rn(6.0, q3));
      t = __dsub_rn(t, q4);
      r = __dmul_rn(0.125, t);
    }
    if (__dmul_rn(__dsub_rn(r, q2), __dsub_rn(q3, r)) < 0.0 || __dmul_rn(dl, dr) <= 0.0)
      r = __dmul_rn(0.5, __dadd_rn(q2, q3));
    return r;
  }
  template <int FMA, class G> __device__ __forceinline__ static double next(int par, G get) {
    if (!par) return get(0);
    return eno1d<FMA>(get(-1), get(0), get(1), get(2));
  }
  template <int FMA, class G> __device__ __forceinline__ static double first(int par, G get) {
    return next<FMA>(par, get);
  }
  static constexpr int D0 = HI, D1 = HI, PHASES = 1;
  template <int FMA, bool FIRST> struct Line : WindowLine<ENO, FMA> {};
};

// cell-centred ENO, prolongate_3d_cc_eno_rf2.cc:198-400 (interp1, interp2
// and interp3 apply the same rule on their axis).  Relative to the coarse
// base c, the fine point of parity DI reads f(-W+DI) .. f(W-1+DI), W = ORDER.
// coeffs1dc<RT,ORDER,OFFSET> (:144-176) as exact dyadic rationals; table t:
// 0 <1,0>, 1 <2,0>, 2 <2,-1>, 3 <3,0>, 4 <3,+1>, 5 <3,-1>.
__device__ __forceinline__ constexpr double ceno_coeff(int t, int j) {
  return t == 0 ? (j == 0 ? 1.0 : 3.0) / 4
       : t == 1 ? (j == 0 ? 5.0 : j == 1 ? 30.0 : -3.0) / 32
       : t == 2 ? (j == 0 ? -3.0 : j == 1 ? 14.0 : 21.0) / 32
       : t == 3 ? (j == 0 ? -5.0 : j == 1 ? 35.0 : j == 2 ? 105.0 : -7.0) / 128
       : t == 4 ? (j == 0 ? 15.0 : j == 1 ? 135.0 : j == 2 ? -27.0 : 5.0) / 128
                : (j == 0 ? 7.0 : j == 1 ? -33.0 : 77.0) / 128;
}
template <int ORDER> struct CCENO {
  static_assert(ORDER == 2 || ORDER == 3, "cell-centred ENO orders 2 and 3");
  static constexpr int LO = -ORDER, HI = ORDER;
  // coeffs1d::get summed from imin: res = 0; res += c*f (reversed for DI=1)
  template <int FMA, int DI, int T, int N, int IMIN, class G>
  __device__ __forceinline__ static double sum(G get) {
    double r = 0.0;
    static_for<N>([&](auto M) {
      constexpr int m = decltype(M)::value;
      r = madd<FMA>(ceno_coeff(T, DI == 0 ? m : N - 1 - m), get(IMIN + m), r);
    });
    return r;
  }
  // undivided differences (diffC1dc, :171-174; never reversed)
  template <int FMA, int IMIN, class G> __device__ __forceinline__ static double diff(G get) {
    double r = 0.0;
    static_for<ORDER + 1>([&](auto M) {
      constexpr int m = decltype(M)::value;
      constexpr double c = ORDER == 2 ? (m == 1 ? -2.0 : 1.0)
                                      : (m == 0 ? 1.0 : m == 1 ? -3.0 : m == 2 ? 3.0 : -1.0);
      r = madd<FMA>(c, get(IMIN + m), r);
    });
    return r;
  }
  template <int FMA, int DI, class G> __device__ __forceinline__ static double rule(G get) {
    const double first = sum<FMA, DI, 0, 2, -1 + DI>(get); // coeffs1d<RT,1,di,0>
    double res;
    if (ORDER == 2) {
      constexpr int SH = DI == 0 ? -1 : 1; // :225-231
      const double lV = diff<FMA, -1 + SH>(get), rV = diff<FMA, -1>(get);
      if (__dmul_rn(lV, rV) <= 0.0) res = first;
      else if (fabs(lV) < fabs(rV)) res = sum<FMA, DI, 2, 3, -1 + SH>(get);
      else res = sum<FMA, DI, 1, 3, -1>(get);
    } else {
      const double V0 = diff<FMA, -3 + DI>(get), V1 = diff<FMA, -2 + DI>(get),
                   V2 = diff<FMA, -1 + DI>(get);
      if (__dmul_rn(V0, V2) <= 0.0 || __dmul_rn(V0, V1) <= 0.0 || __dmul_rn(V1, V2) <= 0.0)
        return first; // :311-329, without the final test
      int mn = 1;
      if (fabs(V0) < fabs(V1)) mn = 0;
      if (fabs(V2) < fabs(mn == 0 ? V0 : V1)) mn = 2;
      // coeffs1dc<3, di == 0 ? OFFSET : -OFFSET> for OFFSET -1, 0, +1
      if (mn == 0) res = sum<FMA, DI, DI == 0 ? 5 : 4, 4, -3 + DI>(get);
      else if (mn == 1) res = sum<FMA, DI, 3, 4, -2 + DI>(get);
      else res = sum<FMA, DI, DI == 0 ? 4 : 5, 4, -1 + DI>(get);
    }
    // :366-395: a result outside the two nearest values falls back
    if (__dmul_rn(__dsub_rn(res, get(DI - 1)), __dsub_rn(get(DI), res)) < 0.0) res = first;
    return res;
  }
  template <int FMA, class G> __device__ __forceinline__ static double next(int par, G get) {
    return par ? rule<FMA, 1>(get) : rule<FMA, 0>(get);
  }
  template <int FMA, class G> __device__ __forceinline__ static double first(int par, G get) {
    return next<FMA>(par, get);
  }
  static constexpr int D0 = HI, D1 = HI, PHASES = 1;
  template <int FMA, bool FIRST> struct Line : WindowLine<CCENO<ORDER>, FMA> {};
};

// ---------------------------------------------------------------- time
// interpolate_3d_2tl.cc:248-249, interpolate_3d_3tl.cc:388-390,
// interpolate_eno_3d_3tl.cc:145-162.  The fused order contracts
// s1*a + s2*b as fma(s1, a, s2*b), then + s3*c as fma(s3, c, .).
template <int FMA> __device__ __forceinline__ double tcomb2(double s1, double a, double s2, double b) {
  if (FMA) return __fma_rn(s1, a, __dmul_rn(s2, b));
  return __dadd_rn(__dmul_rn(s1, a), __dmul_rn(s2, b));
}
template <int FMA, int TK, int NTL>
__device__ __forceinline__ double tcombine(const double *w, const double *v) {
  if (NTL == 1) return v[0];
  if (TK == T_LIN) return tcomb2<FMA>(w[0], v[0], w[1], v[1]);
  double d = madd<FMA>(w[2], v[2], tcomb2<FMA>(w[0], v[0], w[1], v[1]));
  if (TK == T_ENO) {
    double a = v[0], b = v[1], c = v[2];
    double mx = b < c ? c : b; mx = a < mx ? mx : a; // std::max nesting
    double mn = c < b ? c : b; mn = mn < a ? mn : a; // std::min nesting
    if (d > mx || d < mn)
      d = w[7] != 0.0 ? tcomb2<FMA>(w[3], a, w[4], b) : tcomb2<FMA>(w[5], b, w[6], c);
  }
  return d;
}

// ---------------------------------------------------------------- cp.async
__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- copy-like
// copy_3d (copy_3d.cc:113-121) with optional time interpolation of the
// copied timelevels (transfer_time with equal strides, data.cc:506-517),
// restrict_3d_rf2 (restrict_3d_rf2.cc:102-108) and restrict_3d_cc_rf2
// (restrict_3d_cc_rf2.cc:246-262).  soff is the source index of the region
// start; the restrictions step by 2 in the source.
//
// These are pure streaming operations on regions of any shape -- ghost
// zones are 3 points thin in one direction.  A tile is STILE consecutive
// points of the region flattened x-fastest, run by the LANES threads of a
// CTA: every lane is busy whatever the shape, consecutive lanes touch
// consecutive x, and each thread issues a group of loads before its stores.
// A flat index is split into (i, j, k) by 32-bit multiply-high with
// precomputed magic numbers.
//
// Copies whose rows have SECTOR_ROW points or more go by destination sectors
// (32 bytes; d.ns): two threads take two neighbouring sectors, each thread
// one half of either, so that a warp's two 16-byte stores cover whole sectors
// -- L2 fetches the rest of a sector that a store covers in part from DRAM --
// and an index is split once for four points: of 60 instructions per point
// the point-by-point form spent most on that, and half of the issue slots.  A
// tile is then STILE / 4 threads' worth.  They are kernels of their own: in
// one kernel with the point form, inlined or as calls, the latter lost its
// eight loads in flight (211 -> 260 to 373 us).
constexpr int STILE = 1024;
constexpr int SECTOR_ROW = 16; // narrower rows have hardly a whole sector
// The kinds that compute much per point (8 to 216 source values) take tiles
// of HTILE units, one or two per thread: their regions are small (a coarse
// patch of 20^3 points is 8 tiles of 1024) and eight points of a thread ran
// one after another on a GPU two thirds idle.
constexpr int HTILE = 256;

// The streaming kinds, one persistent kernel each.
enum StreamVariant : int {
  SV_COPY1 = 0,       // copy, one timelevel
  SV_COPY2 = 1,       // copy, linear time interpolation
  SV_COPY3Q = 2,      // copy, quadratic time interpolation
  SV_COPY3E = 3,      // copy, ENO time interpolation
  SV_RESTRICT_VC = 4, // injection
  SV_RESTRICT_CC = 5, // 8-point average
  SV_RESTRICT_CC3 = 6, // third-order cell-centred restriction
  SV_RESTRICT_CC5 = 7, // fifth-order cell-centred restriction
  SV_MONO = 8,         // monotone order-5 prolongation
  SV_SECTOR = 9,       // the four copies by destination sectors (d.ns), in the order above
  SV_TIME = 13,        // time combination of temporaries (K_TIME)
  SV_COUNT = 14
};
// A batch launches its segments in order: the time combination of staged
// transfers must come after every kind that writes their temporaries.
static_assert(SV_TIME == SV_COUNT - 1, "the time combination is the last streaming variant");

template <class D> __host__ __device__ __forceinline__ int stream_variant(const D &d) {
  if (d.kind == K_RESTRICT_VC) return SV_RESTRICT_VC;
  if (d.kind == K_RESTRICT_CC) return SV_RESTRICT_CC;
  if (d.kind == K_RESTRICT_CC3) return SV_RESTRICT_CC3;
  if (d.kind == K_RESTRICT_CC5) return SV_RESTRICT_CC5;
  if (d.kind == K_TIME) return SV_TIME;
  if (d.kind == K_PROLONG_MONO) return SV_MONO;
  if (d.kind != K_COPY) return -1;
  return (d.ns ? SV_SECTOR : SV_COPY1) + (d.ntl == 1 ? 0 : d.ntl == 2 ? 1 : d.tkind == T_ENO ? 3 : 2);
}

// Source loads of the streaming tiles: through the read-only path (__ldg)
// in kernels whose sources no CTA of the same launch writes; cached in L2
// only (__ldcg, coherent across SMs) in the chain kernel, whose later tiles
// read what earlier tiles of the same launch wrote.
template <bool CG> __device__ __forceinline__ double ld_src(const double *p) {
  if (CG) return __ldcg(p);
  return __ldg(p);
}

// floor(p / n) for 0 <= p < 2^31 (Granlund & Montgomery, "Division by
// invariant integers using multiplication", 1994, theorem 4.2 with N = 31):
// with l = ceil(log2 n), m = ceil(2^(31+l) / n) < 2^32 and s = l - 1,
// floor(p / n) = umulhi(p, m) >> s; m = 0 encodes n = 1.
__device__ __forceinline__ unsigned div_magic(unsigned p, unsigned m, int s) {
  return m ? (__umulhi(p, m) >> s) : p;
}

template <class D>
__device__ __forceinline__ void unflatten(const D &d, unsigned p, int &i, int &j, int &k) {
  const unsigned q = div_magic(p, d.mg[0], d.sh[0]);
  i = (int)(p - q * (unsigned)d.n[0]);
  const unsigned r = div_magic(q, d.mg[1], d.sh[1]);
  j = (int)(q - r * (unsigned)d.n[1]);
  k = (int)r;
}

// Unit p of the region's destination rows, the rows' first and last sectors
// whole: its row, and the x (-3 .. n[0] + 4) of its first half sector, which
// starts on 16 bytes; the other half lies four points further.
struct Sector {
  int x, j, k;
};
template <class D> __device__ __forceinline__ Sector sector(const D &d, unsigned p, const double *dst) {
  const unsigned q = div_magic(p, d.mg[0], d.sh[0]), r = div_magic(q, d.mg[1], d.sh[1]);
  Sector s;
  s.j = (int)(q - r * (unsigned)d.n[1]);
  s.k = (int)r;
  const unsigned at = (unsigned)(reinterpret_cast<uintptr_t>(dst) >> 3) + (unsigned)s.j * (unsigned)d.dsy +
                      (unsigned)s.k * (unsigned)d.dsz;
  const int u = (int)(p - q * (unsigned)d.ns);
  s.x = 8 * (u >> 1) + 2 * (u & 1) - (int)(at & 3u);
  return s;
}
// stores the points of a half sector that lie in the region; o: its first one
__device__ __forceinline__ void store_half(double *o, int x, int n, double a, double b) {
  if (x >= 0 && x + 1 < n) {
    *reinterpret_cast<double2 *>(o) = make_double2(a, b);
  } else {
    if (x >= 0 && x < n) o[0] = a;
    if (x + 1 >= 0 && x + 1 < n) o[1] = b;
  }
}
// the source points of a half sector from s + x, those outside the row
// replaced by its end points; one load where they start on 16 bytes too
__device__ __forceinline__ void load_half(const double *s, int x, int n, double &a, double &b) {
  if (x >= 0 && x + 1 < n && (reinterpret_cast<uintptr_t>(s + x) & 15) == 0) {
    const double2 v = __ldg(reinterpret_cast<const double2 *>(s + x));
    a = v.x;
    b = v.y;
  } else {
    a = __ldg(s + min(max(x, 0), n - 1));
    b = __ldg(s + min(max(x + 1, 0), n - 1));
  }
}

template <int FMA, int NTL, int TK, int LANES, class D>
__device__ __forceinline__ void copy_sectors(const D &d, int tile, int lid) {
  constexpr int PER = STILE / 4 / LANES, G = NTL == 1 ? PER : 1; // units whose loads are issued before their stores
  const unsigned nunits = (unsigned)d.ns * d.n[1] * d.n[2], p0 = (unsigned)tile * (STILE / 4) + lid;
  const long long so = d.soff[0] + d.soff[1] * d.ssy + d.soff[2] * d.ssz;
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
  double w[NTL == 1 ? 1 : 8];
#pragma unroll
  for (int k = 0; k < (NTL == 1 ? 1 : 8); ++k) w[k] = NTL == 1 ? 0.0 : d.w[k];
#pragma unroll 1
  for (int r0 = 0; r0 < PER; r0 += G) {
    double v[G][NTL][4];
    Sector c[G];
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < nunits) {
        c[r] = sector(d, p, dst);
        const long long row = so + c[r].j * d.ssy + c[r].k * d.ssz;
#pragma unroll
        for (int t = 0; t < NTL; ++t)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            load_half(d.src[t] + row, c[r].x + 4 * h, d.n[0], v[r][t][2 * h], v[r][t][2 * h + 1]);
      }
    }
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < nunits) {
        double o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          double u[NTL];
#pragma unroll
          for (int t = 0; t < NTL; ++t) u[t] = v[r][t][e];
          o[e] = tcombine<FMA, TK, NTL>(w, u);
        }
        double *out = dst + (c[r].x + c[r].j * d.dsy + c[r].k * d.dsz);
#pragma unroll
        for (int h = 0; h < 2; ++h) store_half(out + 4 * h, c[r].x + 4 * h, d.n[0], o[2 * h], o[2 * h + 1]);
      }
    }
  }
}

template <int FMA, int NTL, int TK, int LANES, class D, bool CG = false, int PTS = STILE, int GMAX = 8>
__device__ __forceinline__ void copy_tile(const D &d, int tile, int lid) {
  // ENO time interpolation holds more per point: smaller groups
  constexpr int PER = PTS / LANES;
  constexpr int G0 = PER < (NTL == 1 ? GMAX : 4) ? PER : (NTL == 1 ? GMAX : 4);
  constexpr int G = G0 / (TK == T_ENO ? 2 : 1);
  const unsigned npts = (unsigned)d.n[0] * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * PTS + lid;
  // the pieces of a row that a warp stores start and end inside sectors, whose
  // rest L2 fetches from DRAM as the store arrives: the destination fetched
  // with the sources instead
  const bool ahead = d.ahead;
  const double *src[NTL];
#pragma unroll
  for (int t = 0; t < NTL; ++t) src[t] = d.src[t] + (d.soff[0] + d.soff[1] * d.ssy + d.soff[2] * d.ssz);
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
  double w[NTL == 1 ? 1 : 8];
#pragma unroll
  for (int k = 0; k < (NTL == 1 ? 1 : 8); ++k) w[k] = NTL == 1 ? 0.0 : d.w[k];
#pragma unroll
  for (int r0 = 0; r0 < PER; r0 += G) {
    double v[G][NTL];
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < npts) {
        int i, j, k;
        unflatten(d, p, i, j, k);
        const long long si = i + j * d.ssy + k * d.ssz;
#pragma unroll
        for (int t = 0; t < NTL; ++t) v[r][t] = ld_src<CG>(src[t] + si);
        if (ahead) asm volatile("prefetch.global.L2 [%0];" ::"l"(dst + (i + j * d.dsy + k * d.dsz)));
      }
    }
    // the destination index is recomputed rather than held across the loads
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < npts) {
        int i, j, k;
        unflatten(d, p, i, j, k);
        dst[i + j * d.dsy + k * d.dsz] = tcombine<FMA, TK, NTL>(w, v[r]);
      }
    }
  }
}

template <int LANES, class D, bool CG = false, int PTS = STILE, int GMAX = 8>
__device__ __forceinline__ void restrict_vc_tile(const D &d, int tile, int lid) {
  constexpr int PER = PTS / LANES, G = PER < GMAX ? PER : GMAX;
  const unsigned npts = (unsigned)d.n[0] * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * PTS + lid;
  const double *s = d.src[0] + (d.soff[0] + d.soff[1] * d.ssy + d.soff[2] * d.ssz);
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
#pragma unroll
  for (int r0 = 0; r0 < PER; r0 += G) {
    double v[G];
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < npts) {
        int i, j, k;
        unflatten(d, p, i, j, k);
        v[r] = ld_src<CG>(s + 2 * (i + j * d.ssy + k * d.ssz));
      }
    }
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const unsigned p = p0 + (r0 + r) * LANES;
      if (p < npts) {
        int i, j, k;
        unflatten(d, p, i, j, k);
        dst[i + j * d.dsy + k * d.dsz] = v[r];
      }
    }
  }
}

template <int FMA, int LANES, class D>
__device__ __forceinline__ void restrict_cc_tile(const D &d, int tile, int lid) {
  constexpr int PER = HTILE / LANES;
  const unsigned npts = (unsigned)d.n[0] * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * HTILE + lid;
  const double *s0 = d.src[0] + (d.soff[0] + d.soff[1] * d.ssy + d.soff[2] * d.ssz);
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
  const long long ssy = d.ssy, ssz = d.ssz;
  const double w = 0.125; // f1*f1*f1 with f1 = f2 = 1/2
  // the two x neighbours in one load where every row starts on 16 bytes
  const bool pairs = ((reinterpret_cast<uintptr_t>(s0) | (uintptr_t)(8 * ssy) | (uintptr_t)(8 * ssz)) & 15) == 0;
#pragma unroll 2
  for (int r = 0; r < PER; ++r) {
    const unsigned p = p0 + r * LANES;
    if (p >= npts) break;
    int i, j, k;
    unflatten(d, p, i, j, k);
    const double *q = s0 + 2 * (i + j * ssy + k * ssz);
    auto pair = [&](const double *u) {
      return pairs ? __ldg(reinterpret_cast<const double2 *>(u)) : make_double2(__ldg(u), __ldg(u + 1));
    };
    const double2 b0 = pair(q), b1 = pair(q + ssy), b2 = pair(q + ssz), b3 = pair(q + ssy + ssz);
    const double a0 = b0.x, a1 = b0.y, a2 = b1.x, a3 = b1.y, a4 = b2.x, a5 = b2.y, a6 = b3.x, a7 = b3.y;
    // order of restrict_3d_cc_rf2.cc:253-260
    double res = mul(w, a0);
    res = madd<FMA>(w, a1, res);
    res = madd<FMA>(w, a2, res);
    res = madd<FMA>(w, a3, res);
    res = madd<FMA>(w, a4, res);
    res = madd<FMA>(w, a5, res);
    res = madd<FMA>(w, a6, res);
    res = madd<FMA>(w, a7, res);
    dst[i + j * d.dsy + k * d.dsz] = res;
  }
}

// The second stage of transfer_time (data.cc:506-517) where the fused
// kernels do not apply: d.src[0] holds d.ntl temporaries of the region's
// shape, one after another, x fastest and unpadded; time_interpolate
// (data.cc:1183-1299) combines them into the destination.  4 and 5
// timelevels sum s1*a + s2*b + s3*c + s4*d (+ s5*e) left to right
// (interpolate_3d_4tl.cc:126-131, interpolate_3d_5tl.cc:128-132).
template <int FMA, int LANES, class D>
__device__ __forceinline__ void time_tile(const D &d, int tile, int lid) {
  constexpr int PER = STILE / LANES;
  const unsigned npts = (unsigned)d.n[0] * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * STILE + lid;
  const double *tmp = d.src[0];
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
  const int ntl = d.ntl, tk = d.tkind;
  double w[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) w[k] = d.w[k];
#pragma unroll 2
  for (int r = 0; r < PER; ++r) {
    const unsigned p = p0 + r * LANES;
    if (p >= npts) break;
    double v[5];
#pragma unroll
    for (int t = 0; t < 5; ++t) v[t] = t < ntl ? __ldg(tmp + (size_t)t * npts + p) : 0.0;
    double res;
    if (ntl == 2) res = tcombine<FMA, T_LIN, 2>(w, v);
    else if (ntl == 3 && tk == T_ENO) res = tcombine<FMA, T_ENO, 3>(w, v);
    else {
      res = tcombine<FMA, T_QUAD, 3>(w, v);
      if (ntl >= 4) res = madd<FMA>(w[3], v[3], res);
      if (ntl == 5) res = madd<FMA>(w[4], v[4], res);
    }
    int i, j, k;
    unflatten(d, p, i, j, k);
    dst[i + j * d.dsy + k * d.dsz] = res;
  }
}

// prolongate_3d_o5_monotone_rf2 (prolongate_3d_o5_monotone_rf2.cc:45-793),
// one fine point per lane.  q points at the coarse base; odd axes take the
// tensor-product order-5 stencil over coarse -2 .. +3, summed left to right
// with the lowest odd axis fastest (weights f_a * f_b * f_c formed left to
// right); with three odd axes every z plane is a partial sum of its own and
// the six are added in order (:499-716).  A result outside the nearest 2/4/8
// coarse values (std::min/std::max nested as min4/max4/min8/max8, :19-43)
// falls back to linear, bilinear or trilinear interpolation.
__device__ __forceinline__ double smin(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return a < b ? b : a; }
__device__ __forceinline__ constexpr double mono_f(int m) {
  return (m == 0 || m == 5 ? 3.0 : m == 1 || m == 4 ? -25.0 : 150.0) / 256;
}
template <int FMA>
__device__ __forceinline__ double mono_point(const double *q, int ox, int oy, int oz, long long sy,
                                             long long sz) {
  const int n = ox + oy + oz;
  if (n == 0) return __ldg(q);
  if (n == 1) {
    const long long s = ox ? 1 : oy ? sy : sz;
    double res = mul(mono_f(0), __ldg(q - 2 * s));
#pragma unroll
    for (int m = 1; m < 6; ++m) res = madd<FMA>(mono_f(m), __ldg(q + (m - 2) * s), res);
    const double v0 = __ldg(q), v1 = __ldg(q + s);
    if (res > smax(v0, v1) || res < smin(v0, v1)) res = madd<FMA>(0.5, v1, mul(0.5, v0));
    return res;
  }
  if (n == 2) {
    const long long s0 = ox ? 1 : sy, s1 = oz ? sz : sy;
    double res = 0.0;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
      const double *row = q + (b - 2) * s1 - 2 * s0;
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        const double w = mono_f(a) * mono_f(b);
        const double v = __ldg(row + a * s0);
        res = (a == 0 && b == 0) ? mul(w, v) : madd<FMA>(w, v, res);
      }
    }
    const double x1 = __ldg(q), x2 = __ldg(q + s0), x3 = __ldg(q + s1), x4 = __ldg(q + s0 + s1);
    if (res > smax(smax(x1, x2), smax(x3, x4)) || res < smin(smin(x1, x2), smin(x3, x4))) {
      res = mul(0.25, x1);
      res = madd<FMA>(0.25, x2, res);
      res = madd<FMA>(0.25, x3, res);
      res = madd<FMA>(0.25, x4, res);
    }
    return res;
  }
  double res = 0.0;
#pragma unroll 1
  for (int c = 0; c < 6; ++c) {
    const double fc = (c == 0 || c == 5) ? mono_f(0) : (c == 1 || c == 4) ? mono_f(1) : mono_f(2);
    const double *pl = q + (c - 2) * sz;
    double r = 0.0;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
      const double *row = pl + (b - 2) * sy - 2;
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        const double w = __dmul_rn(mono_f(a) * mono_f(b), fc);
        const double v = __ldg(row + a);
        r = (a == 0 && b == 0) ? mul(w, v) : madd<FMA>(w, v, r);
      }
    }
    res = c == 0 ? r : add(res, r);
  }
  // max8 / min8 of (0,0,0), (1,0,0), (0,1,0), (0,0,1), (1,1,0), (1,0,1), (0,1,1), (1,1,1)
  const double x0 = __ldg(q), x1 = __ldg(q + 1), x2 = __ldg(q + sy), x3 = __ldg(q + sz);
  const double x4 = __ldg(q + 1 + sy), x5 = __ldg(q + 1 + sz), x6 = __ldg(q + sy + sz);
  const double x7 = __ldg(q + 1 + sy + sz);
  const double mx = smax(smax(smax(x0, x1), smax(x2, x3)), smax(smax(x4, x5), smax(x6, x7)));
  const double mn = smin(smin(smin(x0, x1), smin(x2, x3)), smin(smin(x4, x5), smin(x6, x7)));
  if (res > mx || res < mn) {
    // :730-738: the z = 0 plane, then the z = 1 plane, x fastest
    double r1 = mul(0.125, x0);
    r1 = madd<FMA>(0.125, x1, r1);
    r1 = madd<FMA>(0.125, x2, r1);
    r1 = madd<FMA>(0.125, x4, r1);
    double r2 = mul(0.125, x3);
    r2 = madd<FMA>(0.125, x5, r2);
    r2 = madd<FMA>(0.125, x6, r2);
    r2 = madd<FMA>(0.125, x7, r2);
    res = add(r1, r2);
  }
  return res;
}

// A unit is one coarse base of a fine row, both of its fine points (neighbours
// in the destination).  Rows are taken by parity, all even fine y before all
// odd ones and the same in z, so that the threads of a warp evaluate the same
// stencil (but at the seams) and consecutive lanes consecutive coarse points:
// point by point in fine order a warp ran every one of its rows' stencils for
// both x parities.  ns: bases per row.
__device__ __forceinline__ int by_parity(int m, int n, int s0) { // m-th of 0 .. n-1, those with s0 + x even first
  const int first = s0 & 1, ne = (n + 1 - first) >> 1; // first even x; how many
  return m < ne ? first + 2 * m : 1 - first + 2 * (m - ne);
}
template <int FMA, int LANES, class D>
__device__ __forceinline__ void mono_tile(const D &d, int tile, int lid) {
  constexpr int PER = HTILE / LANES;
  const unsigned nunits = (unsigned)d.ns * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * HTILE + lid;
  const long long sy = d.ssy, sz = d.ssz;
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
#pragma unroll 1
  for (int r = 0; r < PER; ++r) {
    const unsigned p = p0 + r * LANES;
    if (p >= nunits) break;
    const unsigned row = div_magic(p, d.mg[0], d.sh[0]), pl = div_magic(row, d.mg[1], d.sh[1]);
    const int b = (int)(p - row * (unsigned)d.ns);
    const int j = by_parity((int)(row - pl * (unsigned)d.n[1]), d.n[1], d.soff[1]);
    const int k = by_parity((int)pl, d.n[2], d.soff[2]);
    const int fy = d.soff[1] + j, fz = d.soff[2] + k;
    const int cx = (d.soff[0] >> 1) + b, i = 2 * cx - d.soff[0]; // the even fine point: -1 .. n[0] - 1
    const double *q = d.src[0] + (cx + (fy >> 1) * sy + (long long)(fz >> 1) * sz);
    double *o = dst + (i + j * d.dsy + k * d.dsz);
    const bool e = i >= 0, f = i + 1 < d.n[0];
    const double v0 = e ? mono_point<FMA>(q, 0, fy & 1, fz & 1, sy, sz) : 0.0;
    const double v1 = f ? mono_point<FMA>(q, 1, fy & 1, fz & 1, sy, sz) : 0.0;
    if (e && f && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      *reinterpret_cast<double2 *>(o) = make_double2(v0, v1);
    } else {
      if (e) o[0] = v0;
      if (f) o[1] = v1;
    }
  }
}

// N source points of a row from q, whose place in 16 bytes `form` gives: 0
// first, 1 second, 2 unknown (rows of any alignment).  Pairs in one load: the
// lanes' rows lie 16 bytes apart, so that a load of single points wastes half
// of every line it touches.
template <class D> __device__ __forceinline__ int row_form(const D &d, const double *first) {
  if ((reinterpret_cast<uintptr_t>(d.src[0]) & 15) || (d.ssy & 1) || (d.ssz & 1)) return 2;
  return (int)((reinterpret_cast<uintptr_t>(first) >> 3) & 1);
}
template <int N> __device__ __forceinline__ void load_row(const double *q, int form, double v[N]) {
  static_assert(N % 2 == 0, "whole pairs");
  if (form == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 2) {
      const double2 a = __ldg(reinterpret_cast<const double2 *>(q + m));
      v[m] = a.x;
      v[m + 1] = a.y;
    }
  } else if (form == 1) { // the pairs from one point before to one point after: both in the row's padded length
#pragma unroll
    for (int m = -1; m < N; m += 2) {
      const double2 a = __ldg(reinterpret_cast<const double2 *>(q + m));
      if (m >= 0) v[m] = a.x;
      if (m + 1 < N) v[m + 1] = a.y;
    }
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) v[m] = __ldg(q + m);
  }
}

// restrict_3d_cc_o3_rf2 (restrict_3d_cc_o3_rf2.cc:147-211): the 4x4x4 fine
// cells 2i-1 .. 2i+2 per axis (from the region's first cell soff), weights
// c_a c_b c_c / 4096 with c = (-1, 9, 9, -1), summed left to right, x
// fastest; the first term is a plain product.
template <int FMA, int LANES, class D>
__device__ __forceinline__ void restrict_cc3_tile(const D &d, int tile, int lid) {
  constexpr int PER = HTILE / LANES;
  const unsigned npts = (unsigned)d.n[0] * d.n[1] * d.n[2];
  const unsigned p0 = (unsigned)tile * HTILE + lid;
  const long long ssy = d.ssy, ssz = d.ssz;
  const double *s0 = d.src[0] + (d.soff[0] - 1 + (d.soff[1] - 1) * ssy + (d.soff[2] - 1) * ssz);
  double *dst = d.dst + (d.doff[0] + d.doff[1] * d.dsy + d.doff[2] * d.dsz);
  const int form = row_form(d, s0);
#pragma unroll 1
  for (int r = 0; r < PER; ++r) {
    const unsigned p = p0 + r * LANES;
    if (p >= npts) break;
    int i, j, k;
    unflatten(d, p, i, j, k);
    const double *q = s0 + 2 * (i + j * ssy + k * ssz);
    double res = 0.0;
    // one plane of 16 cells per pass; every weight is an exact binary
    // fraction, so forming it from the plane's factor loses nothing
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      const double cz = (c == 0 || c == 3) ? -1.0 : 9.0;
      const double *qz = q + c * ssz;
      double v[4][4];
#pragma unroll
      for (int m = 0; m < 4; ++m) load_row<4>(qz + m * ssy, form, v[m]);
      static_for<16>([&](auto M) {
        constexpr int m = decltype(M)::value;
        constexpr double cx = (m & 3) == 0 || (m & 3) == 3 ? -1.0 : 9.0;
        constexpr double cy = (m >> 2) == 0 || (m >> 2) == 3 ? -1.0 : 9.0;
        const double w = cx * cy * cz / 4096.0;
        res = (m == 0 && c == 0) ? mul(w, v[0][0]) : madd<FMA>(w, v[m >> 2][m & 3], res);
      });
    }
    dst[i + j * d.dsy + k * d.dsz] = res;
  }
}

// restrict_3d_cc_o5_rf2 (restrict_3d_cc_o5_rf2.cc:36-78): restrict3 over the
// planes 2k-2 .. 2k+3 of restrict2 over rows of restrict1 over the cells
// 2i-2 .. 2i+3, each a left-to-right sum with weights (3, -25, 150, 150,
// -25, 3) / 256, the first term a plain product.  The CTA marches a tile of
// CC5X x CC5Y x pz coarse points plane by plane: restrict1 of the plane's
// rows into shared memory, restrict2 by the column's thread, which adds it to
// the three sums that the plane belongs to.  Every value is formed once per
// tile: about 100 operations and 30 loads of 16 bytes a point, where a point on
// its own takes 473 and 108 and was bound by L1 (96 uneven regions of 8-32
// coarse points a side: 246 us, two points sharing planes 103 us, this form
// 57 us; a batch of all three restrictions, a third of the regions each, 187 -> 81
// us a call).
// Regions below 2^16 coarse points take short tiles (pz 4), which run at once.
// Larger ones take 16, with fewer halo planes, which has not paid where it was
// measured since: 96 regions of 64-96 points a side 315 us against 311 us with
// short tiles, 8 of them 68 against 35.
constexpr int CC5X = 16, CC5Y = 8;
template <int FMA, int LANES, class D>
__device__ __forceinline__ void restrict_cc5_tile(const D &d, int tile, int lid) {
  constexpr int ROWS = 2 * CC5Y + 4;
  static_assert(CC5X * CC5Y <= LANES, "a thread per column");
  __shared__ double r1[2][ROWS * CC5X];
  const int tx = tile % d.tiles[0], rr = tile / d.tiles[0], ty = rr % d.tiles[1], tz = rr / d.tiles[1];
  const int i0 = tx * CC5X, j0 = ty * CC5Y, k0 = tz * d.pz;
  const int nx = min(CC5X, d.n[0] - i0), ny = min(CC5Y, d.n[1] - j0), nz = min((int)d.pz, d.n[2] - k0);
  const long long ssy = d.ssy, ssz = d.ssz;
  const double *s0 = d.src[0] + (d.soff[0] - 2 + 2 * i0 + (d.soff[1] - 2 + 2 * j0) * ssy + (d.soff[2] - 2 + 2 * k0) * ssz);
  constexpr double w[6] = {3.0 / 256, -25.0 / 256, 150.0 / 256, 150.0 / 256, -25.0 / 256, 3.0 / 256};
  const int form = row_form(d, s0);
  const int i = lid % CC5X, j = lid / CC5X;
  const bool owner = i < nx && j < ny;
  double *out = d.dst + (d.doff[0] + i0 + i + (d.doff[1] + j0 + j) * d.dsy + (d.doff[2] + k0) * d.dsz);
  // the thread's rows of a plane; those of the next plane are loaded before the
  // barrier, so that a plane costs no memory latency of its own
  constexpr int STEP = LANES / CC5X, R = (ROWS + STEP - 1) / STEP;
  const int rows = i < nx ? 2 * ny + 4 : 0, planes = 2 * nz + 4;
  double v[R][6];
  auto fetch = [&](int c) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (j + r * STEP < rows) load_row<6>(s0 + 2 * i + (j + r * STEP) * ssy + c * ssz, form, v[r]);
  };
  fetch(0);
  auto plane = [&](int c) { // restrict2 of plane c of the tile
    double *buf = r1[c & 1];
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (j + r * STEP < rows) {
        double x = mul(w[0], v[r][0]);
#pragma unroll
        for (int a = 1; a < 6; ++a) x = madd<FMA>(w[a], v[r][a], x);
        buf[(j + r * STEP) * CC5X + i] = x;
      }
    if (c + 1 < planes) fetch(c + 1);
    __syncthreads();
    double r2 = 0.0;
    if (owner) {
      const double *col = buf + 2 * j * CC5X + i;
      r2 = mul(w[0], col[0]);
#pragma unroll
      for (int b = 1; b < 6; ++b) r2 = madd<FMA>(w[b], col[b * CC5X], r2);
    }
    return r2;
  };
  double a0 = 0.0, a1 = 0.0, a2 = 0.0; // the sums of points m, m - 1, m - 2
#pragma unroll 1
  for (int m = 0; m < nz + 2; ++m) {
    double r2 = plane(2 * m);
    a0 = mul(w[0], r2);
    a1 = madd<FMA>(w[2], r2, a1);
    a2 = madd<FMA>(w[4], r2, a2);
    r2 = plane(2 * m + 1);
    a0 = madd<FMA>(w[1], r2, a0);
    a1 = madd<FMA>(w[3], r2, a1);
    a2 = madd<FMA>(w[5], r2, a2);
    if (m >= 2) {
      if (owner) *out = a2;
      out += d.dsz;
    }
    a2 = a1;
    a1 = a0;
  }
}

} // namespace cgx
