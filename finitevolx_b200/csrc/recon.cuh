// Face-value reconstructions for flux-form advection on the C-grid.
//
// Point formulas restate finitevolX advection/weno.py (WENO3/5 JS and Z,
// WENO7/9 via the generic Jiang-Shu form) and advection/limiters.py.  They are
// reassociated (WENO3/5 on differences of neighbouring cells, weights over a
// common denominator, van Leer as one quotient): FP64 results agree with the
// reference's order of operations to 1e-12 of the largest flux, not to the
// last bit.  The boundary fallback ladders of advection/reconstruction.py
// (WENO5 :834-864, WENO7/9 :74-236, upwind2/3 and TVD east-boundary
// fallbacks) all reduce to one rule, used by face_value() below:
//
//   c = upwind cell of face i (i for u >= 0, i+1 for u < 0), N = line length,
//   d = min(c, N-1-c) cells available on the short side of c,
//   reach = min(scheme reach, d): 0 -> first-order upwind h[c],
//   1 -> WENO3, 2 -> WENO5, 3 -> WENO7, 4 -> WENO9 (same bias and family).
#pragma once
#include "fvx_common.cuh"
#include "weno_tables.cuh"

namespace fvx {

template <typename T> DEV T sq(T x) { return x * x; }
// FP32 reciprocal by the hardware approximation (rcp.approx.ftz.f32, at
// most 1 ulp): +inf for 0, 0 for |b| > 2^126 (the result would be
// subnormal and is flushed).
DEV float rcp_approx(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
// Division in the reconstruction formulas: exact IEEE division in FP64, a times
// the approximate reciprocal of b in FP32 (<= 2 ulp for |b| <= 2^126; WENO3/5
// keep their denominators below that, WENO7/9 weights beyond it become 0).
template <typename T> DEV T fdiv(T a, T b) {
  if constexpr (sizeof(T) == 8) return a / b;
  else return a * rcp_approx(b);
}
template <typename T> DEV T tabs(T x) { return x < T(0) ? -x : x; }
template <typename T> DEV T tmax(T a, T b) { return a > b ? a : b; }
template <typename T> DEV T tmin(T a, T b) { return a < b ? a : b; }

// The reconstructions below work on the differences d of neighbouring cells:
// a candidate is q0 plus a combination of them, the smoothness forms are
// squares of them, and the weights 1 / s_k (s_k = (b_k + eps)^2) are brought
// to their common denominator, prod_{j != k} s_j, so that one division
// normalises the whole sum (a division costs 13 FP64 FMAs of throughput;
// FP32 takes one reciprocal).  In FP64 no such product underflows, and
// stencils whose products overflow take the form with a division per weight.
// In FP32 stencils whose products leave the range of the type or of the
// reciprocal (2^126, beyond which it is flushed to 0) are scaled first, by a
// call (weno3_wide, weno5_wide); WENO5's products of differences under 1e-9
// are subnormal and keep an absolute error of about 1e-16.
template <typename T> DEV bool recon_finite(T den, T num) {
  if constexpr (sizeof(T) == 8) return den < 1e308 && fabs(num) < 1e308;
  else return den < 8e37f && fabsf(num) < 3e38f;
}
// Power-of-two scale for differences of at most m, to c m in [1, 4), with its
// inverse ic.  A form is homogeneous in (d, sqrt(eps)); eps c^2 is kept within
// [1e-18, 1e8], beyond which it changes a weight by less than 1e-8 (or decides
// between differences 1e9 times smaller than m).
DEV void recon_scale(float m, float eps, float& c, float& ic, float& epsc) {
  const int e = min(max((int)(__float_as_uint(m) >> 23), 1), 253);
  ic = __uint_as_float((unsigned)e << 23);
  c = __uint_as_float((unsigned)(254 - e) << 23);
  epsc = fminf(fmaxf(eps * c * c, 1e-18f), 1e8f);
}

// ---- WENO3 (advection/weno.py:297-347) ------------------------------------
// The right-biased forms (:413-459, :462-522, :597-665) are these functions on
// the mirrored stencil; face_value() below feeds them that way.
// Numerator and denominator of 2 (face - q0): weights 1/3, 2/3 (WENO-Z3: times
// 1 + tau / (b + eps)) and candidates q0 + d/2.
template <typename T, bool Z> DEV void weno3_sums(T d1, T d2, T eps, T& num, T& den) {
  if constexpr (Z) {
    const T b1 = d1 * d1, b2 = d2 * d2, tau = tabs(b2 - b1), t1 = b1 + eps, t2 = b2 + eps;
    const T W1 = (t1 + tau) * t2, W2 = T(2) * ((t2 + tau) * t1);
    den = W1 + W2;
    num = W1 * d1 + W2 * d2;
  } else {
    const T s1 = sq(d1 * d1 + eps), s2 = sq(d2 * d2 + eps);
    den = s2 + T(2) * s1;
    num = s2 * d1 + T(2) * (s1 * d2);
  }
}
// FP32, out of the products' range.
template <bool Z>
__noinline__ __device__ float weno3_wide(float qm, float q0, float qp) {
  const float d1 = q0 - qm, d2 = qp - q0;
  float c, ic, eps, num, den;
  recon_scale(fmaxf(fabsf(d1), fabsf(d2)), Z ? 1e-14f : 1e-8f, c, ic, eps);
  weno3_sums<float, Z>(d1 * c, d2 * c, eps, num, den);
  return q0 + (0.5f * fdiv(num, den)) * ic;
}
// FP64, products that overflow: a division per weight.
template <bool Z>
DEV double weno3_divisions(double qm, double q0, double qp) {
  const double b1 = sq(q0 - qm), b2 = sq(qp - q0);
  double w1, w2;
  if (Z) {
    const double tau = tabs(b2 - b1);
    w1 = 1.0 / 3.0 * (1.0 + tau / (b1 + 1e-14));
    w2 = 2.0 / 3.0 * (1.0 + tau / (b2 + 1e-14));
  } else {
    w1 = 1.0 / 3.0 / sq(b1 + 1e-8);
    w2 = 2.0 / 3.0 / sq(b2 + 1e-8);
  }
  return (w1 * (-0.5 * qm + 1.5 * q0) + w2 * (0.5 * (q0 + qp))) / (w1 + w2);
}
template <typename T, bool Z> DEV T weno3_form(T qm, T q0, T qp) {
  const T d1 = q0 - qm, d2 = qp - q0;
  T num, den;
  weno3_sums<T, Z>(d1, d2, Z ? T(1e-14) : T(1e-8), num, den);
  // FP32: a numerator under the smallest normal number (WENO-Z3 from
  // differences of 1e-10 down, WENO3 of 1e-22) has lost its low bits
  const bool small = sizeof(T) == 4 && !(fabsf((float)num) > 1e-37f) && (d1 != T(0) || d2 != T(0));
  if (recon_finite(den, num) && !small) return q0 + T(0.5) * fdiv(num, den);
  if constexpr (sizeof(T) == 4) return weno3_wide<Z>(qm, q0, qp);
  else return weno3_divisions<Z>(qm, q0, qp);
}
template <typename T> DEV T weno3(T qm, T q0, T qp) { return weno3_form<T, false>(qm, q0, qp); }
template <typename T> DEV T wenoz3(T qm, T q0, T qp) { return weno3_form<T, true>(qm, q0, qp); }
// ---- WENO5 (advection/weno.py:350-410, :462-522) -------------------------
// The form with a division per weight, on the raw values (FP64).
template <bool Z>
__noinline__ __device__ double weno5_divisions(double qmm, double qm, double q0, double qp, double qpp) {
  const double k1 = 13.0 / 12.0, k2 = 0.25;
  const double qi1 = 1.0 / 3.0 * qmm - 7.0 / 6.0 * qm + 11.0 / 6.0 * q0;
  const double qi2 = -1.0 / 6.0 * qm + 5.0 / 6.0 * q0 + 1.0 / 3.0 * qp;
  const double qi3 = 1.0 / 3.0 * q0 + 5.0 / 6.0 * qp - 1.0 / 6.0 * qpp;
  const double b1 = k1 * sq(qmm - 2.0 * qm + q0) + k2 * sq(qmm - 4.0 * qm + 3.0 * q0);
  const double b2 = k1 * sq(qm - 2.0 * q0 + qp) + k2 * sq(qm - qp);
  const double b3 = k1 * sq(q0 - 2.0 * qp + qpp) + k2 * sq(3.0 * q0 - 4.0 * qp + qpp);
  double w1, w2, w3;
  if (Z) {
    const double eps = 1e-16, tau5 = tabs(b1 - b3);
    w1 = 0.1 * (1.0 + tau5 / (b1 + eps));
    w2 = 0.6 * (1.0 + tau5 / (b2 + eps));
    w3 = 0.3 * (1.0 + tau5 / (b3 + eps));
  } else {
    const double eps = 1e-8;
    w1 = 0.1 / sq(b1 + eps);
    w2 = 0.6 / sq(b2 + eps);
    w3 = 0.3 / sq(b3 + eps);
  }
  return (w1 * qi1 + w2 * qi2 + w3 * qi3) / (w1 + w2 + w3);
}
// Numerator and denominator of face - q0 from the four differences; eps4 = 4
// eps.  Returns the sum of the smoothness terms t = 4 (b + eps).
template <typename T, bool Z> DEV T weno5_sums(T d0, T d1, T d2, T d3, T eps4, T& num, T& den) {
  const T a1 = d1 - d0, a2 = d2 - d1, a3 = d3 - d2;
  const T c1 = a1 + T(2) * d1, c2 = d1 + d2, c3 = a3 - T(2) * d2;
  const T k = T(13.0 / 3.0);
  const T t1 = c1 * c1 + (k * a1 * a1 + eps4), t2 = c2 * c2 + (k * a2 * a2 + eps4),
          t3 = c3 * c3 + (k * a3 * a3 + eps4);
  const T g1 = T(5.0 / 6.0) * d1 - T(1.0 / 3.0) * d0, g2 = T(1.0 / 6.0) * d1 + T(1.0 / 3.0) * d2,
          g3 = T(2.0 / 3.0) * d2 - T(1.0 / 6.0) * d3;
  T W1, W2, W3;
  if constexpr (Z) {
    const T tau = tabs(t1 - t3);
    if constexpr (sizeof(T) == 4) {  // products of three t >= 4e-16 would underflow
      W1 = T(0.1) * (T(1) + fdiv(tau, t1));
      W2 = T(0.6) * (T(1) + fdiv(tau, t2));
      W3 = T(0.3) * (T(1) + fdiv(tau, t3));
    } else {
      W1 = T(0.1) * ((t1 + tau) * (t2 * t3));
      W2 = T(0.6) * ((t2 + tau) * (t1 * t3));
      W3 = T(0.3) * ((t3 + tau) * (t1 * t2));
    }
  } else {
    const T s1 = t1 * t1, s2 = t2 * t2, s3 = t3 * t3;
    W1 = T(0.1) * (s2 * s3);
    W2 = T(0.6) * (s1 * s3);
    W3 = T(0.3) * (s1 * s2);
  }
  den = W1 + W2 + W3;
  num = W1 * g1 + W2 * g2 + W3 * g3;
  return t1 + t2 + t3;
}
// FP32, out of the products' range.
template <bool Z>
__noinline__ __device__ float weno5_wide(float qmm, float qm, float q0, float qp, float qpp) {
  const float d0 = qm - qmm, d1 = q0 - qm, d2 = qp - q0, d3 = qpp - qp;
  const float m = fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(d2), fabsf(d3)));
  float c, ic, eps4, num, den;
  recon_scale(m, Z ? 4e-16f : 4e-8f, c, ic, eps4);
  weno5_sums<float, Z>(d0 * c, d1 * c, d2 * c, d3 * c, eps4, num, den);
  return q0 + fdiv(num, den) * ic;
}
template <typename T, bool Z> DEV T weno5(T qmm, T qm, T q0, T qp, T qpp) {
  T num, den;
  const T t = weno5_sums<T, Z>(qm - qmm, q0 - qm, qp - q0, qpp - qp, Z ? T(4e-16) : T(4e-8), num, den);
  // (FP32 WENO-Z5: the reciprocals of the t have to be in range as well)
  if (recon_finite(den, num) && (!Z || sizeof(T) == 8 || t < T(8e37))) return q0 + fdiv(num, den);
  if constexpr (sizeof(T) == 4) return weno5_wide<Z>(qmm, qm, q0, qp, qpp);
  else return weno5_divisions<Z>(qmm, qm, q0, qp, qpp);
}
// ---- WENO7 / WENO9, generic Jiang-Shu form (advection/weno.py:268-294) ---
template <typename T> DEV T tab_c(int R, int k, int j) {
  if constexpr (sizeof(T) == 8) return R == 4 ? kW7_C[k][j] : kW9_C[k][j];
  else return R == 4 ? kW7_Cf[k][j] : kW9_Cf[k][j];
}
template <typename T> DEV T tab_w(int R, int k) {
  if constexpr (sizeof(T) == 8) return R == 4 ? kW7_W[k] : kW9_W[k];
  else return R == 4 ? kW7_Wf[k] : kW9_Wf[k];
}
template <typename T> DEV T tab_b(int R, int k, int i, int j) {
  if constexpr (sizeof(T) == 8) return R == 4 ? kW7_B[k][i][j] : kW9_B[k][i][j];
  else return R == 4 ? kW7_Bf[k][i][j] : kW9_Bf[k][i][j];
}

// v[0..2R-2]: the 2R-1 cells of the big stencil ordered in the upwind
// direction (the mirrored, negative-flow tables of the reference are the
// left-biased tables on the reversed stencil).
//
// FP32: the quadratic forms have O(10^3) alternating coefficients, so on raw
// values they lose ~4 digits to cancellation against the local mean.  The
// FP32 build evaluates them (and the candidates) on values shifted by the
// stencil centre s: exact algebra, because every form annihilates constants
// (B 1 = 0) and every candidate's weights sum to one, so
// cand(v) = s + cand(v - s) and beta(v) = beta(v - s).  FP64 keeps the
// reference's raw-value evaluation order.
template <typename T, int R>
DEV T weno_generic(const T* vin) {
  const T eps = T(1e-8);
  constexpr bool SHIFT = sizeof(T) == 4;
  const T s = SHIFT ? vin[R - 1] : T(0);
  T v[2 * R - 1];
#pragma unroll
  for (int k = 0; k < 2 * R - 1; ++k) v[k] = SHIFT ? vin[k] - s : vin[k];
  T cand[R], st[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    cand[k] = T(0);
#pragma unroll
    for (int j = 0; j < R; ++j) cand[k] = cand[k] + tab_c<T>(R, k, j) * v[k + j];
    T beta = T(0);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      T row = T(0);
#pragma unroll
      for (int j = 0; j < R; ++j) row = row + tab_b<T>(R, k, i, j) * v[k + j];
      beta = beta + v[k + i] * row;
    }
    st[k] = sq(beta + eps);
  }
  T num = T(0), den = T(0);
  if constexpr (sizeof(T) == 8) {  // one division (in FP32 the products of three or four s_k underflow)
    T pre[R], suf = T(1);
    pre[0] = T(1);
#pragma unroll
    for (int k = 1; k < R; ++k) pre[k] = pre[k - 1] * st[k - 1];
#pragma unroll
    for (int k = R - 1; k >= 0; --k) {
      const T a = tab_w<T>(R, k) * (pre[k] * suf);
      suf *= st[k];
      den = den + a;
      num = num + a * cand[k];
    }
    if (recon_finite(den, num)) return num / den;
    num = den = T(0);
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const T a = fdiv(tab_w<T>(R, k), st[k]);
    den = den + a;
    num = num + a * cand[k];
  }
  return SHIFT ? s + fdiv(num, den) : num / den;
}

// ---- limiters (advection/limiters.py:34-123) -----------------------------
template <typename T, int S> DEV T limiter(T r) {
  if (S == FVX_MINMOD) return tmax(T(0), tmin(T(1), r));
  if (S == FVX_VAN_LEER) { T ra = tabs(r); return (r + ra) / (T(1) + ra); }
  if (S == FVX_SUPERBEE) return tmax(T(0), tmax(tmin(T(2) * r, T(1)), tmin(r, T(2))));
  return tmax(T(0), tmin(tmin((T(1) + r) / T(2), T(2) * r), T(2)));  // MC
}

// limiter(r) with r = a / b, van Leer with one division: for r > 0 its value
// is 2a / (a + b) (no cancellation: a and b have one sign), for finite r < 0
// it is 0; zero, overflowing and undefined ratios keep the two-division form.
template <typename T, int S> DEV T limiter_ratio(T a, T b) {
  if constexpr (S == FVX_VAN_LEER) {
    const T p = a * b, big = sizeof(T) == 8 ? T(1e300) : T(1e37f);
    if (p > T(0) && p < big) return T(2) * a / (a + b);
    if (p < T(0) && p > -big) return T(0);
  }
  return limiter<T, S>(a / b);
}

template <int S> struct SchemeInfo {
  static constexpr bool is_weno = (S == FVX_WENO3 || S == FVX_WENOZ3 || S == FVX_WENO5 ||
                                   S == FVX_WENOZ5 || S == FVX_WENO7 || S == FVX_WENO9);
  static constexpr int reach = (S == FVX_WENO3 || S == FVX_WENOZ3) ? 1
                               : (S == FVX_WENO5 || S == FVX_WENOZ5) ? 2
                               : (S == FVX_WENO7) ? 3 : (S == FVX_WENO9) ? 4 : 1;
  static constexpr bool zfam = (S == FVX_WENOZ3 || S == FVX_WENOZ5);
  static constexpr bool tvd = (S == FVX_MINMOD || S == FVX_VAN_LEER || S == FVX_SUPERBEE || S == FVX_MC);
  // cells read on each side of the face's left cell i: [i - lo, i + hi]
};

// Face value at face i (between cells i and i+1) of a line of N cells.
// ``p`` points at cell i; neighbours are p[k*st].  pos: u >= 0.
// Valid for 1 <= i <= N-2 (the faces the reference reconstructs).
template <typename T, int S>
DEV T face_value(const T* p, int st, int i, int N, bool pos) {
  auto at = [&](int k) -> T { return p[k * st]; };
  if (S == FVX_NAIVE) return T(0.5) * (at(0) + at(1));
  if (S == FVX_UPWIND1) return pos ? at(0) : at(1);
  if (S == FVX_UPWIND2) {
    if (pos) return T(1.5) * at(0) - T(0.5) * at(-1);
    return (i <= N - 3) ? T(1.5) * at(1) - T(0.5) * at(2) : at(1);
  }
  if (S == FVX_UPWIND3) {
    if (pos) return T(-1.0 / 6.0) * at(-1) + T(5.0 / 6.0) * at(0) + T(1.0 / 3.0) * at(1);
    return (i <= N - 3) ? T(1.0 / 3.0) * at(0) + T(5.0 / 6.0) * at(1) - T(1.0 / 6.0) * at(2) : at(1);
  }
  if constexpr (SchemeInfo<S>::tvd) {
    if (pos) {
      T dfwd = at(1) - at(0);
      T dbwd = at(0) - at(-1);
      return at(0) + T(0.5) * limiter_ratio<T, S>(dbwd, dfwd + T(1e-8)) * dfwd;
    }
    if (i > N - 3) return at(1);
    T dn = at(0) - at(1);
    T dn2 = at(1) - at(2);
    return at(1) + T(0.5) * limiter_ratio<T, S>(dn2, dn + T(1e-8)) * dn;
  }
  if constexpr (SchemeInfo<S>::is_weno) {
    // Upwind-oriented stencil: e(k) is the cell k steps downstream of the
    // upwind cell c (pos: h[i+k], neg: h[i+1-k]).  Every right-biased formula
    // of the reference is the left-biased one on the mirrored stencil (same
    // candidates, same smoothness squares, same weights), so both flow
    // directions run one code path and warps do not diverge on the sign.
    constexpr bool Z = SchemeInfo<S>::zfam;
    const int c = pos ? i : i + 1;
    const int d = min(c, N - 1 - c);
    const int r = min(SchemeInfo<S>::reach, d);
    const T* b = pos ? p : p + st;
    const int s = pos ? st : -st;
    auto e = [&](int k) -> T { return b[k * s]; };
    if (r >= 4) {
      T v[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = e(k - 4);
      return weno_generic<T, 5>(v);
    }
    if (r == 3) {
      T v[7];
#pragma unroll
      for (int k = 0; k < 7; ++k) v[k] = e(k - 3);
      return weno_generic<T, 4>(v);
    }
    if (r == 2) return weno5<T, Z>(e(-2), e(-1), e(0), e(1), e(2));
    if (r == 1) return Z ? wenoz3(e(-1), e(0), e(1)) : weno3(e(-1), e(0), e(1));
    return e(0);
  }
  return T(0);
}

}  // namespace fvx
