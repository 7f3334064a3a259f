// Column marches over a shared-memory tile, shared by the fused QG stage
// (qg_stage.cuh) and the advection kernel (advect.cu).
//
// A thread owns one column of the tile and walks RW of its rows.  Per row it
// evaluates the east and the north face of its cell from two register
// windows of 2R + 2 cells (R the scheme's reach): the row's cells around it,
// read from the tile, and the column's, which slides by one cell per row.
// The south face is the previous row's north one, the west face the left
// lane's east one (a shuffle), so no flux goes through shared memory.
// FP32 WENO5 / WENO-Z5 evaluates both faces as one packed f32x2 pair.  A warp
// whose cells all have the scheme's full reach takes the branch-free form;
// one that touches an edge (or, masked, a coast) picks each face's order.
#pragma once
#include "f32x2.cuh"
#include "recon.cuh"

namespace fvx {

// WENO5 / WENO-Z5 (weno5<float, Z> in recon.cuh, the same formulas) on two
// stencils at once: 38 packed operations and one reciprocal per lane for
// WENO5 (four for WENO-Z5).  Candidates and weights are scaled by 6 and 10
// so that most coefficients become sums (a packed constant occupies a
// register pair).  Stencils whose products leave the range go through
// weno5_wide.
template <bool Z>
DEV float2 weno5_x2(float2 qmm, float2 qm, float2 q0, float2 qp, float2 qpp) {
  const float2 d0 = f2sub(qm, qmm), d1 = f2sub(q0, qm), d2 = f2sub(qp, q0), d3 = f2sub(qpp, qp);
  const float2 a1 = f2sub(d1, d0), a2 = f2sub(d2, d1), a3 = f2sub(d3, d2);
  const float2 b1 = f2add(a1, d1);                                      // 2 d1 - d0
  const float2 c1 = f2add(b1, d1), c2 = f2add(d1, d2), c3 = f2sub(f2sub(a3, d2), d2);
  const float2 k = f2s(13.f / 3.f), eps4 = f2s(Z ? 4e-16f : 4e-8f);
  const float2 t1 = f2fma(c1, c1, f2fma(f2mul(k, a1), a1, eps4));
  const float2 t2 = f2fma(c2, c2, f2fma(f2mul(k, a2), a2, eps4));
  const float2 t3 = f2fma(c3, c3, f2fma(f2mul(k, a3), a3, eps4));
  // 6 (candidate - q0): 5 d1 - 2 d0, d1 + 2 d2, 4 d2 - d3
  const float2 g1 = f2add(c1, b1), g2 = f2add(c2, d2), g3 = f2sub(d2, c3);
  float2 W1, W2, W3;
  if (Z) {
    const float2 u = f2sub(t1, t3), tau = make_float2(fabsf(u.x), fabsf(u.y)), one = f2s(1.f);
    W1 = f2fma(tau, make_float2(rcp_approx(t1.x), rcp_approx(t1.y)), one);
    W2 = f2fma(tau, make_float2(rcp_approx(t2.x), rcp_approx(t2.y)), one);
    W3 = f2fma(tau, make_float2(rcp_approx(t3.x), rcp_approx(t3.y)), one);
  } else {
    const float2 s1 = f2mul(t1, t1), s2 = f2mul(t2, t2), s3 = f2mul(t3, t3);
    W1 = f2mul(s2, s3);
    W2 = f2mul(s1, s3);
    W3 = f2mul(s1, s2);
  }
  W2 = f2mul(f2s(6.f), W2);
  W3 = f2mul(f2s(3.f), W3);
  const float2 num = f2fma(W3, g3, f2fma(W2, g2, f2mul(W1, g1)));
  const float2 den = f2add(f2add(W1, W2), W3);
  bool ok = recon_finite(den.x, num.x) && recon_finite(den.y, num.y);
  if (Z) {
    const float2 t = f2add(f2add(t1, t2), t3);
    ok = ok && t.x < 8e37f && t.y < 8e37f;
  }
  if (ok) {
    const float s = 1.f / 6.f;
    return make_float2(fmaf(num.x * s, rcp_approx(den.x), q0.x), fmaf(num.y * s, rcp_approx(den.y), q0.y));
  }
  return make_float2(weno5_wide<Z>(qmm.x, qm.x, q0.x, qp.x, qpp.x), weno5_wide<Z>(qmm.y, qm.y, q0.y, qp.y, qpp.y));
}

// Window of a scheme: cells i - R .. i + R + 1 around face i at w[0 .. 2R+1].
template <int S> struct MarchWin {
  static constexpr int R = SchemeInfo<S>::is_weno ? SchemeInfo<S>::reach : 1;
  static constexpr int W = 2 * R + 2;
};
template <typename T, int N> struct Vals { T v[N]; };

// The scheme at its full reach on the upwind-oriented stencil e[0 .. 2R]
// (e[R] the upwind cell, e[R + 1] downstream of it): face_value's formulas.
template <typename T, int S>
DEV T recon_oriented(const T* e) {
  constexpr int R = MarchWin<S>::R;
  if constexpr (S == FVX_NAIVE) return T(0.5) * (e[R] + e[R + 1]);
  else if constexpr (S == FVX_UPWIND1) return e[R];
  else if constexpr (S == FVX_UPWIND2) return T(1.5) * e[R] - T(0.5) * e[R - 1];
  else if constexpr (S == FVX_UPWIND3) return T(-1.0 / 6.0) * e[R - 1] + T(5.0 / 6.0) * e[R] + T(1.0 / 3.0) * e[R + 1];
  else if constexpr (SchemeInfo<S>::tvd) {
    const T dn = e[R + 1] - e[R];
    return e[R] + T(0.5) * limiter_ratio<T, S>(e[R] - e[R - 1], dn + T(1e-8)) * dn;
  } else if constexpr (R == 1) return SchemeInfo<S>::zfam ? wenoz3(e[0], e[1], e[2]) : weno3(e[0], e[1], e[2]);
  else if constexpr (R == 2) return weno5<T, SchemeInfo<S>::zfam>(e[0], e[1], e[2], e[3], e[4]);
  else return weno_generic<T, R + 1>(e);
}
// WENO7 / WENO9 through a call: inlined in the march the compiler keeps the
// schemes' table coefficients in registers across the rows.
template <typename T, int S>
__noinline__ __device__ T recon_oriented_call(Vals<T, 2 * MarchWin<S>::R + 1> e) {
  return recon_oriented<T, S>(e.v);
}
template <typename T, int S>
DEV T march_face(const T (&w)[MarchWin<S>::W], bool pos) {
  constexpr int R = MarchWin<S>::R;
  Vals<T, 2 * R + 1> e;
#pragma unroll
  for (int k = 0; k <= 2 * R; ++k) e.v[k] = pos ? w[k] : w[2 * R + 1 - k];
  if constexpr (R >= 3) return recon_oriented_call<T, S>(e);
  else return recon_oriented<T, S>(e.v);
}
// Both faces of a cell at full reach.
template <typename T, int S>
DEV void march_faces(const T (&wx)[MarchWin<S>::W], const T (&wy)[MarchWin<S>::W], bool px, bool py, T& hx, T& hy) {
  if constexpr (sizeof(T) == 4 && (S == FVX_WENO5 || S == FVX_WENOZ5)) {
    float2 e[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) e[k] = make_float2(px ? wx[k] : wx[5 - k], py ? wy[k] : wy[5 - k]);
    const float2 r = weno5_x2<SchemeInfo<S>::zfam>(e[0], e[1], e[2], e[3], e[4]);
    hx = r.x;
    hy = r.y;
  } else {
    hx = march_face<T, S>(wx, px);
    hy = march_face<T, S>(wy, py);
  }
}
// Reach of face i on a line of N cells (face_value's ladder): R, or less
// near the ends.
template <int S>
DEV int march_reach(int i, int N, bool pos) {
  if constexpr (SchemeInfo<S>::is_weno) {
    const int c = pos ? i : i + 1;
    return min(MarchWin<S>::R, min(c, N - 1 - c));
  } else if constexpr (S == FVX_NAIVE || S == FVX_UPWIND1) return 1;
  else return !pos && i > N - 3 ? 0 : 1;
}
// The face at reach r <= R: first order for r = 0, then WENO3, 5, 7, 9 of
// the scheme's family (other schemes have r <= 1).
template <typename T, int S>
__noinline__ __device__ T march_ladder(Vals<T, MarchWin<S>::W> w, bool pos, int r) {
  constexpr int R = MarchWin<S>::R;
  T e[2 * R + 1];
#pragma unroll
  for (int k = 0; k <= 2 * R; ++k) e[k] = pos ? w.v[k] : w.v[2 * R + 1 - k];
  if (r == R) return recon_oriented<T, S>(e);
  if constexpr (SchemeInfo<S>::is_weno) {
    if constexpr (R >= 4) { if (r == 3) return weno_generic<T, 4>(e + R - 3); }
    if constexpr (R >= 3) { if (r == 2) return weno5<T, false>(e[R - 2], e[R - 1], e[R], e[R + 1], e[R + 2]); }
    if constexpr (R >= 2) {
      if (r == 1)
        return SchemeInfo<S>::zfam ? wenoz3(e[R - 1], e[R], e[R + 1]) : weno3(e[R - 1], e[R], e[R + 1]);
    }
  }
  return e[R];
}
template <typename T, int S>
DEV T march_edge_face(const T (&w)[MarchWin<S>::W], bool pos, int r) {
  Vals<T, MarchWin<S>::W> a;
#pragma unroll
  for (int k = 0; k < MarchWin<S>::W; ++k) a.v[k] = w[k];
  return march_ladder<T, S>(a, pos, r);
}

// ---- asynchronous global -> shared copies (cp.async, no register staging) --
template <typename T>
DEV void cp_async_elem(T* dst, const T* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
DEV void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
DEV void cp_async_8(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
// ROWS x COLS elements at src (row pitch ld) into dst (row pitch LD), issued
// by NT threads: 8-byte pieces, one column of pieces per thread walking the
// rows, when the rows allow (v8), else single elements.
template <typename T, int NT, int ROWS, int COLS, int LD>
DEV void tile_copy(T* dst, const T* src, long long ld, bool v8, int tid) {
  constexpr int E = 8 / (int)sizeof(T), C = COLS / E, RP = NT / C;
  static_assert(COLS % E == 0, "whole pieces");
  if (v8 || E == 1) {
    if constexpr (RP >= 1) {
      int r = tid / C;
      const int c = (tid - r * C) * E;
      if (r < RP)
        for (src += r * ld + c, dst += r * LD + c; r < ROWS; r += RP, src += RP * ld, dst += RP * LD) cp_async_8(dst, src);
    } else {
      for (int k = tid; k < ROWS * C; k += NT) {
        const int r = k / C, c = (k - r * C) * E;
        cp_async_8(dst + r * LD + c, src + r * ld + c);
      }
    }
  } else {
    for (int k = tid; k < ROWS * COLS; k += NT) {
      const int r = k / COLS, c = k - r * COLS;
      cp_async_elem(dst + r * LD + c, src + r * ld + c);
    }
  }
}

}  // namespace fvx
