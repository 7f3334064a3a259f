// Fused QG RK stage: the per-tile body shared by the single-field kernel
// (qg.cu) and the ensemble's persistent work-queue kernel (ensemble.cu).
#pragma once
#include "march.cuh"

#include <cuda_bf16.h>

#include <type_traits>

namespace fvx {
namespace qg {

constexpr int THREADS = 128;
// Tile shapes (fvx_qg_tile_config): TX x TY cells, TX TY / 128 rows per thread.
constexpr int kTileTX[6] = {64, 32, 128, 64, 128, 16};
constexpr int kTileTY[6] = {16, 16, 8, 32, 16, 16};
constexpr int kTileConfigs = 6;

struct StageArgs {
  const void* qs;      // stage state [Ny][Nx]
  const void* qn;      // step-start state (null on stage 1)
  const void* psi;     // interior-only [Ny-2][Nx-2]
  const void* forcing; // [Ny][Nx] or null
  void* out;           // [Ny][Nx]
  __nv_bfloat16* split_hi;  // [Ny-2][Nx-2] or null (FP64 stages: a double [Ny-2][Nx-2] interior copy)
  __nv_bfloat16* split_lo;  // (FP64 stages: null)
  int split_layout;         // 1: x de-interleaved (the even/odd DST operand layout)
  int ny, nx;
  double a, b, c;      // out = a*qn + b*qs + c*rhs
  double dx, dy, beta, drag, visc;
  int periodic;        // 1: periodic ghost ring, 0: zero (wall) ghost ring
  int write_ghost;
};

// ---- tile geometry ----------------------------------------------------------
// The q tile covers rows y0-H .. y0+TY+H-1 and columns x0-H .. x0+TX+H-1;
// element (ly, lx) sits at [ly * QW + SH + lx].  SH makes each stored row
// start at an even column (x0 is even), so that FP32 rows can be copied in
// 8-byte pieces.
template <typename T, int S, int TX, int TY>
struct Geom {
  static constexpr int R = MarchWin<S>::R, W = MarchWin<S>::W;
  static constexpr int H = R + 1;
  static constexpr int SH = H & 1;
  static constexpr int QW = (TX + 2 * H + SH + 1) & ~1;
  static constexpr int QH = TY + 2 * H;
  static constexpr int PW = TX + 2;                // psi, origin (y0-1, x0-1)
  static constexpr int NQ = QH * QW, NP = (TY + 2) * PW;
  static constexpr int RW = TX * TY / THREADS;     // rows a thread marches
  static constexpr int WC = TX < 32 ? TX : 32;     // columns whose west neighbour is the lane to the left
  static constexpr int NWEST = TY * (TX / WC);     // west faces from the other columns (first pass)
  static_assert(RW * THREADS == TX * TY && TY % RW == 0 && NWEST <= THREADS, "whole marches");
};

// One tile of the stage (march.cuh).  Bound by instruction issue at large
// sizes, by the latency of a row's reconstruction (times RW) at small ones.
// Velocities away from the edges come straight from psi: u = -(X[j] -
// X[j-1]) / dy with X = T_to_X(psi) is -(psi[j+1][i] + psi[j+1][i+1] -
// psi[j-1][i] - psi[j-1][i+1]) / (4 dy) (the psi[j] terms cancel), v likewise.  The earlier body (per-tile X, flux and velocity arrays in
// shared memory, a loop per array, quotients by dx and dy in FP64) took 44.4
// us at 2048^2 FP32 WENO5 and 15.1 us at 256^2 FP64 (ncu).
template <typename T, int S, int TX, int TY>
DEV void stage_body(const StageArgs& A, uint8_t* sm, const bool in, const int x0, const int y0) {
  using G = Geom<T, S, TX, TY>;
  constexpr int R = G::R, W = G::W, H = G::H, QW = G::QW, QH = G::QH, PW = G::PW, RW = G::RW, WC = G::WC;
  T* base = (T*)sm;
  T* qt = base + G::SH;                    // q (ly, lx) at qt[ly * QW + lx]
  T* pt = base + G::NQ;                    // psi [TY+2][PW], origin (y0-1, x0-1)
  T* west = pt + G::NP;                    // [TX / WC][TY] fluxes through the faces x0 - 1 + k WC
  const int ny = A.ny, nx = A.nx, nxi = nx - 2;
  const int tid = threadIdx.x;
  const T* qs = (const T*)A.qs;
  const T* psi = (const T*)A.psi;
  // ---- loads: q with BC applied on the fly, psi with zero outside --------
  if (in) {
    const bool v8 = (((uintptr_t)qs | (uintptr_t)psi) & 7) == 0 && (nx & 1) == 0;
    tile_copy<T, THREADS, QH, QW, QW>(base, qs + (size_t)(y0 - H) * nx + (x0 - H - G::SH), nx, v8, tid);
    tile_copy<T, THREADS, TY + 2, PW, PW>(pt, psi + (size_t)(y0 - 2) * nxi + (x0 - 2), nxi, v8, tid);
  } else {
    // wrap-around / zero-ring sources resolved per element
    for (int k = tid; k < QH * (QW - G::SH); k += THREADS) {
      const int ly = k / (QW - G::SH), lx = k - ly * (QW - G::SH);
      const int gy = y0 - H + ly, gx = x0 - H + lx;
      const T* src = nullptr;
      if (gy >= 0 && gy < ny && gx >= 0 && gx < nx) {
        const bool gh = gy == 0 || gy == ny - 1 || gx == 0 || gx == nx - 1;
        if (!gh) src = qs + (size_t)gy * nx + gx;
        else if (A.periodic) {
          const int sy = gy == 0 ? ny - 2 : (gy == ny - 1 ? 1 : gy);
          const int sx = gx == 0 ? nx - 2 : (gx == nx - 1 ? 1 : gx);
          src = qs + (size_t)sy * nx + sx;
        }
      }
      if (src) cp_async_elem(qt + ly * QW + lx, src);
      else qt[ly * QW + lx] = T(0);
    }
    for (int k = tid; k < (TY + 2) * PW; k += THREADS) {
      const int ly = k / PW, lx = k - ly * PW;
      const int gy = y0 - 1 + ly, gx = x0 - 1 + lx;
      if (gy >= 1 && gy <= ny - 2 && gx >= 1 && gx <= nx - 2) cp_async_elem(pt + k, psi + (size_t)(gy - 1) * nxi + (gx - 1));
      else pt[k] = T(0);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  const T rdx = T(1.0 / A.dx), rdy = T(1.0 / A.dy);
  const T cu = T(-0.25) * rdy, cv = T(0.25) * rdx;
  // full reach and interior velocities on both axes (also: none of the
  // two outermost interior rows / columns)
  constexpr int E = R > 2 ? R : 2;
  auto row_full = [&](int j) { return j >= E && j + 1 <= ny - 1 - R; };
  auto col_full = [&](int c) { return c >= E && c + 1 <= nx - 1 - R; };
  auto inside = [&](int j, int c) { return j >= 1 && j <= ny - 2 && c >= 1 && c <= nx - 2; };
  // velocities of cell (j, c) next to the edges, p at psi (j, c): the same
  // differences, or one X alone where its neighbour is a ghost (zero)
  auto xcorner = [&](const T* p) -> T { return T(0.25) * (p[0] + p[1] + p[PW] + p[PW + 1]); };
  auto u_edge = [&](const T* p, int j, int c) -> T {
    if (!inside(j, c)) return T(0);
    return j > 1 ? cu * ((p[PW] - p[-PW]) + (p[PW + 1] - p[-PW + 1])) : -xcorner(p) * rdy;
  };
  auto v_edge = [&](const T* p, int j, int c) -> T {
    if (!inside(j, c)) return T(0);
    return c > 1 ? cv * ((p[1] - p[-1]) + (p[PW + 1] - p[PW - 1])) : xcorner(p) * rdx;
  };
  const int col = tid % TX, seg = tid / TX, c = x0 + col, jb = y0 + seg * RW;
  const T* qc = qt + (seg * RW + H) * QW + (col + H);      // q (jb, c)
  const T* pc = pt + (seg * RW + 1) * PW + (col + 1);      // psi (jb, c)
  const bool cf = col_full(c);
  // ---- first pass: the south face of the march's first row, and the west
  // faces that no lane to the left has ----------------------------------------
  T wy[W];  // column window of the north face last evaluated
  T fs, vs;
  {
    const int t = tid < G::NWEST ? tid : 0;
    const int grp = t / TY, wr = t - grp * TY;
    const int jw = y0 + wr, cw = x0 + grp * WC - 1, js = jb - 1;
    const T* qw = qt + (wr + H) * QW + (grp * WC - 1 + H);
    const T* pw = pt + (wr + 1) * PW + (grp * WC);         // psi (jw, cw)
    const T* ps = pc - PW;                                 // psi (js, c)
    T wx[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      wx[k] = qw[k - R];
      wy[k] = qc[(k - R - 1) * QW];
    }
    T uw, hx, hy;
    if (__all_sync(0xffffffffu, cf && row_full(js) && row_full(jw) && col_full(cw))) {
      uw = cu * ((pw[PW] - pw[-PW]) + (pw[PW + 1] - pw[-PW + 1]));
      vs = cv * ((ps[1] - ps[-1]) + (ps[PW + 1] - ps[PW - 1]));
      march_faces<T, S>(wx, wy, uw >= T(0), vs >= T(0), hx, hy);
    } else {
      uw = u_edge(pw, jw, cw);
      vs = v_edge(ps, js, c);
      hx = march_edge_face<T, S>(wx, uw >= T(0), march_reach<S>(cw, nx, uw >= T(0)));
      hy = march_edge_face<T, S>(wy, vs >= T(0), march_reach<S>(js, ny, vs >= T(0)));
      if (!inside(jw, cw)) hx = T(0);
      if (!inside(js, c)) hy = T(0);
    }
    if (tid < G::NWEST) west[t] = hx * uw;
    fs = hy * vs;
  }
  __syncthreads();
  // ---- the march ------------------------------------------------------------
  const T beta = T(A.beta), ca = T(A.a), cb = T(A.b), cc = T(A.c);
  const bool has_qn = A.qn != nullptr, split = A.split_hi != nullptr;
  const bool extra = A.forcing || A.drag != 0.0 || A.visc != 0.0;
  const bool first = col % WC == 0;
  const T* wst = west + (col / WC) * TY + seg * RW;
  const long long g = (long long)jb * nx + c;
  const T* qn = (const T*)A.qn + g;
  const T* F = (const T*)A.forcing + g;
  T* out = (T*)A.out + g;
  const int xi = c - 1;
  const int scol = A.split_layout ? ((xi & 1) ? (nxi >> 1) + (xi >> 1) : (xi >> 1)) : xi;
  const long long si = (long long)(jb - 1) * nxi + scol;
  double* s64 = (double*)(void*)A.split_hi + si;  // FP64 stages: the interior itself
  __nv_bfloat16 *shi = A.split_hi + si, *slo = A.split_lo + si;
  T pmc = pc[-PW], pmr = pc[-PW + 1], p0c = pc[0], p0r = pc[1], e0 = p0r - pc[-1];
  // FULL: every row of every lane of the warp is away from the edges
  auto rows = [&](auto full_c) {
    constexpr bool FULL = decltype(full_c)::value;
#pragma unroll(FULL ? (RW < 4 ? RW : 4) : 1)
    for (int r = 0; r < RW; ++r) {
      const int j = jb + r;
      const bool all = FULL || __all_sync(0xffffffffu, cf && row_full(j));
      const bool store = FULL || all || inside(j, c);
      T qnv = T(0);
      if (has_qn && store) qnv = *qn;
      T wx[W];
#pragma unroll
      for (int k = 0; k + 1 < W; ++k) wy[k] = wy[k + 1];
      wy[W - 1] = qc[(R + 1) * QW];
#pragma unroll
      for (int k = 0; k < W; ++k) wx[k] = k == R ? wy[R] : qc[k - R];
      const T npc = pc[PW], npr = pc[PW + 1], e1 = npr - pc[PW - 1];
      T u, v, hx, hy;
      if (FULL || all) {
        u = cu * ((npc - pmc) + (npr - pmr));
        v = cv * (e0 + e1);
        march_faces<T, S>(wx, wy, u >= T(0), v >= T(0), hx, hy);
      } else {
        u = u_edge(pc, j, c);
        v = v_edge(pc, j, c);
        hx = march_edge_face<T, S>(wx, u >= T(0), march_reach<S>(c, nx, u >= T(0)));
        hy = march_edge_face<T, S>(wy, v >= T(0), march_reach<S>(j, ny, v >= T(0)));
        if (!inside(j, c)) hx = hy = T(0);
      }
      const T fe = hx * u, fn = hy * v;
      T fw = __shfl_up_sync(0xffffffffu, fe, 1);
      if (first) fw = wst[r];
      T rhs = -((fe - fw) * rdx + (fn - fs) * rdy);
      if (!FULL && !(j >= 2 && j <= ny - 3 && c >= 2 && c <= nx - 3)) rhs = T(0);
      rhs = rhs + (-beta * (T(0.5) * (v + vs)));
      if (extra) {
        if (A.forcing && store) rhs = rhs + *F;
        if (A.drag != 0.0) {
          const T d2x = ((p0r - p0c) - (p0c - pc[-1])) * (rdx * rdx);
          const T d2y = ((npc - p0c) - (p0c - pmc)) * (rdy * rdy);
          rhs = rhs - T(A.drag) * (d2x + d2y);
        }
        if (A.visc != 0.0) {
          const T d2x = ((wx[R + 1] - wx[R]) - (wx[R] - wx[R - 1])) * (rdx * rdx);
          const T d2y = ((wy[R + 1] - wy[R]) - (wy[R] - wy[R - 1])) * (rdy * rdy);
          rhs = rhs + T(A.visc) * (d2x + d2y);
        }
      }
      T q = cb * wx[R];
      if (has_qn) q = ca * qnv + q;
      q = q + cc * rhs;
      if (store) {
        *out = q;
        if (split) {
          if constexpr (sizeof(T) == 8) {
            *s64 = q;
          } else {
            const float f = (float)q;
            const __nv_bfloat16 h = __float2bfloat16_rn(f);
            *shi = h;
            *slo = __float2bfloat16_rn(f - __bfloat162float(h));
          }
        }
      }
      if (!FULL && A.write_ghost && !all) {
        T* o = (T*)A.out;
        if (A.periodic && store) {
          // copies of this interior cell into the ghost ring (S, N, W, E fill)
          const int yg = j == ny - 2 ? 0 : (j == 1 ? ny - 1 : -1), xg = c == nx - 2 ? 0 : (c == 1 ? nx - 1 : -1);
          if (yg >= 0) o[(size_t)yg * nx + c] = q;
          if (xg >= 0) o[(size_t)j * nx + xg] = q;
          if (yg >= 0 && xg >= 0) o[(size_t)yg * nx + xg] = q;
        } else if (!A.periodic && !store && j < ny && c < nx) {
          *out = T(0);
        }
      }
      qn += nx; F += nx; out += nx;
      if constexpr (sizeof(T) == 8) s64 += nxi;
      else { shi += nxi; slo += nxi; }
      qc += QW;
      pc += PW;
      pmc = p0c; pmr = p0r; p0c = npc; p0r = npr; e0 = e1;
      fs = fn;
      vs = v;
    }
  };
  if (__all_sync(0xffffffffu, cf && row_full(jb) && row_full(jb + RW - 1))) rows(std::true_type{});
  else rows(std::false_type{});
}

// Tile (x0, y0) of one field; `in`: the tile and its halo lie inside the
// interior, so its loads are plain copies.
template <typename T, int S, int TX, int TY>
DEV void stage_tile(const StageArgs& A, uint8_t* sm, int x0, int y0) {
  using G = Geom<T, S, TX, TY>;
  const bool in = x0 - G::H - G::SH >= 1 && x0 - G::H - G::SH + G::QW - 1 <= A.nx - 2 && y0 - G::H >= 1 &&
                  y0 + TY + G::H - 1 <= A.ny - 2;
  stage_body<T, S, TX, TY>(A, sm, in, x0, y0);
}

// Interior tile rectangle [txa, txb] x [tya, tyb] (empty when txa > txb or
// tya > tyb): the tiles whose loads are plain copies (stage_tile's test,
// solved for the tile index).
struct TileSplit {
  int ntx, nty, txa, txb, tya, tyb;
};

template <typename T, int S, int TX, int TY>
static TileSplit tile_split(int ny, int nx) {
  using G = Geom<T, S, TX, TY>;
  TileSplit t;
  t.ntx = (nx + TX - 1) / TX;
  t.nty = (ny + TY - 1) / TY;
  auto in_x = [&](int x0) { return x0 - G::H - G::SH >= 1 && x0 - G::H - G::SH + G::QW - 1 <= nx - 2; };
  auto in_y = [&](int y0) { return y0 - G::H >= 1 && y0 + TY + G::H - 1 <= ny - 2; };
  t.txa = 0; while (t.txa < t.ntx && !in_x(t.txa * TX)) ++t.txa;
  t.txb = t.txa; while (t.txb + 1 < t.ntx && in_x((t.txb + 1) * TX)) ++t.txb;
  t.tya = 0; while (t.tya < t.nty && !in_y(t.tya * TY)) ++t.tya;
  t.tyb = t.tya; while (t.tyb + 1 < t.nty && in_y((t.tyb + 1) * TY)) ++t.tyb;
  if (t.txa >= t.ntx || t.tya >= t.nty) { t.txa = 1; t.txb = 0; t.tya = 1; t.tyb = 0; }  // no interior tile
  return t;
}

// Block b -> tile: the boundary tiles (the slower loads) get the
// lowest block indices so that they start first instead of forming the
// launch's tail, then the interior rectangle row by row.
DEV void tile_of_block(const TileSplit& t, int b, int& tx, int& ty) {
  const int wi = t.txb - t.txa + 1, hi = t.tyb - t.tya + 1;
  const int ni = (wi > 0 && hi > 0) ? wi * hi : 0;
  const int nb = t.ntx * t.nty - ni;
  if (b >= nb) {
    const int k = b - nb;
    ty = t.tya + k / wi;
    tx = t.txa + k % wi;
    return;
  }
  // rows below the rectangle, rows beside it (the columns outside), rows above
  const int full_lo = ni ? t.tya * t.ntx : nb;
  if (b < full_lo) { ty = b / t.ntx; tx = b % t.ntx; return; }
  const int side = t.ntx - wi;
  const int mid = hi * side;
  if (b < full_lo + mid) {
    const int k = b - full_lo;
    ty = t.tya + k / side;
    const int c = k % side;
    tx = c < t.txa ? c : c + wi;
    return;
  }
  const int k = b - full_lo - mid;
  ty = t.tyb + 1 + k / t.ntx;
  tx = k % t.ntx;
}

// FP32: at most 80 registers, so that six blocks' warps cover a row's chain of
// dependent operations (108 registers without the bound: 457 us per 2048^2
// step against 440); FP64 bodies keep their 106 (four blocks; 80 spill: 256^2
// step 86 us against 77).
template <typename T, int S, int TX, int TY>
__global__ void __launch_bounds__(THREADS, sizeof(T) == 4 ? 6 : 1)
stage_kernel(StageArgs A, TileSplit ts) {
  extern __shared__ __align__(16) uint8_t sm[];
  // launched programmatically: psi comes from the kernel before this one
  grid_dep_wait();
  grid_dep_launch();
  int tx, ty;
  tile_of_block(ts, blockIdx.x, tx, ty);
  stage_tile<T, S, TX, TY>(A, sm, tx * TX, ty * TY);
}

template <typename T, int S, int TX, int TY>
static size_t smem_bytes() {
  using G = Geom<T, S, TX, TY>;
  return (size_t)(G::NQ + G::NP + G::NWEST) * sizeof(T);
}

}  // namespace qg
}  // namespace fvx
