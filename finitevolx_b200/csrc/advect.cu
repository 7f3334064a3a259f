// Flux-form advection (Advection2D.__call__, advection/advection.py:329-420):
//   out[2:-2,2:-2] = -((fe[j,i]-fe[j,i-1])/dx + (fn[j,i]-fn[j-1,i])/dy),
//   zero elsewhere, then * mask.h when a mask is given.
// Masked dispatchable methods pick, per face, the reconstruction of the tier
// of the upwind cell (upwind_flux, advection/flux.py:221-253).
#include "march.cuh"

#include <type_traits>

namespace fvx {
namespace adv {

constexpr int THREADS = 128;

// h tile: rows y0-H .. y0+TY+H-1, columns x0-H .. x0+TX+H-1 at [ly * HW + SH +
// lx] (SH: rows start at an even column, 8-byte copies in FP32).
template <typename T, int S, int TX, int TY>
struct Geom {
  static constexpr int R = MarchWin<S>::R, W = MarchWin<S>::W, H = R + 1, SH = H & 1;
  static constexpr int HW = (TX + 2 * H + SH + 1) & ~1, HH = TY + 2 * H;
  static constexpr int RW = TX * TY / THREADS;  // rows a thread marches
  static constexpr int NWEST = TY * (TX / 32);  // west faces no lane to the left has
  static constexpr int SMEM = (HH * HW + NWEST) * (int)sizeof(T);
  static_assert(RW * THREADS == TX * TY && TY % RW == 0 && NWEST <= THREADS && TX % 32 == 0, "whole marches");
};

// A thread marches down a column of the tile (march.cuh); u and v are read
// straight from memory, one row ahead.  MASKED: tier codes per cell (bits 0-1
// x, 2-3 y: 0 dry, 1 first order, 2 third, 3 full) bound each face's reach by
// the upwind cell's tier; a march over full-tier cells only runs the same
// loop as without a mask.  Bound by instruction issue (FP32) and the FP64
// pipe.  The tile kernel it replaces kept faces in shared memory, a loop per
// array, with scalar boundary ladders at every face.
template <typename T, int S, bool MASKED, int TX, int TY>
__global__ void __launch_bounds__(THREADS, sizeof(T) == 4 ? 6 : 1)
advect_march_kernel(const T* __restrict__ h, const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ out,
                    int ny, int nx, T rdx, T rdy, const uint8_t* __restrict__ tiers, const uint8_t* __restrict__ mh) {
  using G = Geom<T, S, TX, TY>;
  constexpr int R = G::R, W = G::W, H = G::H, HW = G::HW, HH = G::HH, RW = G::RW;
  extern __shared__ __align__(16) uint8_t adv_smem[];
  T* base = (T*)adv_smem;
  T* ht = base + G::SH;
  T* west = base + HH * HW;  // [TX / 32][TY]
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, tid = threadIdx.x;
  if (x0 - H - G::SH >= 0 && x0 - H - G::SH + HW <= nx && y0 - H >= 0 && y0 + TY + H <= ny) {
    const bool v8 = ((uintptr_t)h & 7) == 0 && (nx & 1) == 0;
    tile_copy<T, THREADS, HH, HW, HW>(base, h + (size_t)(y0 - H) * nx + (x0 - H - G::SH), nx, v8, tid);
  } else {
    for (int k = tid; k < HH * (HW - G::SH); k += THREADS) {
      const int ly = k / (HW - G::SH), lx = k - ly * (HW - G::SH);
      const int gy = y0 - H + ly, gx = x0 - H + lx;
      if (gy >= 0 && gy < ny && gx >= 0 && gx < nx) cp_async_elem(ht + ly * HW + lx, h + (size_t)gy * nx + gx);
      else ht[ly * HW + lx] = T(0);
    }
  }
  constexpr int E = R > 2 ? R : 2;
  auto row_full = [&](int j) { return j >= E && j + 1 <= ny - 1 - R; };
  auto col_full = [&](int c) { return c >= E && c + 1 <= nx - 1 - R; };
  auto inside = [&](int j, int c) { return j >= 1 && j <= ny - 2 && c >= 1 && c <= nx - 2; };
  auto tier = [&](int j, int c) -> int { return j >= 0 && j < ny && c >= 0 && c < nx ? tiers[(size_t)j * nx + c] : 0; };
  constexpr int FULLX = R >= 2 ? 3 : 2;  // the tier that allows the scheme itself (third-order schemes: 2 and 3)
  auto full_tier = [&](int t) { return (t & 3) >= FULLX && (t >> 2 & 3) >= FULLX; };
  // flux through a face next to an edge or a coast (axis: 0 x, 1 y)
  auto edge_flux = [&](const T(&w)[W], T vel, int j, int c, int axis) -> T {
    if (!inside(j, c)) return T(0);
    const bool pos = vel >= T(0);
    int r = axis ? march_reach<S>(j, ny, pos) : march_reach<S>(c, nx, pos);
    if constexpr (MASKED) {
      const int code = axis ? tier(pos ? j : j + 1, c) >> 2 & 3 : tier(j, pos ? c : c + 1) & 3;
      if (code == 0) return T(0) * vel;
      r = min(r, min(R, code - 1));
    }
    return march_edge_face<T, S>(w, pos, r) * vel;
  };
  const int col = tid % TX, seg = tid / TX, c = x0 + col, jb = y0 + seg * RW;
  const T* hc = ht + (seg * RW + H) * HW + (col + H);  // h (jb, c)
  const bool cf = col_full(c);
  const bool cin = c >= 1 && c <= nx - 2;
  // ---- west faces of the tile's column groups, south face of the march ------
  const int t = tid < G::NWEST ? tid : 0;
  const int grp = t / TY, wr = t - grp * TY, jw = y0 + wr, cw = x0 + grp * 32 - 1, js = jb - 1;
  const T uw = inside(jw, cw) ? u[(size_t)jw * nx + cw] : T(0);
  const T vs = inside(js, c) ? v[(size_t)js * nx + c] : T(0);
  bool wide = cf && row_full(js) && row_full(jb + RW - 1);  // the march and its south face
  bool whole = wide && row_full(jw) && col_full(cw);
  if constexpr (MASKED) {
    if (__all_sync(0xffffffffu, wide)) {
      // rows js .. jb + RW of columns c and c + 1: every upwind cell the march may use
      const uint8_t* tp = tiers + (size_t)js * nx + c;
      bool ok = true;
#pragma unroll
      for (int r = 0; r <= RW + 1; ++r) ok = ok & full_tier(tp[(size_t)r * nx]) & full_tier(tp[(size_t)r * nx + 1]);
      wide = ok;
      whole = whole && ok;
    } else {
      wide = whole = false;
    }
    whole = whole && full_tier(tier(jw, cw)) && full_tier(tier(jw, cw + 1));
  }
  cp_async_wait_all();
  __syncthreads();
  T wy[W], fs;
  {
    const T* hw = ht + (wr + H) * HW + (grp * 32 - 1 + H);
    T wx[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      wx[k] = hw[k - R];
      wy[k] = hc[(k - R - 1) * HW];
    }
    T fw;
    if (__all_sync(0xffffffffu, whole)) {
      T hx, hy;
      march_faces<T, S>(wx, wy, uw >= T(0), vs >= T(0), hx, hy);
      fw = hx * uw;
      fs = hy * vs;
    } else {
      fw = edge_flux(wx, uw, jw, cw, 0);
      fs = edge_flux(wy, vs, js, c, 1);
    }
    if (tid < G::NWEST) west[t] = fw;
  }
  __syncthreads();
  // ---- the march ------------------------------------------------------------
  const bool first = (col & 31) == 0;
  const T* wst = west + (col >> 5) * TY + seg * RW;
  auto rows = [&](auto full_c) {
    constexpr bool FULL = decltype(full_c)::value;
    const long long g0 = (long long)jb * nx + c;
    const T *up = u + g0, *vp = v + g0;
    T* op = out + g0;
    auto load = [&](const T* p, int j) -> T { return FULL || (cin && j >= 1 && j <= ny - 2) ? *p : T(0); };
    T un = load(up, jb), vn = load(vp, jb);
#pragma unroll(FULL ? 4 : 1)
    for (int r = 0; r < RW; ++r) {
      const int j = jb + r;
      const T uu = un, vv = vn;
      up += nx;
      vp += nx;
      if (r + 1 < RW) {
        un = load(up, j + 1);
        vn = load(vp, j + 1);
      }
      T wx[W];
#pragma unroll
      for (int k = 0; k + 1 < W; ++k) wy[k] = wy[k + 1];
      wy[W - 1] = hc[(R + 1) * HW];
#pragma unroll
      for (int k = 0; k < W; ++k) wx[k] = k == R ? wy[R] : hc[k - R];
      T fe, fn;
      bool all = FULL;
      if constexpr (!FULL) {
        all = cf && row_full(j);
        if constexpr (MASKED) all = all && full_tier(tier(j, c)) && full_tier(tier(j, c + 1)) && full_tier(tier(j + 1, c));
        all = __all_sync(0xffffffffu, all);
      }
      if (all) {
        T hx, hy;
        march_faces<T, S>(wx, wy, uu >= T(0), vv >= T(0), hx, hy);
        fe = hx * uu;
        fn = hy * vv;
      } else {
        fe = edge_flux(wx, uu, j, c, 0);
        fn = edge_flux(wy, vv, j, c, 1);
      }
      T fw = __shfl_up_sync(0xffffffffu, fe, 1);
      if (first) fw = wst[r];
      T res = -((fe - fw) * rdx + (fn - fs) * rdy);
      if constexpr (FULL) {
        if (!MASKED && mh) res = res * T(mh[g0 + (long long)r * nx]);
        *op = res;
      } else {
        if (!(j >= 2 && j <= ny - 3 && c >= 2 && c <= nx - 3)) res = T(0);
        if (j < ny && c < nx) {
          if (mh) res = res * T(mh[g0 + (long long)r * nx]);
          *op = res;
        }
      }
      op += nx;
      hc += HW;
      fs = fn;
    }
  };
  if (__all_sync(0xffffffffu, wide)) rows(std::true_type{});
  else rows(std::false_type{});
}

template <typename T, int S, bool MASKED, int TX, int TY>
static int launch_t(const T* h, const T* u, const T* v, T* out, int ny, int nx, double dx, double dy,
                    const uint8_t* tiers, const uint8_t* mh, cudaStream_t st) {
  using G = Geom<T, S, TX, TY>;
  const dim3 g((nx + TX - 1) / TX, (ny + TY - 1) / TY);
  if (g.y > 65535) return FVX_ERR_SHAPE;
  advect_march_kernel<T, S, MASKED, TX, TY>
      <<<g, THREADS, G::SMEM, st>>>(h, u, v, out, ny, nx, T(1.0 / dx), T(1.0 / dy), tiers, mh);
  return fvx_cuda_status();
}
// 16-row marches (64 x 32 tiles) once they fill the SMs several times over,
// else 4-row ones (32 x 16).
template <typename T, int S, bool MASKED>
static int launch(const T* h, const T* u, const T* v, T* out, int ny, int nx, double dx, double dy,
                  const uint8_t* tiers, const uint8_t* mh, cudaStream_t st) {
  if ((long long)ny * nx >= 2500000) return launch_t<T, S, MASKED, 64, 32>(h, u, v, out, ny, nx, dx, dy, tiers, mh, st);
  return launch_t<T, S, MASKED, 32, 16>(h, u, v, out, ny, nx, dx, dy, tiers, mh, st);
}

// Minimum line length each scheme's boundary ladder is defined for.
static int min_len(int m) {
  switch (m) {
    case FVX_WENO9: return 8;   // shortest line the reference's ladder concatenation accepts
    case FVX_WENO7: return 6;
    case FVX_WENO5: case FVX_WENOZ5: return 4;
    default: return 3;
  }
}

template <typename T>
static int advect2d(const T* h, const T* u, const T* v, T* out, int ny, int nx, double dx, double dy, int method,
                    const uint8_t* tiers, const uint8_t* mh, cudaStream_t st) {
  if (!h || !u || !v || !out) return FVX_ERR_ARG;
  if (method < 0 || method >= FVX_WENOZ3) return FVX_ERR_METHOD;
  if (ny < min_len(method) || nx < min_len(method)) return FVX_ERR_SHAPE;
  if (tiers) {
    if (!mh) return FVX_ERR_ARG;
    switch (method) {
#define FVX_CASE(M) case M: return launch<T, M, true>(h, u, v, out, ny, nx, dx, dy, tiers, mh, st);
      FVX_CASE(FVX_WENO3) FVX_CASE(FVX_WENO5) FVX_CASE(FVX_WENOZ5) FVX_CASE(FVX_MINMOD) FVX_CASE(FVX_VAN_LEER)
      FVX_CASE(FVX_SUPERBEE) FVX_CASE(FVX_MC)
#undef FVX_CASE
      default: return FVX_ERR_METHOD;
    }
  }
  switch (method) {
#define FVX_CASE(M) case M: return launch<T, M, false>(h, u, v, out, ny, nx, dx, dy, nullptr, mh, st);
    FVX_CASE(FVX_NAIVE) FVX_CASE(FVX_UPWIND1) FVX_CASE(FVX_UPWIND2) FVX_CASE(FVX_UPWIND3) FVX_CASE(FVX_WENO3)
    FVX_CASE(FVX_WENO5) FVX_CASE(FVX_WENOZ5) FVX_CASE(FVX_WENO7) FVX_CASE(FVX_WENO9) FVX_CASE(FVX_MINMOD)
    FVX_CASE(FVX_VAN_LEER) FVX_CASE(FVX_SUPERBEE) FVX_CASE(FVX_MC)
#undef FVX_CASE
    default: return FVX_ERR_METHOD;
  }
}

}  // namespace adv
}  // namespace fvx

#define FVX_DEF_ADVECT(SFX, T)                                                                             \
  extern "C" int fvx_advect2d_##SFX(const T* h, const T* u, const T* v, T* out, int ny, int nx, double dx, \
                                    double dy, int method, const uint8_t* tiers, const uint8_t* mask_h,   \
                                    void* stream) {                                                        \
    return fvx::adv::advect2d<T>(h, u, v, out, ny, nx, dx, dy, method, tiers, mask_h, fvx_stream(stream)); \
  }
FVX_DEF_ADVECT(f32, float)
FVX_DEF_ADVECT(f64, double)
