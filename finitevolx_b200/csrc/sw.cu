// Shallow-water operators on the Arakawa C-grid, each one fused kernel:
// Coriolis2D (operators/coriolis.py:34-133), Vorticity2D's potential
// vorticity and PV fluxes (operators/vorticity.py:60-235) and
// MomentumAdvection2D (diffusion/momentum.py:35-216).
//
// The reference composes Interpolation2D / Difference2D calls, each writing
// a full staggered array with a zero ghost ring and (under a mask) the
// output stagger's mask applied.  Here the intermediates live in registers,
// with the same arithmetic, ring and mask rules (T -> mask.h, U -> mask.u, V ->
// mask.v, X -> mask.xy_corner_strict); quotients by dx and dy are products
// with their reciprocals (within an ulp of the quotients).
#include "fvx_common.cuh"

namespace fvx {
namespace sw {

enum SwOp {
  CORIOLIS = 0,        // (u, v, f) -> (du, dv)
  PV_FLUX_ENERGY = 1,  // (q, u, v) -> (qu, qv)
  PV_FLUX_ENSTROPHY = 2,
  PV_FLUX_AL = 3,      // alpha blend
  MOM_ENERGY = 4,      // (u, v) -> (du, dv)
  MOM_ENSTROPHY = 5,
  MOM_AL = 6,
  POT_VORTICITY = 7,   // (u, v, h, f) -> q
  N_OPS = 8
};

template <typename T>
struct Fields {
  const T *a, *b, *c, *d;
  int ny, nx;
  T rdx, rdy, alpha, beta;  // beta = 1 - alpha, rounded once from the double
  const uint8_t *mh, *mu, *mv, *mxy;
};

// A lane owns a column and marches down its rows: values of the row above are
// carried, those of the columns to the left and right come from the
// neighbouring lanes (lanes 0 and 31 only feed their neighbours: 30 output
// columns per warp).  Every input element is loaded once per warp, every
// corner vorticity and kinetic energy formed once; bound by memory (36 bytes
// per cell, FP64 momentum) and, below ~10^6 cells, by the march's latency.
// The per-cell form it replaces re-read and recomputed all of them at every
// output (9 FP64 divisions and a 64-bit index division per cell): Coriolis
// plus Arakawa-Lamb momentum at 1020 x 764 FP64 took 59 us.
constexpr int kWarps = 4, kCols = 30;
template <typename T, int OP>
__global__ void __launch_bounds__(32 * kWarps)
sw_kernel(Fields<T> F, int RW, T* __restrict__ o1, T* __restrict__ o2) {
  constexpr bool MOM = OP == MOM_ENERGY || OP == MOM_ENSTROPHY || OP == MOM_AL;
  constexpr bool PVF = OP == PV_FLUX_ENERGY || OP == PV_FLUX_ENSTROPHY || OP == PV_FLUX_AL;
  constexpr bool PE = OP == PV_FLUX_ENERGY || OP == PV_FLUX_AL || OP == MOM_ENERGY || OP == MOM_AL;
  constexpr bool PZ = OP == PV_FLUX_ENSTROPHY || OP == PV_FLUX_AL || OP == MOM_ENSTROPHY || OP == MOM_AL;
  constexpr bool PV = OP == POT_VORTICITY;
  const int ny = F.ny, nx = F.nx, lane = threadIdx.x & 31;
  const int i = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * kCols + lane - 1;
  const int j0 = blockIdx.y * RW, j1 = min(ny, j0 + RW);
  if (i - lane + 1 >= nx) return;  // the whole warp
  const bool ci = i >= 0 && i < nx, cin = i >= 1 && i <= nx - 2;
  const bool put = lane >= 1 && lane <= kCols && ci;
  const T *pu = MOM || OP == CORIOLIS || PV ? F.a : F.b, *pv = MOM || OP == CORIOLIS || PV ? F.b : F.c;
  // one row's inputs of this column (zero outside the array; masks 1 when absent)
  struct Row { T u, v, q, d, mh, mu, mv, mxy; };
  auto load = [&](int j) -> Row {
    Row r = {T(0), T(0), T(0), T(0), T(1), T(1), T(1), T(1)};
    if (!ci || j < 0 || j >= ny) return r;
    const size_t k = (size_t)j * nx + i;
    r.u = pu[k];
    r.v = pv[k];
    if constexpr (OP == CORIOLIS || PV) r.q = F.c[k];  // f or h
    if constexpr (PVF) r.q = F.a[k];
    if constexpr (PV) r.d = F.d[k];
    if constexpr (MOM) { if (F.mh) r.mh = T(F.mh[k]); }
    if constexpr (!PV) {
      if (F.mu) r.mu = T(F.mu[k]);
      if (F.mv) r.mv = T(F.mv[k]);
    }
    if constexpr (OP != CORIOLIS) { if (F.mxy) r.mxy = T(F.mxy[k]); }
    return r;
  };
  auto rgt = [&](T x) { return __shfl_down_sync(0xffffffffu, x, 1); };
  auto lft = [&](T x) { return __shfl_up_sync(0xffffffffu, x, 1); };
  auto inr = [&](int j) { return cin && j >= 1 && j <= ny - 2; };
  // corner vorticity (difference.py:47-59), kinetic energy (momentum.py:108-122)
  auto curl = [&](T v, T ve, T u, T up, int j, T mxy) -> T {
    return inr(j) ? ((ve - v) * F.rdx - (up - u) * F.rdy) * mxy : T(0);
  };
  auto kin = [&](T u, T uw, T v, T vs, int j, T m) -> T {
    if (!inr(j)) return T(0);
    const T ut = T(0.5) * (u + uw) * m, vt = T(0.5) * (v + vs) * m;
    return T(0.5) * (ut * ut + vt * vt);
  };
  // rows j0 - 1, j0, j0 + 1 in flight together; in the march each row's loads
  // are issued one row before they are used
  const Row A = load(j0 - 1);
  Row B = load(j0), C = load(j0 + 1);
  T vm = A.v, vme = rgt(A.v), uw0 = lft(B.u);
  T qm = A.q, zm = T(0), zum = T(0), zvm = T(0), k0 = T(0);
  if constexpr (MOM) {
    zm = curl(A.v, vme, A.u, B.u, j0 - 1, A.mxy);
    k0 = kin(B.u, uw0, B.v, A.v, j0, B.mh);
  }
  if constexpr (PZ) {
    // MOM: X_to_U of zeta V_to_X(v) and X_to_V of zeta U_to_X(u); PV
    // fluxes: X_to_U of q U_to_X(u) and X_to_V of q V_to_X(v)
    const T z = MOM ? zm : A.q;
    zum = inr(j0 - 1) ? z * (T(0.5) * (A.u + B.u) * A.mxy) : T(0);
    zvm = inr(j0 - 1) ? z * (T(0.5) * (A.v + vme) * A.mxy) : T(0);
  }
  for (int j = j0; j < j1; ++j) {
    Row N = {};
    if (j + 1 < j1) N = load(j + 2);
    const T u0 = B.u, v0 = B.v, up = C.u;
    const T ve = rgt(v0), uwp = lft(up);
    const bool in = inr(j);
    T r1 = T(0), r2 = T(0);
    if constexpr (OP == CORIOLIS) {  // a = u, b = v, c = f; unmasked interpolation, final mask
      const T fe = rgt(B.q);
      if (in) {
        r1 = (T(0.5) * (B.q + fe)) * (T(0.25) * (v0 + vm + ve + vme));
        r2 = -(T(0.5) * (B.q + C.q)) * (T(0.25) * (u0 + up + uw0 + uwp));
      }
      r1 = r1 * B.mu;
      r2 = r2 * B.mv;
    } else if constexpr (PV) {  // a = u, b = v, c = h, d = f; vorticity.py:60-118
      const T he = rgt(B.q), de = rgt(B.d), hpe = rgt(C.q), dpe = rgt(C.d);
      if (in) {
        const T num = ((ve - v0) * F.rdx - (up - u0) * F.rdy) * B.mxy + T(0.25) * (B.d + de + C.d + dpe) * B.mxy;
        const T den = T(0.25) * (B.q + he + C.q + hpe) * B.mxy;
        r1 = den == T(0) ? T(NAN) : num / den;
      }
      if (B.mxy == T(0)) r1 = T(0);
    } else {
      const T mxy = B.mxy, mu = B.mu, mv = B.mv;
      const T z = MOM ? curl(v0, ve, u0, up, j, mxy) : B.q;
      const T zs = MOM ? zm : qm, zl = lft(z);  // the corners below and to the left
      T e1 = T(0), e2 = T(0), s1 = T(0), s2 = T(0);
      if constexpr (PE) {
        if (in) {
          const T zu = T(0.5) * (z + zs) * mu, zv = T(0.5) * (z + zl) * mv;
          e1 = zu * (MOM ? T(0.25) * (v0 + vm + ve + vme) * mu : u0);
          e2 = zv * (MOM ? T(0.25) * (u0 + up + uw0 + uwp) * mv : v0);
        }
      }
      if constexpr (PZ) {
        const T zu = in ? z * (T(0.5) * (u0 + up) * mxy) : T(0), zv = in ? z * (T(0.5) * (v0 + ve) * mxy) : T(0);
        const T zul = lft(zu), zvl = lft(zv);
        if (in) {
          s1 = T(0.5) * (MOM ? zv + zvm : zu + zum) * mu;
          s2 = T(0.5) * (MOM ? zu + zul : zv + zvl) * mv;
        }
        zum = zu;
        zvm = zv;
      }
      constexpr bool AL = OP == PV_FLUX_AL || OP == MOM_AL;
      r1 = AL ? F.alpha * e1 + F.beta * s1 : (PE ? e1 : s1);
      r2 = AL ? F.alpha * e2 + F.beta * s2 : (PE ? e2 : s2);
      if constexpr (MOM) {  // momentum.py:124-216
        const T kp = kin(up, uwp, C.v, v0, j + 1, C.mh), ke = rgt(k0);
        const bool out = j >= 2 && j <= ny - 3 && i >= 2 && i <= nx - 3;
        r1 = out ? (r1 - (ke - k0) * F.rdx * mu) * mu : T(0);
        r2 = out ? (-r2 - (kp - k0) * F.rdy * mv) * mv : T(0);
        k0 = kp;
      }
      zm = z;
      qm = B.q;
    }
    if (put) {
      const size_t k = (size_t)j * nx + i;
      o1[k] = r1;
      if (!PV) o2[k] = r2;
    }
    vm = v0;
    vme = ve;
    uw0 = uwp;
    B = C;
    C = N;
  }
}

// 16 rows per march on large fields (the two rows around the march cost 1/8
// more loads), fewer on small ones, where a march's chain of rows is the
// kernel's time, and more where the marches would not fit the grid's y.
// Coriolis plus Arakawa-Lamb momentum, FP64, masked, before -> now: 2400^2 382
// -> 127 us, 1020 x 764 52.9 -> 19.3, 130 x 98 7.9 -> 4.2.
template <typename T, int OP>
static int launch(const Fields<T>& F, T* o1, T* o2, cudaStream_t st) {
  const long long cells = (long long)F.ny * F.nx;
  int RW = cells >= 2000000 ? 16 : (cells >= 400000 ? 8 : (cells >= 100000 ? 4 : 1));
  while (F.ny > 65535LL * RW) RW *= 2;
  const dim3 g((F.nx + kWarps * kCols - 1) / (kWarps * kCols), (unsigned)((F.ny - 1LL) / RW + 1));
  sw_kernel<T, OP><<<g, 32 * kWarps, 0, st>>>(F, RW, o1, o2);
  return fvx_cuda_status();
}
template <typename T>
static int dispatch(int op, const Fields<T>& F, T* o1, T* o2, cudaStream_t st) {
  switch (op) {
    case CORIOLIS: return launch<T, CORIOLIS>(F, o1, o2, st);
    case PV_FLUX_ENERGY: return launch<T, PV_FLUX_ENERGY>(F, o1, o2, st);
    case PV_FLUX_ENSTROPHY: return launch<T, PV_FLUX_ENSTROPHY>(F, o1, o2, st);
    case PV_FLUX_AL: return launch<T, PV_FLUX_AL>(F, o1, o2, st);
    case MOM_ENERGY: return launch<T, MOM_ENERGY>(F, o1, o2, st);
    case MOM_ENSTROPHY: return launch<T, MOM_ENSTROPHY>(F, o1, o2, st);
    case MOM_AL: return launch<T, MOM_AL>(F, o1, o2, st);
    default: return launch<T, POT_VORTICITY>(F, o1, o2, st);
  }
}

}  // namespace sw
}  // namespace fvx

using namespace fvx;
using namespace fvx::sw;

// op as SwOp; a..d inputs (see SwOp); masks may be NULL (unmasked);
// out2 unused (NULL) for POT_VORTICITY.  Coriolis applies mask_u / mask_v
// to its outputs only; the others pass the masks down to every
// intermediate like the reference's masked Difference2D / Interpolation2D.
#define FVX_DEF_SW(SFX, T)                                                                                        \
  extern "C" int fvx_sw2d_##SFX(int op, const T* a, const T* b, const T* c, const T* d, T* out1, T* out2, int ny, \
                                int nx, double dx, double dy, double alpha, const uint8_t* mask_h,               \
                                const uint8_t* mask_u, const uint8_t* mask_v, const uint8_t* mask_xy,            \
                                void* stream) {                                                                   \
    if (op < 0 || op >= N_OPS) return FVX_ERR_METHOD;                                                             \
    if (!a || !b || !out1 || (op != POT_VORTICITY && !out2)) return FVX_ERR_ARG;                                  \
    if ((op <= PV_FLUX_AL || op == POT_VORTICITY) && !c) return FVX_ERR_ARG;                                      \
    if (op == POT_VORTICITY && !d) return FVX_ERR_ARG;                                                            \
    if (ny < 3 || nx < 3) return FVX_ERR_SHAPE;                                                                   \
    Fields<T> F{a, b, c, d, ny, nx, T(1.0 / dx), T(1.0 / dy), T(alpha), T(1.0 - alpha), mask_h, mask_u, mask_v,  \
                mask_xy};                                                                                         \
    return dispatch<T>(op, F, out1, out2, fvx_stream(stream));                                                    \
  }

FVX_DEF_SW(f32, float)
FVX_DEF_SW(f64, double)
