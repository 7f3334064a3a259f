// FP64 transform products of the rectangular spectral solvers, folded by
// parity and run on the FP64 tensor instruction (included by dst.cu).
//
// Every transform used here maps index j -> mir - j of one of its sides to a
// sign, so a length-N product splits into two half-size sums P and Q:
//   MIRROR  C[n] = P[n] + Q[n], C[mir - n] = P[n] - Q[n]  with P the sum over
//           the even input columns and Q over the odd ones.  DST-I (mir =
//           N - 1: S[N-1-n][j] = (-1)^j S[n][j]) and the inverse DCT-II
//           (mir = N - 1, coefficient parity); the inverse periodic
//           transform (mir = N) with cosine coefficients in the even columns
//           and sine coefficients in the odd ones.
//   PAIR    C[2n] = P[n], C[2n+1] = Q[n], on input columns that hold the
//           folded samples x_j + x_{mir-j} (even columns) and x_j - x_{mir-j}
//           (odd ones): the forward DCT-II (even and odd coefficients) and
//           the forward periodic transform (cosine and sine coefficients).
// Both need N^2 / 2 multiply-adds per row instead of N^2.
#pragma once
#include "fvx_common.cuh"

namespace fvx {
namespace dst {

// D (8 x 8) += A (8 x 4, row) B (4 x 8, col): lane l holds A[l/4][l%4],
// B[l%4][l/4] and D[l/4][2(l%4) .. +1].
DEV void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
// Global -> shared copies of which only the first `bytes` are read (the rest
// of the destination is zero-filled).
DEV void cp_async16(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
DEV void cp_async8(uint32_t dst, const double* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> DEV void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct FoldArgs {
  const double* X;      // row m = (b, r) at X + b * xbs + r * xld, K contiguous elements
  long long xbs, xld;
  int R, M, K;          // rows per batch, rows, contraction length
  const double* T;      // table [NH][tld]: column j multiplies input column j
  int tld, NH;
  int mir;              // MIRROR: the mirrored index of n is mir - n; < 0: PAIR
  int n_out;            // output rows per batch
  void* out;            // element (b, n, r) at out[b * obs + n * old + r]
  long long obs, old;
  int out_f32, vec;     // vec: r, r + 1 (r even) of one row may be stored as one vector
  double alpha;
  const double *en, *er;  // eigenvalues along n and r: scale by 1 / (en[n] + er[r] - lam); null: no scale
  const double* lam;
  int n_lam;
};

// TN x TM output tile (TN values of n for both P and Q, TM rows m), four
// warps of (TN / 2) x (TM / 2).  Bound by the FP64 tensor pipe at large
// sizes (an m8n8k4 issues every 16 cycles per SM quarter, 37 TFLOP/s in all)
// and by load and launch latency at 256^2.  The SIMT product it replaces
// ran at 8 TFLOP/s of twice the multiply-adds (a shared load per two FMAs).
// A dependent m8n8k4 takes 26 cycles, so one warp's P and Q chains alone
// keep its quarter of the SM busy and the 16 x 16 tile needs no split of the
// contraction: every output sums over j in the same order whatever the tile.
// Input columns stay in their natural order: one 16-byte shared load of
// columns 2t, 2t + 1 is the even operand of P and the odd one of Q.  16-byte
// chunks are XORed with bit 0 of the row so that the eight lanes of a load
// phase (two rows) cover all banks.  DB: fragments double-buffered in
// registers (the 32 x 32 tile, 12.5 -> 10.9 us at 512^2; it costs the 32 x 64
// tile a resident block and the small ones an earlier barrier).
// Solve of 3 x 1024 x 768: 1114 us (SIMT) -> 300 us; 256^2 QG step 156 -> 94 us.
template <int TN, int TM, int BK, int ST, bool DB, bool XV>
__global__ void __launch_bounds__(128) gemm_f64_fold_kernel(const FoldArgs a) {
  constexpr int WTN = TN / 2, WTM = TM / 2, FN = WTN / 8, FM = WTM / 8;
  constexpr int CPR = BK / 2, RPP = 128 / CPR;  // 16-byte chunks per row, rows per pass of the block
  constexpr int NPT = TN / RPP, NPX = TM / RPP;
  static_assert(TN % RPP == 0 && TM % RPP == 0, "whole passes");
  extern __shared__ __align__(128) uint8_t fold_smem[];
  constexpr uint32_t ROWB = BK * 8, STAGE = (TN + TM) * ROWB;
  const uint32_t sm = (uint32_t)__cvta_generic_to_shared(fold_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = blockIdx.x * TN, m0 = blockIdx.y * TM;
  const int c = tid % CPR, r0 = tid / CPR;
  const int KT = (a.K + BK - 1) / BK;
  // this thread's chunk column c of rows r0, r0 + RPP, ... of both operands
  const double* tp = a.T + (long long)(n0 + r0) * a.tld + 2 * c;
  const double* xp[NPX];
  uint32_t dst[NPX > NPT ? NPX : NPT];
#pragma unroll
  for (int p = 0; p < NPX; ++p) {
    const int m = m0 + r0 + p * RPP;
    if (m < a.M) {
      const int b = m / a.R;
      xp[p] = a.X + b * a.xbs + (long long)(m - b * a.R) * a.xld + 2 * c;
    } else {
      xp[p] = nullptr;
    }
  }
#pragma unroll
  for (int p = 0; p < (NPX > NPT ? NPX : NPT); ++p) {
    const int row = r0 + p * RPP;
    dst[p] = sm + row * ROWB + (uint32_t)((c ^ ((row & 1) << 2)) * 16);
  }
  auto load_t = [&](int kt) {
    const uint32_t off = (uint32_t)(kt % ST) * STAGE;
    const int left = (a.K - kt * BK - 2 * c) * 8;  // bytes of the row from this chunk on
    const int nb = left >= 16 ? 16 : (left > 0 ? left : 0);
#pragma unroll
    for (int p = 0; p < NPT; ++p) {
      const bool ok = nb > 0 && n0 + r0 + p * RPP < a.NH;
      cp_async16(dst[p] + off, ok ? tp + (long long)p * RPP * a.tld + kt * BK : a.T, ok ? nb : 0);
    }
  };
  auto load_x = [&](int kt) {
    const uint32_t off = (uint32_t)(kt % ST) * STAGE + TN * ROWB;
    const int left = (a.K - kt * BK - 2 * c) * 8;
    const int nb = left >= 16 ? 16 : (left > 0 ? left : 0);
#pragma unroll
    for (int p = 0; p < NPX; ++p) {
      const bool ok = nb > 0 && xp[p];
      const double* s = ok ? xp[p] + kt * BK : a.X;
      if constexpr (XV) {
        cp_async16(dst[p] + off, s, ok ? nb : 0);
      } else {
        cp_async8(dst[p] + off, s, ok ? 8 : 0);
        cp_async8(dst[p] + off + 8, ok && nb == 16 ? s + 1 : a.X, ok && nb == 16 ? 8 : 0);
      }
    }
  };
  // the tables are constant; X belongs to the kernel before until the wait
  for (int s = 0; s < ST - 1 && s < KT; ++s) load_t(s);
  grid_dep_wait();
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (s < KT) load_x(s);
    cp_async_commit();
  }
  double P[FN][FM][2] = {}, Q[FN][FM][2] = {};
  const int wn = (warp >> 1) * WTN, wm = (warp & 1) * WTM;
  const int lr = lane >> 2, lt = lane & 3;
  // row of a fragment = multiple of 8 + lr, so its swizzle bit is lr's
  const uint32_t fa = sm + (uint32_t)(wn + lr) * ROWB, fb = sm + (uint32_t)(TN + wm + lr) * ROWB;
  const uint32_t sw = (uint32_t)((lr & 1) << 2);
  constexpr int NK = BK / 8;
  double2 va[DB ? 2 : 1][FN], vb[DB ? 2 : 1][FM];
  auto frags = [&](int kt, int k8, int buf) {
    const uint32_t o = (uint32_t)(kt % ST) * STAGE + (((uint32_t)(k8 * 4 + lt)) ^ sw) * 16;
#pragma unroll
    for (int i = 0; i < FN; ++i)
      asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];"
                   : "=d"(va[buf][i].x), "=d"(va[buf][i].y)
                   : "r"(fa + o + i * 8 * ROWB));
#pragma unroll
    for (int j = 0; j < FM; ++j)
      asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];"
                   : "=d"(vb[buf][j].x), "=d"(vb[buf][j].y)
                   : "r"(fb + o + j * 8 * ROWB));
  };
  auto multiply = [&](int buf) {
#pragma unroll
    for (int i = 0; i < FN; ++i)
#pragma unroll
      for (int j = 0; j < FM; ++j) {
        mma_f64(P[i][j], va[buf][i].x, vb[buf][j].x);
        mma_f64(Q[i][j], va[buf][i].y, vb[buf][j].y);
      }
  };
  static_assert(NK % 2 == 0, "the buffer of a stage's first columns is fixed");
  if constexpr (DB) {
    cp_async_wait<ST - 2>();
    __syncthreads();
    frags(0, 0, 0);
  }
  for (int kt = 0; kt < KT; ++kt) {
    if constexpr (!DB) {
      cp_async_wait<ST - 2>();
      __syncthreads();
    }
    // stage (kt + ST - 1) % ST was read before the last barrier
    if (kt + ST - 1 < KT) {
      load_t(kt + ST - 1);
      load_x(kt + ST - 1);
    }
    cp_async_commit();
#pragma unroll
    for (int k8 = 0; k8 < NK; ++k8) {
      if constexpr (DB) {  // the next 8 columns' fragments load while these are multiplied
        if (k8 + 1 < NK) {
          frags(kt, k8 + 1, (k8 + 1) & 1);
        } else if (kt + 1 < KT) {
          cp_async_wait<ST - 2>();
          __syncthreads();
          frags(kt + 1, 0, 0);
        }
        multiply(k8 & 1);
      } else {
        frags(kt, k8, 0);
        multiply(0);
      }
    }
  }
  // the next kernel may launch while this one stores its results
  grid_dep_launch();
  // Epilogue through the idle ring, [P, Q][TN][TM] doubles with the same
  // chunk swizzle, then one short loop over rows of whole-tile stores.  (A
  // store per fragment, unrolled, took 12 of 67 us at 3 x 1024 x 768: tens of
  // KB of straight-line code run once per block, and 64-byte segments.)
  static_assert(2 * TN * TM * 8 <= ST * (TN + TM) * BK * 8, "the tile fits in the ring");
  cp_async_wait<0>();
  __syncthreads();
  double2* tile = (double2*)fold_smem;
  constexpr int CM = TM / 2, QO = TN * CM;  // chunks per row, offset of Q
#pragma unroll
  for (int i = 0; i < FN; ++i)
#pragma unroll
    for (int j = 0; j < FM; ++j) {
      const int row = wn + i * 8 + lr, ch = ((wm + j * 8) / 2 + lt) ^ (int)sw;
      tile[row * CM + ch] = make_double2(P[i][j][0], P[i][j][1]);
      tile[QO + row * CM + ch] = make_double2(Q[i][j][0], Q[i][j][1]);
    }
  __syncthreads();
  static_assert(128 % CM == 0, "a thread keeps its column pair");
  const int ch = tid % CM, m = m0 + 2 * ch;
  if (m >= a.M) return;
  const int b0 = m / a.R, q0 = m - b0 * a.R;
  const bool two = m + 1 < a.M;
  const int b1 = q0 + 1 < a.R ? b0 : b0 + 1, q1 = q0 + 1 < a.R ? q0 + 1 : 0;
  double er0 = 0, er1 = 0, l0 = 0, l1 = 0;
  if (a.er) {  // (e_n + e_r) - lambda below, in that order
    er0 = a.er[q0];
    l0 = a.lam[b0 % a.n_lam];
    if (two) {
      er1 = a.er[q1];
      l1 = a.lam[b1 % a.n_lam];
    }
  }
  auto put = [&](int n, double x0, double x1) {
    x0 *= a.alpha;
    x1 *= a.alpha;
    if (a.er) {
      // a zero eigenvalue (the null mode of a Poisson problem) divides out as 0
      const double e = a.en[n], d0 = (e + er0) - l0, d1 = (e + er1) - l1;
      x0 *= d0 == 0.0 ? 0.0 : 1.0 / d0;
      x1 *= d1 == 0.0 ? 0.0 : 1.0 / d1;
    }
    const long long i0 = b0 * a.obs + (long long)n * a.old + q0, i1 = b1 * a.obs + (long long)n * a.old + q1;
    if (a.out_f32) {
      float* o = (float*)a.out;
      if (a.vec) {
        *(float2*)(o + i0) = make_float2((float)x0, (float)x1);
      } else {
        o[i0] = (float)x0;
        if (two) o[i1] = (float)x1;
      }
    } else {
      double* o = (double*)a.out;
      if (a.vec) {
        *(double2*)(o + i0) = make_double2(x0, x1);
      } else {
        o[i0] = x0;
        if (two) o[i1] = x1;
      }
    }
  };
#pragma unroll 2
  for (int row = tid / CM; row < TN; row += 128 / CM) {
    const int n = n0 + row;
    if (n >= a.NH) break;
    const int o = row * CM + (ch ^ ((row & 1) << 2));
    const double2 p = tile[o], q = tile[QO + o];
    const bool mirror = a.mir >= 0;
    const int n1 = mirror ? n : 2 * n, n2 = mirror ? a.mir - n : 2 * n + 1;
    put(n1, mirror ? p.x + q.x : p.x, mirror ? p.y + q.y : p.y);
    // MIRROR: the middle (or first periodic) row has no partner
    if (!mirror || (n2 > n && n2 < a.n_out)) put(n2, mirror ? p.x - q.x : q.x, mirror ? p.y - q.y : q.y);
  }
}

// Samples of a [batch][ny][nx] view folded along both axes into
// [batch][2 hy][2 hx]: column 2a holds x_a + x_{mir-a}, column 2a + 1 the
// difference (a sample that is its own partner, or has none, stands alone:
// the sum is the sample, the difference 0); rows likewise.
template <typename T>
__global__ void fold_in_f64_kernel(const T* in, long long bstride, long long ld, int ny, int nx, int hy, int hx,
                                   int miry, int mirx, int batch, double* out) {
  grid_dep_wait();
  const int rows = batch * hy;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const int b = row / hy, y = row - b * hy, y2 = miry - y;
    const bool py = y2 > y && y2 < ny;
    const T* s0 = in + b * bstride + (long long)y * ld;
    const T* s1 = in + b * bstride + (long long)y2 * ld;
    double* o0 = out + ((long long)b * hy + y) * 2 * (2 * hx);
    double* o1 = o0 + 2 * hx;
    for (int x = threadIdx.x; x < hx; x += blockDim.x) {
      const int x2 = mirx - x;
      const bool px = x2 > x && x2 < nx;
      const double a0 = (double)__ldcg(s0 + x), a1 = px ? (double)__ldcg(s0 + x2) : 0.0;
      const double b0 = py ? (double)__ldcg(s1 + x) : 0.0, b1 = py && px ? (double)__ldcg(s1 + x2) : 0.0;
      const double as = px ? a0 + a1 : a0, ad = px ? a0 - a1 : 0.0;
      const double bs = px ? b0 + b1 : b0, bd = px ? b0 - b1 : 0.0;
      *(double2*)(o0 + 2 * x) = py ? make_double2(as + bs, ad + bd) : make_double2(as, ad);
      *(double2*)(o1 + 2 * x) = py ? make_double2(as - bs, ad - bd) : make_double2(0.0, 0.0);
    }
  }
  grid_dep_launch();
}

template <int TN, int TM, int BK, int ST, bool DB>
static int launch_fold(const FoldArgs& a, bool xv, cudaStream_t st) {
  constexpr int smem = ST * (TN + TM) * BK * 8;
  static fvx_once_per_device attr;
  if (fvx_once_on_device(attr, [] {
        return fvx_set_max_smem(gemm_f64_fold_kernel<TN, TM, BK, ST, DB, true>, smem) &&
               fvx_set_max_smem(gemm_f64_fold_kernel<TN, TM, BK, ST, DB, false>, smem);
      }))
    return FVX_ERR_CUDA;
  const dim3 grid((a.NH + TN - 1) / TN, (a.M + TM - 1) / TM);
  if (grid.y > 65535) return FVX_ERR_SHAPE;
  const cudaError_t e =
      xv ? fvx_launch_pdl(gemm_f64_fold_kernel<TN, TM, BK, ST, DB, true>, grid, dim3(128), smem, st, a)
         : fvx_launch_pdl(gemm_f64_fold_kernel<TN, TM, BK, ST, DB, false>, grid, dim3(128), smem, st, a);
  return e == cudaSuccess ? fvx_cuda_status() : FVX_ERR_CUDA;
}

// Tile shapes and what c tiles on one SM take per column of the contraction,
// in ns, measured over 96^2 .. 2048^2 and batches: g[c] for c up to the r
// blocks that an SM holds at once, whole groups of r after that.  The 16 x 16
// tile is bound by its shared loads (two per two products), the larger ones
// by the tensor pipe once enough blocks hide each other's barriers.
struct FoldTile {
  int tn, tm, r;
  float g[5];
};
constexpr FoldTile kFoldTiles[4] = {{16, 16, 2, {0, 4.5f, 9.4f}},
                                    {32, 16, 2, {0, 11.f, 13.f}},
                                    {32, 32, 3, {0, 17.5f, 28.f, 33.f}},
                                    {32, 64, 4, {0, 32.f, 53.f, 62.f, 81.f}}};

// One folded product on the tile with the least work on the fullest SM, of
// those whose rows fit the grid's 65535 blocks in y (e.g. us per product, 16 x
// 16 / 32 x 16 / 32 x 32 / 32 x 64: 256^2 3.3 / 4.2 / 6.5 / 11, 512^2 11.5 /
// 8.7 / 10.9 / 18.6, 896^2 45 / 39 / 32 / 46, 2048^2 - / - / 323 / 280).  The
// result does not depend on the tile.
static int gemm_f64_fold(FoldArgs a, cudaStream_t st) {
  // 16-byte loads of X need even row and batch pitches and an aligned base
  const bool xv = ((uintptr_t)a.X & 15) == 0 && a.xld % 2 == 0 && a.xbs % 2 == 0;
  const uintptr_t oa = a.out_f32 ? 8 : 16;
  a.vec = a.R % 2 == 0 && ((uintptr_t)a.out & (oa - 1)) == 0 && a.old % 2 == 0 && a.obs % 2 == 0;
  int best = -1;
  double least = 0;
  for (int k = 0; k < 4; ++k) {
    const FoldTile& t = kFoldTiles[k];
    if ((a.M + t.tm - 1) / t.tm > 65535) continue;
    const long long tiles = (long long)((a.NH + t.tn - 1) / t.tn) * ((a.M + t.tm - 1) / t.tm);
    const long long c = (tiles + 147) / 148;
    const double cost = (double)(c / t.r) * t.g[t.r] + t.g[c % t.r];
    if (best < 0 || cost < least) { best = k; least = cost; }
  }
  switch (best) {
    case 0: return launch_fold<16, 16, 64, 5, false>(a, xv, st);
    case 1: return launch_fold<32, 16, 64, 4, false>(a, xv, st);
    case 2: return launch_fold<32, 32, 32, 4, true>(a, xv, st);
    default: return launch_fold<32, 64, 16, 4, false>(a, xv, st);
  }
}

}  // namespace dst
}  // namespace fvx
