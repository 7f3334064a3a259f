// FP32 transform products folded by parity on the tcgen05 tensor cores, any
// size (included by dst.cu inside its namespace, after the PTX helpers and
// the even/odd product, whose ring and role split it shares).
//
// The algebra is dst_f64.cuh's: the contraction columns are kept in two
// halves, even logical indices (or folded sums, cosine coefficients) first,
// odd ones (differences, sine coefficients) from element `half` on, and the
// two half-length products are
//   P = X_even T_P,  Q = X_odd T_Q      (3xBF16 split each, FP32 in TMEM)
//   MIRROR: C[n] = P + Q, C[mir - n] = P - Q;   PAIR: C[2n] = P, C[2n+1] = Q.
#pragma once

struct FoldEpi {
  Epi e;          // mode, rows_per_batch, m_total, out0/out1, batch_stride, ld, alpha, inv_eig, n_eig, n_cols, err, ...
  int nh;         // table rows
  int mir;        // mirrored index of n is mir - n; < 0: PAIR
  int half_out;   // > 0: store r at (r odd ? half_out : 0) + r / 2, the next product's operand layout
};

// A CTA owns 128 rows x NT table rows of both P and Q (TMEM columns 0..NT-1
// and NT..2NT-1) and loads 128-element-row tiles of A and NT-row tiles of
// the tables per 64-element K block.  Bound by those loads (L2 -> shared
// memory, 4 (128 + NT) bytes per K element, hi and lo) and by latency at
// small sizes; the tensor pipe needs 32 cycles per 128 x NT x 16 product for
// NT <= 64 whatever NT.  NT = 32 or 64 instead of the dense product's 256
// because one field of a few hundred cells a side has only that many tiles:
// at 720 x 1440 the dense form ran 36 CTAs, 60 and 102 us per product; this
// one 14.3 and 20.8 (ncu), the solve 249 -> 64 us.
template <int NT> struct FoldCfg {
  static constexpr int B_T = NT * BK * 2;
  static constexpr int STAGE = 2 * A_TILE + 2 * B_T;
  static constexpr int STAGES = NT == 32 ? 5 : (NT == 64 ? 4 : 3);
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int GROUPS = NT == 32 ? 2 : 4;  // epilogue groups of four warps (one per TMEM lane quadrant)
  static constexpr int COLS = NT / GROUPS;         // columns per group
  static constexpr int THREADS = 64 + 128 * GROUPS;
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) |
                                    ((uint32_t)(BM >> 4) << 24);
  static_assert(COLS % 16 == 0, "16-column epilogue steps");
};

template <int NT>
__global__ void __launch_bounds__(FoldCfg<NT>::THREADS, 1)
gemm_fold_bf16_kernel(const __grid_constant__ CUtensorMap mAPh, const __grid_constant__ CUtensorMap mAPl,
                      const __grid_constant__ CUtensorMap mAQh, const __grid_constant__ CUtensorMap mAQl,
                      const __grid_constant__ CUtensorMap mPh, const __grid_constant__ CUtensorMap mPl,
                      const __grid_constant__ CUtensorMap mQh, const __grid_constant__ CUtensorMap mQl, int h,
                      const __grid_constant__ FoldEpi fe) {
  using C = FoldCfg<NT>;
  const Epi& ep = fe.e;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE);  // full[S], empty[S], acc
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * C::STAGES + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * NT;
  const int KT = 2 * ((h + BK - 1) / BK);  // P and Q blocks alternate
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[C::STAGES + s]); };
  const uint32_t accb = smem_u32(&bars[2 * C::STAGES]);

  if (threadIdx.x == 0) {
    prefetch_map(&mAPh); prefetch_map(&mAPl); prefetch_map(&mAQh); prefetch_map(&mAQl);
    prefetch_map(&mPh); prefetch_map(&mPl); prefetch_map(&mQh); prefetch_map(&mQl);
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    mbar_init(accb, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * NT));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // staggered start (an even shift keeps the P / Q alternation)
  const int kshift = 2 * (int)((blockIdx.x * 5u + blockIdx.y * 3u) % (unsigned)(KT / 2));
  if (warp == 0 && lane == 0) {
    auto load_b = [&](int kt0) {
      const int s = kt0 % C::STAGES;
      mbar_expect_tx(full(s), C::STAGE);
      const uint32_t base = smem_u32(smem + s * C::STAGE);
      const int kt = (kt0 + kshift) % KT, kb = (kt >> 1) * BK;
      tma_load_2d(base + 2 * A_TILE, (kt & 1) ? &mQh : &mPh, full(s), kb, n0);
      tma_load_2d(base + 2 * A_TILE + C::B_T, (kt & 1) ? &mQl : &mPl, full(s), kb, n0);
    };
    const int KTL = ep.stall ? 0 : KT;  // ep.stall: no loads (the timeout test)
    // tables of the first ring fill before waiting for the previous kernel
    for (int kt0 = 0; kt0 < KTL && kt0 < C::STAGES; ++kt0) load_b(kt0);
    grid_dep_wait();
    int issued = 0;
    for (int kt0 = 0; kt0 < KTL; ++kt0) {
      const int s = kt0 % C::STAGES;
      if (kt0 >= C::STAGES) {
        if (!mbar_wait(empty(s), ((kt0 / C::STAGES) - 1) & 1, abort_flag, ep.err, ep.wait_cycles)) break;
        load_b(kt0);
      }
      const uint32_t base = smem_u32(smem + s * C::STAGE);
      const int kt = (kt0 + kshift) % KT, kb = (kt >> 1) * BK;
      tma_load_2d(base, (kt & 1) ? &mAQh : &mAPh, full(s), kb, m0);
      tma_load_2d(base + A_TILE, (kt & 1) ? &mAQl : &mAPl, full(s), kb, m0);
      issued = kt0 + 1;
    }
    drain_ring(full(0), C::STAGES, issued);
  } else if (warp == 1 && lane == 0) {
    bool ok = true;
    for (int kt0 = 0; kt0 < KT && ok; ++kt0) {
      const int s = kt0 % C::STAGES;
      ok = mbar_wait(full(s), (kt0 / C::STAGES) & 1, abort_flag, ep.err, ep.wait_cycles);
      if (!ok) break;
      tc_fence_after();
      const uint32_t base = smem_u32(smem + s * C::STAGE);
      const uint64_t ah = sdesc_sw128(base), al = sdesc_sw128(base + A_TILE);
      const uint64_t bh = sdesc_sw128(base + 2 * A_TILE), bl = sdesc_sw128(base + 2 * A_TILE + C::B_T);
      const uint32_t d = tmem + (((kt0 + kshift) & 1) ? (uint32_t)NT : 0u);
      const bool first = kt0 < 2;  // the first P block and the first Q block overwrite
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) {
        const uint64_t o = (uint64_t)(kk * 32 >> 4);
        umma_bf16<COLL_FILL>(d, ah + o, bh + o, C::IDESC, !(first && kk == 0));
        umma_bf16<COLL_LASTUSE>(d, ah + o, bl + o, C::IDESC, 1u);
        umma_bf16(d, al + o, bh + o, C::IDESC, 1u);
      }
      umma_commit(empty(s));
    }
    umma_commit(accb);
  } else if (warp >= 2) {
    const int wq = warp & 3, grp = (warp - 2) >> 2;
    const int m = m0 + wq * 32 + lane;
    const bool mvalid = m < ep.m_total;
    const int R = ep.rows_per_batch;
    const int b = mvalid ? m / R : 0, r = mvalid ? m - b * R : 0;
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    const int rs = fe.half_out ? ((r & 1) ? fe.half_out : 0) + (r >> 1) : r;
    const bool pair = fe.mir < 0;
    const long long row0 = (long long)b * ep.batch_stride + rs, ld = ep.ld;
    const float alpha = (float)ep.alpha;
    const float* ie = ep.inv_eig ? ep.inv_eig + (long long)(b % ep.n_eig) * ep.n_cols * R + r : nullptr;
    float ivp[16], ivm[16];
    auto scales = [&](int nb) {  // 1/Lambda of the two outputs of table rows nb .. nb + 15
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int n = nb + j, np = pair ? 2 * n : n, nm = pair ? 2 * n + 1 : fe.mir - n;
        ivp[j] = n < fe.nh ? __ldg(ie + (long long)np * R) : 0.f;
        ivm[j] = n < fe.nh && nm < ep.n_cols ? __ldg(ie + (long long)nm * R) : 0.f;
      }
    };
    if (ie) scales(n0 + grp * C::COLS);  // while the main loop runs
    const bool ok = mbar_wait(accb, 0, abort_flag, ep.err, ep.wait_cycles);
    if (ok) tc_fence_after();
    grid_dep_launch();  // the next kernel may start its set-up while this tile drains
    if (ok && !*abort_flag) {
#pragma unroll 1
      for (int sc = 0; sc < C::COLS; sc += 16) {
        const int c0 = grp * C::COLS + sc, nb = n0 + c0;
        if (nb >= fe.nh) break;
        if (ie && sc) scales(nb);
        uint32_t vp[16], vq[16];
        __syncwarp();
        tmem_ld16(tmem + lanes + (uint32_t)c0, vp);
        tmem_ld16(tmem + lanes + (uint32_t)(NT + c0), vq);
        tmem_wait_ld();
        long long op = row0 + (long long)(pair ? 2 * nb : nb) * ld;
        long long om = row0 + (long long)(pair ? 2 * nb + 1 : fe.mir - nb) * ld;
        const long long sp = pair ? 2 * ld : ld, sm = pair ? 2 * ld : -ld;
        // number of valid table rows here, and of those with a second output
        // (MIRROR: mir - n beyond n and inside the array; periodic row 0 and
        // a middle row have none)
        const int nv = mvalid ? min(16, fe.nh - nb) : 0;
        const int lo = pair || fe.mir - nb < ep.n_cols ? 0 : 1;
        const int hi = pair ? nv : min(nv, (fe.mir + 1) / 2 - nb);
        if (ep.mode == EPI_SPLIT) {
          bf16 *o0 = (bf16*)ep.out0, *o1 = (bf16*)ep.out1;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float P = __uint_as_float(vp[j]), Q = __uint_as_float(vq[j]);
            float xp = pair ? P : P + Q, xm = pair ? Q : P - Q;
            if (ie) { xp *= ivp[j]; xm *= ivm[j]; }
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(xp, xm);
            const __nv_bfloat162 l2 = __floats2bfloat162_rn(xp - __low2float(h2), xm - __high2float(h2));
            if (j < nv) { o0[op] = h2.x; o1[op] = l2.x; }
            if (j >= lo && j < hi) { o0[om] = h2.y; o1[om] = l2.y; }
            op += sp;
            om += sm;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float P = __uint_as_float(vp[j]), Q = __uint_as_float(vq[j]);
            const float yp = pair ? P : P + Q, ym = pair ? Q : P - Q;
            const bool two = j >= lo && j < hi;
            if (ep.mode == EPI_F32) {
              float* o = (float*)ep.out0;
              if (j < nv) o[op] = yp * alpha;
              if (two) o[om] = ym * alpha;
            } else if (ep.mode == EPI_F32_ACC) {
              float* o = (float*)ep.out0;
              if (j < nv) o[op] += yp * alpha;
              if (two) o[om] += ym * alpha;
            } else {  // EPI_F64_ACC
              double* o = (double*)ep.out0;
              if (j < nv) o[op] += (double)yp * ep.alpha;
              if (two) o[om] += (double)ym * ep.alpha;
            }
            op += sp;
            om += sm;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (lane == 0) mbar_drain(accb, 0);  // the MMAs issued before an abort have completed
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * NT));
  }
}

// ---- operand producers ----------------------------------------------------
// FP32 / FP64 samples of a [batch][ny][nx] view folded along both axes (sums
// and differences with the mirrored sample, dst_f64.cuh) and split, rows of
// `pitch` elements with the differences along x from element `half` on; row
// 2a holds the sums along y, row 2a + 1 the differences.  HL: the view is a
// hi / lo pair of bf16 arrays instead (their sum is exact in FP32).
template <typename T, bool HL>
__global__ void fold_split_kernel(const T* in, const T* in_lo, long long bstride, long long ld, int ny, int nx, int hy,
                                  int hx, int miry, int mirx, int batch, int pitch, int half, bf16* hi, bf16* lo) {
  grid_dep_wait();
  const int rows = batch * hy;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const int b = row / hy, y = row - b * hy, y2 = miry - y;
    const bool py = y2 > y && y2 < ny;
    const long long s0 = b * bstride + (long long)y * ld, s1 = b * bstride + (long long)y2 * ld;
    const long long d0 = ((long long)b * hy + y) * 2 * pitch, d1 = d0 + pitch;
    auto at = [&](long long k) -> double {
      if constexpr (HL) {
        const __nv_bfloat16_raw h{__ldcg((const unsigned short*)in + k)}, l{__ldcg((const unsigned short*)in_lo + k)};
        return (double)(__bfloat162float(bf16(h)) + __bfloat162float(bf16(l)));
      } else {
        return (double)__ldcg(in + k);
      }
    };
    auto put = [&](long long k, double v) {
      const float f = (float)v;
      const bf16 h = __float2bfloat16_rn(f);
      hi[k] = h;
      lo[k] = __float2bfloat16_rn(f - __bfloat162float(h));
    };
    for (int x = threadIdx.x; x < hx; x += blockDim.x) {
      const int x2 = mirx - x;
      const bool px = x2 > x && x2 < nx;
      const double a0 = at(s0 + x), a1 = px ? at(s0 + x2) : 0.0;
      const double b0 = py ? at(s1 + x) : 0.0, b1 = py && px ? at(s1 + x2) : 0.0;
      const double as = px ? a0 + a1 : a0, ad = px ? a0 - a1 : 0.0;
      const double bs = px ? b0 + b1 : b0, bd = px ? b0 - b1 : 0.0;
      put(d0 + x, py ? as + bs : as);
      put(d0 + half + x, py ? ad + bd : ad);
      put(d1 + x, py ? as - bs : 0.0);
      put(d1 + half + x, py ? ad - bd : 0.0);
    }
  }
  grid_dep_launch();
}

// A natural-order hi / lo operand [rows][nx] de-interleaved into rows of
// `pitch` elements (odd columns from `half` on).
__global__ void deinterleave_kernel(const bf16* ih, const bf16* il, long long rows, int nx, int pitch, int half,
                                    bf16* hi, bf16* lo) {
  grid_dep_wait();
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    const unsigned int *h = (const unsigned int*)(ih + r * nx), *l = (const unsigned int*)(il + r * nx);
    unsigned short *oh = (unsigned short*)(hi + r * pitch), *ol = (unsigned short*)(lo + r * pitch);
    for (int p = threadIdx.x; p < nx / 2; p += blockDim.x) {
      const unsigned int a = __ldcg(h + p), c = __ldcg(l + p);
      oh[p] = (unsigned short)a; oh[half + p] = (unsigned short)(a >> 16);
      ol[p] = (unsigned short)c; ol[half + p] = (unsigned short)(c >> 16);
    }
  }
  grid_dep_launch();
}
