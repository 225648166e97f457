// Pieces shared by the tcgen05 beamformers (fnum_pw_tc.cu, fnum_sa_tc.cu): the block's shape,
// waits on mbarriers, aperture decisions, phasors and the split operand.
#pragma once
#include "fnum_device.cuh"
#include "fnum_internal.h"
#include "fnum_tc_ptx.cuh"

namespace fnum {
namespace tcx {

constexpr int P5_CW = 16;                         // compute warps: 4 element slots x 4 lane quadrants
constexpr int P5_CT = P5_CW * 32;
constexpr int P5_THREADS = P5_CT + 128;           // + a warpgroup that issues products and copies
constexpr int P5_M = TILE_X * TILE_Z;             // voxels per tile = TMEM lanes = mma M
// registers per thread after the launch's 96 (61440 / 640 threads) are shared out anew:
// 512 x 104 + 128 x 64 = 61440
constexpr int P5_REGS = 96, P5_REGS_C = 104, P5_REGS_I = 64;
static_assert(P5_CT * P5_REGS_C + 128 * P5_REGS_I <= P5_REGS * P5_THREADS, "register split");
static_assert(P5_M == 128, "a voxel per TMEM lane");

// A test of an mbarrier's phase takes about 160 cycles to answer, so it is asked ahead of the
// work before the wait (p5_ask) and the answer handed to the wait.
__device__ __forceinline__ uint32_t p5_ask(uint32_t bar, uint32_t parity) { return mbar_test(bar, parity) ? 1u : 0u; }

// Waits for the phase of parity `parity`.  It gives up after WAIT_NS of the global timer (read every
// P5_TESTS failed tests: a test may suspend the thread for a time of the hardware's choice, so a
// count alone is no bound), records the timeout and tells the others, whose failing waits then end
// at once; the work after it runs on stale data and ends.  The entry points that wait for the
// device (the host-buffer calls, the gradients, fnum_plan_info_get) report the recorded timeout.
constexpr unsigned P5_TESTS = 64;
static_assert(WAIT_NS < (1ull << 32), "the lower half of the timer measures it");
__device__ __forceinline__ bool p5_wait(uint32_t bar, uint32_t parity, uint32_t answer, volatile int* abort_flag,
                                        unsigned long long* err) {
  if (answer) return true;
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p, q;\n.reg .u32 f, n, t0;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n@p bra P5_DONE;\n"
      "mov.u32 t0, %globaltimer_lo;\n"
      "P5_MORE:\nmov.u32 n, %3;\n"
      "P5_AGAIN:\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n@p bra P5_DONE;\n"
      "ld.volatile.shared.u32 f, [%4];\nsetp.ne.u32 q, f, 0;\n@q bra P5_DONE;\n"
      "sub.u32 n, n, 1;\nsetp.ne.u32 q, n, 0;\n@q bra P5_AGAIN;\n"
      "mov.u32 f, %globaltimer_lo;\nsub.u32 f, f, t0;\nsetp.lt.u32 q, f, %5;\n@q bra P5_MORE;\n"
      "P5_DONE:\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "n"(P5_TESTS), "r"(smem_u32((const void*)abort_flag)), "n"((unsigned)WAIT_NS)
      : "memory");
  if (ok) return true;
  *abort_flag = 1;
  atomicOr(err, ERR_TC_TIMEOUT);
  return false;
}

__device__ __forceinline__ void p5_bar() { asm volatile("bar.sync 1, %0;" ::"n"(P5_CT) : "memory"); }

// a value known to be the same in all lanes, as a uniform register
__device__ __forceinline__ uint32_t p5_uni(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }

// aperture() with its decisions taken in FP32 where they cannot differ: the rounding of
// xp -+ zp g is below 3 2^-24 (|xp| + |zp g|), so a bound at least 2^-21 (..) away from an
// integer rounds the same way; the others take the double-float path
__device__ __forceinline__ void p5_aperture(dfl xp, dfl zp, dfl g, int ne, int& ilb, int& iub) {
  const float w = zp.x * g.x;
  const float tl = xp.x - w, tr = xp.x + w;
  const float cl = ceilf(tl), fr = floorf(tr);
  const float a = cl - tl, b = tr - fr;
  const float eps = 4.76837158e-7f * (fabsf(xp.x) + fabsf(w));     // 2^-21
  if (g.x > 0.0f && fminf(a, b) > eps && fmaxf(a, b) < 1.0f - eps) {
    ilb = (int)fminf(fmaxf(cl, 0.0f), (float)ne);
    iub = (int)fminf(fmaxf(fr, -1.0f), (float)(ne - 1));
    return;
  }
  aperture(xp, zp, g, ne, ilb, iub);
}

// A column's part of the window table: tab[row wt_w + e] and sum[row] by the numbers of the outermost
// element (the row) and of the element, and the row of zeros.
struct P5Window {
  const float* tab;
  const float* sum;
  int zero;
};
__device__ __forceinline__ P5Window p5_window(const PWDev& d, int cc, int e0) {
  const int rows = d.wt_rows + 1;
  return {d.w_tab + ((ptrdiff_t)cc * rows * d.wt_w - (ptrdiff_t)e0 * (d.wt_w + 1)), d.w_sum + ((ptrdiff_t)cc * rows - e0),
          e0 + d.wt_rows};
}

// Spectrum entries that are NaN or infinite stay out of the operands, where a weight of 0 (an
// element of the same group outside the aperture) would turn them into NaN.  They are added to
// the voxels whose aperture holds their element with a weight, whose values are then not finite
// either: out[a stride] gains those of bins kt .. kt - nb + 1 and angles a = a0, a0 + step, ..  Rare,
// so a plain loop does, in a function of its own: inlined it takes registers of the kernels'
// loops (11 angles, 128 elements, 512 x 512: 15.96 ms, inlined 16.03).
__device__ __forceinline__ bool p5_finite(float2 x) { return isfinite(x.x) && isfinite(x.y); }
[[maybe_unused]] static __device__ __noinline__ void p5_nonfinite(const PWDev& d, float2* out, size_t stride, int cc,
                                                                  int jc, int kt, int nb, int a0, int step) {
  const int ne = d.ne, ic = d.wt_c0 + cc, emid = d.col_emid[ic];
  const P5Window t = p5_window(d, cc, d.col_e0[ic]);
  for (int b = 0; b < nb; ++b) {
    const int kk = kt - b - d.k_lb;
    int ilb, iub;
    p5_aperture(d.col_p[ic], d.row_p[jc], d.g[kk], ne, ilb, iub);
    const int row_l = ilb < emid ? ilb : t.zero, row_r = iub >= emid ? iub : t.zero;
    if (!(t.sum[row_l] + t.sum[row_r] > 0.0f)) continue;
    for (int e = min(ilb, emid); e <= max(iub, emid - 1); ++e) {
      const float w = t.tab[(size_t)(e < emid ? row_l : row_r) * d.wt_w + e];
      if (!(w > 0.0f)) continue;
      for (int a = a0; a < d.na; a += step) {
        const float2 x = d.X[((size_t)e * d.K + kk) * d.x_na + d.x_a0 + a];
        if (p5_finite(x)) continue;
        const float v = w * (x.x + x.y);
        float2& o = out[(size_t)a * stride];
        o = make_float2(o.x + v, o.y + v);
      }
    }
  }
}

__device__ __forceinline__ unsigned p5_join(const unsigned (&r)[4]) {
  const uint4 v = *reinterpret_cast<const uint4*>(r);
  return __vminu2(__vminu2(v.x, v.y), __vminu2(v.z, v.w));
}

__device__ __forceinline__ float2 p5_dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 p5_neg(float2 v) { return make_float2(-v.x, -v.y); }

// e^{2 pi i k u} of two double-float delays u = {h, l}: k u reduced exactly to [-1/2, 1/2]
// cycles, then to an eighth of a cycle around the nearest quarter, with the polynomials of
// sin(2 pi f) and cos(2 pi f) on |f| <= 1/8 (least maximum error fits in f^2: 2.4e-9 and
// 5e-11 before rounding, 8.4e-8 and 5.8e-8 evaluated in FP32).  Packed FP32x2, about a third
// of cis_ku's instructions.
__device__ __forceinline__ void p5_cis2(float kf, float2 h, float2 l, float2& re, float2& im) {
  const float2 k2 = p5_dup(kf), nk2 = p5_dup(-kf);
  const float2 p = __fmul2_rn(k2, h);
  const float2 e = __ffma2_rn(nk2, h, p);             // -(k h - p), exact
  const float2 rl = __ffma2_rn(nk2, l, e);            // -(trailing part of k u)
  const float2 n = make_float2(rintf(p.x), rintf(p.y));
  const float2 m1 = p5_dup(-1.0f);
  const float2 rh = __ffma2_rn(n, m1, p);             // exact
  const float2 magic = p5_dup(12582912.0f);           // 1.5 2^23: rounds to an integer in the low bits
  const float2 t = __ffma2_rn(rh, p5_dup(4.0f), magic);
  const float2 qf = __ffma2_rn(magic, m1, t);
  const float2 f = __ffma2_rn(rl, m1, __ffma2_rn(qf, p5_dup(-0.25f), rh));
  const float2 s = __fmul2_rn(f, f);
  float2 S = __ffma2_rn(p5_dup(-75.4000015f), s, p5_dup(81.592514f));
  S = __ffma2_rn(S, s, p5_dup(-41.3416634f));
  S = __ffma2_rn(S, s, p5_dup(6.28318548f));
  S = __fmul2_rn(S, f);
  float2 Cc = __ffma2_rn(p5_dup(59.218758f), s, p5_dup(-85.44281f));
  Cc = __ffma2_rn(Cc, s, p5_dup(64.939316f));
  Cc = __ffma2_rn(Cc, s, p5_dup(-19.739208f));
  Cc = __ffma2_rn(Cc, s, p5_dup(1.0f));
  const unsigned q0 = __float_as_uint(t.x), q1 = __float_as_uint(t.y);
  const float c0 = (q0 & 1u) ? S.x : Cc.x, s0 = (q0 & 1u) ? Cc.x : S.x;
  const float c1 = (q1 & 1u) ? S.y : Cc.y, s1 = (q1 & 1u) ? Cc.y : S.y;
  re = make_float2(__uint_as_float(__float_as_uint(c0) ^ (((q0 + 1u) & 2u) << 30)),
                   __uint_as_float(__float_as_uint(c1) ^ (((q1 + 1u) & 2u) << 30)));
  im = make_float2(__uint_as_float(__float_as_uint(s0) ^ ((q0 & 2u) << 30)),
                   __uint_as_float(__float_as_uint(s1) ^ ((q1 & 2u) << 30)));
}

template <int C>
__device__ __forceinline__ void p5_ld_cols(uint32_t t, float (&v)[C]) {
  if constexpr (C == 4) {
    tmem_ld4_nowait(t, v);
  } else {
#pragma unroll
    for (int i = 0; i + 8 <= C; i += 8) tmem_ld8_nowait(t + i, *reinterpret_cast<float(*)[8]>(&v[i]));
    if constexpr (C % 8 == 4) tmem_ld4_nowait(t + (C / 8) * 8, *reinterpret_cast<float(*)[4]>(&v[(C / 8) * 8]));
  }
}

// p <- p conj(rho) of 8 elements, two per packed FP32 instruction; pv holds {Re, Re, Im, Im}
// per element pair, rv the steps
__device__ __forceinline__ void p5_rotate(float (&pv)[16], const float (&rv)[16]) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 rr = make_float2(rv[4 * p], rv[4 * p + 1]), ri = make_float2(rv[4 * p + 2], rv[4 * p + 3]);
    const float2 a = make_float2(pv[4 * p], pv[4 * p + 1]), m = make_float2(pv[4 * p + 2], pv[4 * p + 3]);
    const float2 x = __ffma2_rn(m, ri, __fmul2_rn(a, rr));
    const float2 y = __ffma2_rn(m, rr, p5_neg(__fmul2_rn(a, ri)));
    pv[4 * p] = x.x;
    pv[4 * p + 1] = x.y;
    pv[4 * p + 2] = y.x;
    pv[4 * p + 3] = y.y;
  }
}
// the A values w p of 8 elements as fp16 hi and lo, {Re, Im} per element
__device__ __forceinline__ void p5_operand(const float4 w0, const float4 w1, const float (&pv)[16], uint32_t (&hq)[8],
                                           uint32_t (&lq)[8]) {
  const float2 wp[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y),
                        make_float2(w1.z, w1.w)};
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 br = __fmul2_rn(wp[p], make_float2(pv[4 * p], pv[4 * p + 1]));
    const float2 bi = __fmul2_rn(wp[p], make_float2(pv[4 * p + 2], pv[4 * p + 3]));
    tc_split_mx(br.x, bi.x, hq[2 * p], lq[2 * p]);
    tc_split_mx(br.y, bi.y, hq[2 * p + 1], lq[2 * p + 1]);
  }
}

}  // namespace tcx
}  // namespace fnum
