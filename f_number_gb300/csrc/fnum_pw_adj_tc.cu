// The adjoint of the compounded plane-wave beamformer on the Blackwell tensor cores (tcgen05).
//
// Per band bin k, with R_k(v, e) = w_k(v, e) e^{2 pi i k u_e(v)} as in fnum_pw_tc.cu,
//     gX_k(e, a) = s sum_v conj(R_k(v, e)) Q_k(v, a),   Q_k(v, a) = n_k(v) G_v conj(t_{v,a}^k):
// the forward product transposed and reduced over the voxels, a GEMM with a row per element,
// D[e][n] = sum_{v,q} A[e][2v + q] B[n][2v + q], A = (Re R, Im R), B the real form of Q.  Both
// operands are split into fp16 hi + lo (Q scaled by a power of two) and hi.lo + lo.hi + hi.hi
// accumulate in FP32 in tensor memory.  No counterpart in the reference.
//
// An item is a chunk of bins (their D's take up to 384 columns: 24 bins of 8 angles, 12 of 16, 8 of 24), a
// slice of AJ_SLICE voxels, 128 elements and a pass of angles; the chunks of a slice run side by side,
// so the receive table's rows come from L2.  16 warps form A: warp w serves lane quadrant w % 4
// (an element per thread) and slot w / 4, which takes every fourth group of 8 voxels.  Per group
// the slot's threads form the aperture rows and n_k of its voxels and bins and the B tiles of the
// chunk (shared memory, double-buffered); then, bin by bin, the receive phasors of the 8 voxels
// (registers, stepped by conj(rho) from an exact anchor at the first bin whose apertures touch the
// quadrant) times the window values are split into fp16 and stored to one of the slot's two A
// tiles in tensor memory.  Quadrants outside a bin's apertures store zeros.  Four threads issue
// the products, each those of every fourth bin (a D belongs to one thread).  At the end of the
// slice D is added to FP64 sums.
//
// The tensor cores' FP32 accumulation rounds toward zero, three times a group: 3.5e-5 of the
// gradient (rel-L2) with slices of 8192 voxels, as in the mma.sync kernel before this one (4e-5); with
// 1024 it would be 8e-6.
//
// What bounds it: the compute warps' instructions, about 110 a unit (8 voxels x 32 elements x a
// bin) and 600 a group for its set-up.  256 x 256 voxels, 128 elements, 11 angles: 12.9 ms with
// warp-level mma.sync (6 bins a chunk, window evaluated per term), 8.4 ms here; 150 x 203 voxels,
// 96 elements, 5 angles: 5.2 and 2.4 ms (an 8-angle pass costs half the products of a 12-angle
// one, and its chunks are twice as long).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "fnum_tc_beam.cuh"

namespace fnum {

namespace {

using namespace tcx;

constexpr int AJ_SLICE = 8192;      // voxels of an item
constexpr int AJ_DCOLS = 384;       // TMEM columns of the chunk's D's; then the A tiles
constexpr int AJ_BB = 24576;        // B bytes of a group: 64 N per bin
constexpr int AJ_BMAX = 24;         // bins of a chunk at most
static_assert(AJ_SLICE % 32 == 0, "a round is a group of 8 voxels per slot");

struct AjShared {
  // per slot and buffer: window-table offsets of the left and right row, n_k and the element range by
  // bin (lo | hi << 16; lo > hi: none)
  uint2 off[4][2][AJ_BMAX][8];
  float nk[4][2][AJ_BMAX][8];
  unsigned rng[4][2][AJ_BMAX];
  int abort_flag;
  uint32_t tmem;
  uint64_t bars[4 * 8 + 4 * 2 + 4 * 2 + 4 * 2 + 1];
};
constexpr int aj_smem() { return ((int)sizeof(AjShared) + 127) / 128 * 128 + 4 * 2 * AJ_BB; }

// fp16 scale of Q: the power of two that brings max|G| max(n_k), a bound of |Q|, below 2^14
// (gmax: float bits of max |G component| and of max n_k)
__device__ __forceinline__ float aj_scale(const unsigned* gmax) {
  const float m = __uint_as_float(gmax[0]) * __uint_as_float(gmax[1]);
  if (!(m > 0.0f) || !(m < 3.0e38f)) return 1.0f;
  int ex;
  frexpf(m, &ex);
  return ldexpf(1.0f, min(max(14 - ex, -126), 126));
}

__device__ __forceinline__ dfl aj_urx(const PWDev& d, int e, int i, int j) {
  return df_sqrt(df_add(df_sqr(df_sub(d.el_u[e], d.col_u[i])), d.row_u2[j]));
}

// the receive table: u in double-float and the step e^{2 pi i u} of every (voxel, element) pair
__global__ void __launch_bounds__(256) aj_table_kernel(const PWDev d) {
  const size_t n = (size_t)d.nx * d.nz * d.ne;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const size_t v = idx / d.ne;
    const int e = (int)(idx - v * d.ne);
    const int i = (int)(v / d.nz), j = (int)(v - (size_t)i * d.nz);
    const dfl u = aj_urx(d, e, i, j);
    float2 re, im;
    p5_cis2(1.0f, make_float2(u.x, u.x), make_float2(u.y, u.y), re, im);
    d.rx_tab[idx] = make_float4(u.x, u.y, re.x, im.x);
  }
}

// whether the window table's elements of the columns of voxels v0 .. v1 - 1 reach elements e .. e + 127
__device__ __forceinline__ bool aj_touched(const PWDev& d, long long v0, long long v1, int e) {
  int lo = 0x7fffffff, hi = -1;
  for (int i = ((int)(v0 / d.nz) & ~(TILE_X - 1)) + TILE_X * (int)(threadIdx.x & 31); i <= (int)((v1 - 1) / d.nz);
       i += TILE_X * 32) {
    lo = min(lo, d.col_e0[i]);
    hi = max(hi, d.col_e0[i]);
  }
  return __reduce_min_sync(0xffffffffu, lo) < e + 128 && __reduce_max_sync(0xffffffffu, hi) + d.wt_w > e;
}

// N: D columns of a bin, two per angle.  [v_begin, v_end): the voxels of the window table's columns.  NB: bins of a
// chunk (at most AJ_DCOLS / N).  BAND: the window table holds only the elements that the apertures reach;
// items without any of them are passed over.
template <int N, bool BAND>
__global__ void __launch_bounds__(P5_THREADS, 1)
aj_tc_kernel(const PWDev d, const float2* __restrict__ cot, const unsigned* __restrict__ gmax, double* __restrict__ acc,
             long long v_begin, long long v_end, int NB) {
  constexpr int NA = N / 2;                 // angles of a pass
  static_assert(AJ_DCOLS / N <= AJ_BMAX && AJ_DCOLS * 64 == AJ_BB, "chunk");
  extern __shared__ __align__(128) unsigned char dyn[];
  AjShared& sh = *reinterpret_cast<AjShared*>(dyn);
  unsigned char* bbuf = dyn + (sizeof(AjShared) + 127) / 128 * 128;
  const uint32_t bbase = smem_u32(bbuf);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = (int)p5_uni((uint32_t)tid >> 5);
  volatile int* abort_flag = &sh.abort_flag;
  unsigned long long* err = &d.counters[2];
  const uint32_t bar0 = smem_u32(sh.bars);
  // A tile written: a barrier per issuing thread (b % 4) and round parity, so that its next phase
  // cannot complete before that thread has seen this one
  auto s_full = [&](uint32_t s, uint32_t b, uint32_t r) { return bar0 + 8u * (8u * s + 2u * b + r); };
  auto s_empty = [&](uint32_t s, uint32_t b) { return bar0 + 8u * (32u + 2u * s + b); };
  auto b_full = [&](uint32_t s, uint32_t b) { return bar0 + 8u * (40u + 2u * s + b); };
  auto b_empty = [&](uint32_t s, uint32_t b) { return bar0 + 8u * (48u + 2u * s + b); };
  const uint32_t d_full = bar0 + 8u * 56u;
  if (tid == 0) {
    for (int s = 0; s < 4; ++s) {
      for (int b = 0; b < 8; ++b) mbar_init(s_full(s, b >> 1, b & 1), 4);
      for (int b = 0; b < 2; ++b) {
        mbar_init(s_empty(s, b), 1);
        mbar_init(b_full(s, b), 4);
        mbar_init(b_empty(s, b), 4);
      }
    }
    mbar_init(d_full, 4);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = p5_uni(sh.tmem);
  const int n_chunk = (d.K + NB - 1) / NB, n_ap = (d.na + NA - 1) / NA, n_ep = (d.ne + 127) / 128;
  const int n_slice = (int)((v_end - v_begin + AJ_SLICE - 1) / AJ_SLICE);
  const int n_items = n_chunk * n_ap * n_ep * n_slice;
  uint32_t un = 0;                  // units (a group and a bin) of a slot so far
  uint32_t rd = 0;                  // rounds (groups of a slot) so far
  uint32_t it = 0;                  // items so far
  // The block's items: every gridDim.x-th, with BAND of those that an aperture reaches (seen: such items
  // of the slices and elements before `pair`), so that these are spread evenly over the blocks.
  const int n_in = n_chunk * n_ap;
  int next = blockIdx.x, seen = 0, pair = 0;
  auto fetch = [&]() {
    if constexpr (BAND) {
      for (; pair < n_slice * n_ep; ++pair) {
        const long long v0 = v_begin + (long long)(pair / n_ep) * AJ_SLICE;
        if (!aj_touched(d, v0, min(v_end, v0 + AJ_SLICE), pair % n_ep * 128)) continue;
        if (next < seen + n_in) return pair * n_in + next - seen;
        seen += n_in;
      }
      return n_items;
    } else {
      return next;
    }
  };

  if (warp >= P5_CW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P5_REGS_I));
    const uint32_t me = (uint32_t)(warp - P5_CW);       // issues the bins b % 4 = me of a chunk
    uint32_t ph2 = 0;                                   // phases of its s_full barriers (bit per round parity)
    for (int item; (item = fetch()) < n_items; next += gridDim.x) {
      const int chunk = item % n_chunk;
      const int slice = item / (n_chunk * n_ap * n_ep);
      const int nb = min(NB, d.K - chunk * NB);
      const long long v0 = v_begin + (long long)slice * AJ_SLICE;
      const int rounds = (int)((min((long long)AJ_SLICE, v_end - v0) + 31) / 32);
      if (lane == 0) {
        constexpr uint64_t HI = smem_desc_plain_hi(256);
        constexpr uint32_t idesc = idesc_f16(P5_M, N);
        for (int r = 0; r < rounds && !*abort_flag; ++r, un += (uint32_t)nb, ++rd) {
          for (uint32_t s = 0; s < 4u; ++s) p5_wait(b_full(s, rd & 1u), (rd >> 1) & 1u, 0u, abort_flag, err);
          for (uint32_t b = me; b < (uint32_t)nb; b += 4u, ph2 ^= 1u << (rd & 1u)) {
            const uint32_t bf = (un + b) & 1u, rp = rd & 1u, ph = (ph2 >> rp) & 1u;
            uint32_t ask = p5_ask(s_full(0, me, rp), ph);
#pragma unroll 1
            for (uint32_t s = 0; s < 4u; ++s) {
              p5_wait(s_full(s, me, rp), ph, ask, abort_flag, err);
              if (s < 3u) ask = p5_ask(s_full(s + 1u, me, rp), ph);
              const uint32_t a = tmem + AJ_DCOLS + 32u * s + 16u * bf, dcol = tmem + b * N;
              const uint32_t bd =
                  (uint32_t)smem_desc_plain(bbase + (2u * s + (rd & 1u)) * AJ_BB + b * (64u * N), 128, 256);
              fence_after_sync();
              // the small cross products first, so that fewer steps round a full-size sum
              mma_f16_ts(dcol, a, HI | (uint64_t)(bd + 2u * N), idesc, (r | (int)s) ? 1u : 0u);
              mma_f16_ts(dcol, a + 8u, HI | (uint64_t)bd, idesc, 1u);
              mma_f16_ts(dcol, a, HI | (uint64_t)bd, idesc, 1u);
              mma_commit(s_empty(s, bf));
            }
          }
          for (uint32_t s = 0; s < 4u; ++s) mma_commit(b_empty(s, rd & 1u));
        }
        mma_commit(d_full);
      }
      __syncwarp();
      __syncthreads();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P5_REGS_C));
    const int q = warp & 3, slot = warp >> 2;
    const int ts = 32 * q + lane;                       // thread of the slot
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    const uint32_t lead = lane == 0 ? 1u : 0u;
    const float sigma = aj_scale(gmax);
    const int ne = d.ne;
    auto slot_bar = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory"); };
    for (int item; (item = fetch()) < n_items; next += gridDim.x) {
      const int chunk = item % n_chunk;
      int rest = item / n_chunk;
      const int a0 = (rest % n_ap) * NA;
      rest /= n_ap;
      const int e_lo = (rest % n_ep) * 128 + 32 * q, e = e_lo + lane;
      const int slice = rest / n_ep;
      const int ec = min(e, ne - 1);
      const int kt = d.k_ub - chunk * NB;               // the chunk's bins: kt down
      const int nb = min(NB, d.K - chunk * NB);
      const long long v0 = v_begin + (long long)slice * AJ_SLICE;
      const long long v1 = min(v_end, v0 + AJ_SLICE);
      const int rounds = (int)((v1 - v0 + 31) / 32);
#pragma unroll 1
      for (int r = 0; r < rounds; ++r, ++rd, un += (uint32_t)nb) {
        const long long vg = v0 + 32ll * r + 8 * slot;  // the group's voxels vg .. vg + 7
        const int i0 = (int)(min(vg, v1 - 1) / d.nz), j0 = (int)(min(vg, v1 - 1) - (long long)i0 * d.nz);
        const int n_v = (int)max(min(8ll, v1 - vg), 1ll);   // the voxels beyond the slice repeat its last
        auto voxel = [&](int x, int& i, int& j) {
          i = i0;
          for (j = j0 + min(x, n_v - 1); j >= d.nz; j -= d.nz) ++i;
        };
        const uint32_t buf = rd & 1u;
        const uint32_t ask_b = p5_ask(b_empty((uint32_t)slot, buf), ((rd >> 1) & 1u) ^ 1u);
        // rows, n_k and ranges of the (bin, voxel) pairs
        for (int idx = ts; idx < ((nb * 8 + 31) & ~31); idx += 128) {
          const int b = idx >> 3, vv = idx & 7;
          const bool ok = b < nb && vg + vv < v1;
          int i, j;
          voxel(vv, i, j);
          const int kk = max(kt - b - d.k_lb, 0), cc = i - d.wt_c0, emid = d.col_emid[i];
          const int e0 = BAND ? d.col_e0[i] : 0, zero = e0 + d.wt_rows;
          int ilb, iub;
          p5_aperture(d.col_p[i], d.row_p[j], d.g[kk], ne, ilb, iub);
          // a side without elements takes the zero row
          const int row_l = ilb < emid ? ilb : zero, row_r = iub >= emid ? iub : zero;
          const float* sc = d.w_sum + ((ptrdiff_t)cc * (d.wt_rows + 1) - e0);
          const float W = __ldg(sc + row_l) + __ldg(sc + row_r);
          const int lo = min(ilb, emid), hi = max(iub, emid - 1);
          const bool act = ok && W > 0.0f && lo <= hi;
          int mn = act ? lo : 0x7fff, mx = act ? hi : -1;
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) {
            mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          }
          if (b < nb) {
            // modulo 2^32: the element's number is added
            const unsigned base = (unsigned)(cc * (d.wt_rows + 1) - e0), w = (unsigned)d.wt_w;
            sh.off[slot][buf][b][vv] =
                make_uint2((base + (unsigned)row_l) * w - (unsigned)e0, (base + (unsigned)row_r) * w - (unsigned)e0);
            sh.nk[slot][buf][b][vv] = act ? (d.norm ? __frcp_rn(W) : 1.0f) : 0.0f;
            if (vv == 0) sh.rng[slot][buf][b] = (unsigned)mn | ((unsigned)(mx + 1) << 16);   // hi + 1: 0 for none
          }
        }
        // the group's receive delays and steps, on which side of the voxel the element lies and, with BAND,
        // whether the table holds it for the voxel's column: a group within one tile has all elements
        // of a quadrant that an aperture touches
        float2 uh[4], ul[4];
        float rv[16];
        unsigned left = 0u, held = 0u;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          int i, j;
          voxel(x, i, j);
          if (e < d.col_emid[i]) left |= 1u << x;
          if (BAND && (unsigned)(ec - d.col_e0[i]) < (unsigned)d.wt_w) held |= 1u << x;
          float4 t;
          if (d.rx_tab) {
            t = d.rx_tab[((size_t)i * d.nz + j) * ne + ec];
          } else {
            const dfl u = aj_urx(d, ec, i, j);
            float2 re, im;
            p5_cis2(1.0f, make_float2(u.x, u.x), make_float2(u.y, u.y), re, im);
            t = make_float4(u.x, u.y, re.x, im.x);
          }
          reinterpret_cast<float*>(&uh[x >> 1])[x & 1] = t.x;
          reinterpret_cast<float*>(&ul[x >> 1])[x & 1] = t.y;
          rv[4 * (x >> 1) + (x & 1)] = t.z;
          rv[4 * (x >> 1) + 2 + (x & 1)] = t.w;
        }
        const bool whole = !BAND || __all_sync(0xffffffffu, held == 0xffu);
        slot_bar();     // rows and n_k of all the group's pairs
        // B: thread (voxel, angle) and, with 8 angles, half of the bins; the angles beyond 16 in a second turn
        p5_wait(b_empty((uint32_t)slot, buf), ((rd >> 1) & 1u) ^ 1u, ask_b, abort_flag, err);
#pragma unroll 1
        for (int al = (ts >> 3) & (NA == 8 ? 7 : 15); al < NA; al += 16) {
          const int vv = ts & 7, half = (NB + 1) / 2, b_lo = NA == 8 ? (ts >> 6) * half : 0;
          const int b_hi = min(nb, NA == 8 ? b_lo + half : NB), a = a0 + al;
          const bool ok = vg + vv < v1 && a < d.na;
          const int ac = min(a, d.na - 1);
          int i, j;
          voxel(vv, i, j);
          const dfl u = df_add(d.tx_ax[(size_t)ac * d.nx + i], d.tx_az[(size_t)ac * d.nz + j]);
          float2 re, im, tr, ti;
          // conj(t^k) G sigma at the first bin; going down, conj(t^(k-1)) = conj(t^k) t
          p5_cis2((float)(kt - b_lo), make_float2(u.x, u.x), make_float2(u.y, u.y), re, im);
          p5_cis2(1.0f, make_float2(u.x, u.x), make_float2(u.y, u.y), tr, ti);
          const float2 g = ok ? cot[(size_t)i * d.nz + j] : make_float2(0.0f, 0.0f);
          float br = sigma * (g.x * re.x + g.y * im.x), bi = sigma * (g.y * re.x - g.x * im.x);
          const int n = 2 * al;
          unsigned char* o = bbuf + (2 * slot + (int)buf) * AJ_BB + b_lo * (64 * N) + (n >> 3) * 256 + (vv >> 2) * 128 +
                             (n & 7) * 16 + (vv & 3) * 4;
#pragma unroll 1
          for (int b = b_lo; b < b_hi; ++b, o += 64 * N) {
            const float w = sh.nk[slot][buf][b][vv];
            const float qr = w * br, qi = w * bi;
            unsigned h0, l0, h1, l1;
            tc_split_mx(qr, qi, h0, l0);        // row Re: Re R Qr + Im R Qi
            tc_split_mx(qi, -qr, h1, l1);       // row Im: Re R Qi - Im R Qr
            *reinterpret_cast<unsigned*>(o) = h0;
            *reinterpret_cast<unsigned*>(o + 16) = h1;
            *reinterpret_cast<unsigned*>(o + 32 * N) = l0;
            *reinterpret_cast<unsigned*>(o + 32 * N + 16) = l1;
            const float t = br * tr.x - bi * ti.x;
            bi = br * ti.x + bi * tr.x;
            br = t;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        mbar_arrive_if(lead, b_full((uint32_t)slot, buf));
        // A, bin by bin
        bool live = false;        // p holds the phasors of the previous bin
        float p[16];
#pragma unroll 1
        for (int b = 0; b < nb; ++b) {
          const uint32_t u = un + (uint32_t)b, bf = u & 1u, ph = ((u >> 1) & 1u) ^ 1u;
          const uint32_t ask = p5_ask(s_empty((uint32_t)slot, bf), ph);
          const unsigned rg = sh.rng[slot][buf][b];
          const int lo = (int)(rg & 0xffffu), hi = (int)(rg >> 16) - 1;
          uint32_t h[8], l[8];
          if (lo < e_lo + 32 && hi >= e_lo) {
            float w[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
              const uint2 of = sh.off[slot][buf][b][x];
              const unsigned o = ((left >> x) & 1u ? of.x : of.y) + (unsigned)ec;
              w[x] = __ldg(d.w_tab + (whole || (held >> x) & 1u ? o : 0u));
            }
            if (live) {
              p5_rotate(p, rv);
            } else {
              live = true;
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                float2 re, im;
                p5_cis2((float)(kt - b), uh[x], ul[x], re, im);
                p[4 * x] = re.x;
                p[4 * x + 1] = re.y;
                p[4 * x + 2] = im.x;
                p[4 * x + 3] = im.y;
              }
            }
            if (BAND && !whole) {
#pragma unroll
              for (int x = 0; x < 8; ++x)
                if (!((held >> x) & 1u)) w[x] = 0.0f;
            }
            p5_operand(make_float4(w[0], w[1], w[2], w[3]), make_float4(w[4], w[5], w[6], w[7]), p, h, l);
          } else {
            live = false;
#pragma unroll
            for (int x = 0; x < 8; ++x) h[x] = l[x] = 0u;
          }
          // the A tile is free once the products that read it last are complete
          p5_wait(s_empty((uint32_t)slot, bf), ph, ask, abort_flag, err);
          fence_after_sync();
          const uint32_t ta = tl + AJ_DCOLS + 32u * (uint32_t)slot + 16u * bf;
          tmem_st8(ta, h);
          tmem_st8(ta + 8u, l);
          tmem_wait_st();
          fence_before_sync();
          __syncwarp();
          mbar_arrive_if(lead, s_full((uint32_t)slot, (uint32_t)b & 3u, buf));
        }
      }
      // the chunk's D's into the FP64 sums: this warp's lanes of the bins b % 4 = slot
      p5_wait(d_full, it & 1u, 0u, abort_flag, err);
      fence_after_sync();
#pragma unroll 1
      for (int b = slot; b < nb; b += 4) {
        const int kk = kt - b - d.k_lb;
#pragma unroll 1
        for (int c = 0; c < N; c += 8) {
          float y[8];
          tmem_ld8_nowait(tl + (uint32_t)(b * N + c), y);
          tmem_wait_ld();
          if (e < ne && !*abort_flag) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int a = a0 + (c >> 1) + x;
              if (a < d.na) {
                double* o = acc + 2 * (((size_t)e * d.K + kk) * d.na + a);
                atomicAdd(o, (double)y[2 * x]);
                atomicAdd(o + 1, (double)y[2 * x + 1]);
              }
            }
          }
          __syncwarp();
        }
      }
      fence_before_sync();
      __syncthreads();
      ++it;
    }
  }
  // after a timeout, give the products in flight time to land before the tensor memory is freed
  if (tid == 0 && *abort_flag) {
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 20000000ull) {
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// FP64 sums {Re, Im} per (element, bin, angle) -> dL/dX* (scaled by 2 / N, the fp16 scale undone)
__global__ void __launch_bounds__(256) aj_finish_kernel(const double* __restrict__ acc, size_t n, double scale,
                                                        const unsigned* __restrict__ gmax, float2* __restrict__ gX) {
  const double sc = scale / (double)aj_scale(gmax);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    gX[i] = make_float2((float)(sc * acc[2 * i]), (float)(sc * acc[2 * i + 1]));
}

// Bins per chunk of passes of N / 2 angles: the most that D holds gives the fewest set-ups of a
// group (about as dear as five bins), fewer give the SMs equal shares.  cost: of the whole.
int aj_bins(const PWDev& d, int N, int slices, int nsm, long long* cost) {
  const int per = slices * ((d.na + N / 2 - 1) / (N / 2)) * ((d.ne + 127) / 128);
  int best = AJ_DCOLS / N;
  *cost = 0;
  for (int nb = AJ_DCOLS / N; nb >= 4; --nb) {
    const long long items = (long long)((d.K + nb - 1) / nb) * per;
    const long long c = (items + nsm - 1) / nsm * (nb + 5);
    if (*cost == 0 || c < *cost) {
      *cost = c;
      best = nb;
    }
  }
  return best;
}

// D columns of a bin: passes of 8 angles, or of 16 or 24, whichever cost less (20 angles in passes of
// 16 | 24: 128 elements, 400 x 300 voxels 11.5 | 7.1 ms, 64 x 64 0.77 | 0.80 ms).
int aj_columns(const PWDev& d, int slices, int nsm) {
  if (d.na <= 8) return 16;
  long long c32, c48;
  aj_bins(d, 32, slices, nsm, &c32);
  aj_bins(d, 48, slices, nsm, &c48);
  return c48 < c32 ? 48 : 32;
}

}  // namespace

cudaError_t launch_pw_adjoint(const PWDev& d0, const float2* cot, unsigned* gmax, float2* gX, double* acc,
                              cudaStream_t s) {
  const size_t n = (size_t)d0.ne * d0.K * d0.na;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto slices = [](long long v) { return (int)((v + AJ_SLICE - 1) / AJ_SLICE); };
  const int N = aj_columns(d0, slices((long long)d0.wt_nc * d0.nz), nsm);
  const bool band = d0.wt_w < d0.ne_pad;
  const auto kernel = N == 16 ? (band ? aj_tc_kernel<16, true> : aj_tc_kernel<16, false>)
                    : N == 32 ? (band ? aj_tc_kernel<32, true> : aj_tc_kernel<32, false>)
                              : (band ? aj_tc_kernel<48, true> : aj_tc_kernel<48, false>);
  const void* fn = (const void*)kernel;
  // the compute warps' register share needs the full allocation at launch
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, fn);
  if (e == cudaSuccess && a.numRegs != P5_REGS) e = cudaErrorInvalidConfiguration;
  if (e == cudaSuccess) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, aj_smem());
  }
  // gmax[1] (max n_k) is set once per plan; max |G| per call
  if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, 2 * n * sizeof(double), s);
  if (e == cudaSuccess) e = launch_absmax(reinterpret_cast<const float*>(cot), 2 * (size_t)d0.nx * d0.nz, gmax, s);
  if (e != cudaSuccess) return e;
  if (d0.rx_tab) aj_table_kernel<<<1216, 256, 0, s>>>(d0);
  PWDev d = d0;
  for (int c0 = 0; c0 < d0.nx; c0 += d0.wt_nc) {
    d.wt_c0 = c0;
    d.wt_nc = std::min(d0.wt_nc, d0.nx - c0);
    // a window table that does not hold all columns is refilled for each slab of them
    if (d0.wt_nc < d0.nx && (e = launch_pw_tc_window(d, const_cast<float*>(d.w_tab), const_cast<float*>(d.w_sum), s)) !=
                                cudaSuccess)
      return e;
    const long long v0 = (long long)c0 * d.nz, v1 = v0 + (long long)d.wt_nc * d.nz;
    long long cost;
    const int nb = aj_bins(d, N, slices(v1 - v0), nsm, &cost);
    kernel<<<nsm, P5_THREADS, aj_smem(), s>>>(d, cot, gmax, acc, v0, v1, nb);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  aj_finish_kernel<<<608, 256, 0, s>>>(acc, n, (double)d0.scale, gmax, gX);
  return cudaGetLastError();
}

}  // namespace fnum
