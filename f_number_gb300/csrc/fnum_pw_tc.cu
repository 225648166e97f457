// The plane-wave beamformer on the Blackwell tensor cores (tcgen05 + TMEM), kernel variant 9.
//
// Replaces the reference's per-bin phase matrix, cublasCgemm and normalisation
// (+cuda/gpu_bf_das_pw_rf.cu:1014-1057, +cuda/das_kernel_phase_shifts.cu:8-147).  For a
// voxel v and band bin k the compounded image gains
//     I_k(v) = n_k(v) sum_a t_{v,a}^k G_k(v, a),   G_k(v, a) = sum_e R_k(v, e) X_k(e, a),
//     R_k(v, e) = w_k(v, e) e^{2 pi i k u_e(v)},   t_{v,a} = e^{2 pi i u_a(v)},
// with the window value w, the receive and transmit delays u_e, u_a in cycles per bin and
// n_k = 1 / sum_e w (or 1).  G is a GEMM per bin: for a tile of 128 voxels (4 columns x 32
// rows, a voxel per TMEM lane) D[v][n] = sum_{e,q} A[v][2e + q] B[n][2e + q] with A = (Re R,
// Im R) in tensor memory and B the real form of X_k in shared memory (n: Re or Im of one
// angle).  Both operands are split into fp16 hi + lo and hi.lo + lo.hi + hi.hi accumulate in
// FP32 in tensor memory, restarted from zero at every bin.
//
// Kernel (persistent, one block per SM).  16 warps form A: warp w serves lane quadrant w % 4 (a
// tile column, a voxel per thread) and element slot w / 4, and works in units of 8 elements x 2
// bins: the phasors (kept in tensor memory, stepped by p <- p conj(rho), exact every 32 bins)
// times the window values, split into fp16, stored to the slot's A tiles.  Two threads issue the
// products, one for each bin of the pair, and a third copies B (bulk copies, two pairs in
// flight).  D is double-buffered; the slots read their angles' columns of it a pair later and
// run the transmit recurrence H <- H t + n_k D in registers, with the exact phase every 32 bins.
// The window of a voxel depends only on its column and the outermost element of each side, so
// its values come from a table built with the plan; per bin and voxel remain two table rows and
// n_k, formed 8 bins ahead.  An element pass holds as many groups of 8 as tensor memory has room
// for phasors.
//
// What bounds it: forming the A operand (step, window, split: about 20 instructions a term
// beside 3 x 8 NA fp16 FLOP of products).  One thread issues a tcgen05 instruction every ~45
// cycles whatever its size, and an mbarrier answers a test after ~160, which set the two
// issuers, the 8 x 2 unit (four products-worth a commit) and the tests asked ahead.
// 11 angles, 128 elements, 512 x 512 voxels: 22.6 ms with warp-level mma.sync (window and
// apertures re-formed per element pass, transmit recurrence per 16 elements), 16.0 ms here;
// 31 angles, 192 elements, 301 x 451: 79.3 and 28.9 ms (fewer, wider angle passes); 11 images of
// 161 x 224 kept apart: 47.7 and 2.5 ms (one launch instead of one FP32 launch per angle).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "fnum_device.cuh"
#include "fnum_internal.h"
#include "fnum_tc_beam.cuh"

namespace fnum {

namespace {

using namespace tcx;

constexpr int P5_TT = 8;                          // bins per aperture table
constexpr int P5_TP = P5_TT / 2;                  // pairs of bins
constexpr int P5_NT = 4;                          // element ranges in flight (aperture tables: 2)
constexpr int P5_NB = 2;                          // pairs of bins of B tiles in flight
// NT: angles per thread (a pass holds 4 NT: angle a0 + 4 j + slot belongs to a thread of that
// slot).  GP: element groups (of 8) per element pass.
template <int NT, int GP>
struct P5Cfg {
  static constexpr int N = NT <= 2 ? 16 : 8 * NT;     // D columns of a bin (mma N)
  static constexpr int SLOT = N / 4;                  // D columns of one slot's angles
  static constexpr int GROUP = 64 * N;                // B bytes per 8 elements: hi, lo
  static constexpr int B_BIN = GP * GROUP;
  static constexpr int A0 = 4 * N;                    // TMEM: per slot and bin of the pair the A tiles (8 hi, 8 lo)
  static constexpr int PH = A0 + 128;                 // TMEM: per group the phasors (16 columns)
  static constexpr int RHO = GP * P5_M * 64;          // shared memory: the phasor steps
  static constexpr int SMEM = RHO + P5_NB * 2 * B_BIN;
  static_assert(PH + 16 * GP <= 512, "tensor memory");
};

struct P5Shared {
  int4 tab[2][P5_TP][P5_M];          // per bin of a pair and voxel: row of w left | row right << 16, n_k (float bits)
  unsigned rng[P5_NT][P5_TP][4];     // per pair and column: element range lo | (0xffff - hi) << 16
  unsigned un[4];                    // the same over the whole band
  float2 red[3][P5_M];
  unsigned long long n_active, n_empty, n_exec;
  int item, frame, last;
  int abort_flag;
  uint32_t tmem;
  uint64_t bars[2 * 4 + 2 * 2 + 4 + 2 * P5_NT];
};

// Element groups a pass holds at most: all of a short array, else 8, which leave half of the
// block's shared memory to the L1 cache that the window loads want (128 elements, 11 angles,
// 512 x 512: 15.9 ms, with 12 groups 16.2; 96 elements, 5 angles: 1.92 and 1.79 ms).  A frame's
// own, so that it sums in the same order in a batch.
__host__ __device__ inline int p5_groups(const PWDev& d) { return d.ne <= 96 && d.na <= 16 ? 12 : 8; }
// groups per element pass: the tile's groups in as few passes as hold them, of equal width
__device__ __forceinline__ int p5_pass(int GP, int E_lo, int E_hi) {
  if (E_lo > E_hi) return GP;
  const int n = (E_hi >> 3) - (E_lo >> 3) + 1, passes = (n + GP - 1) / GP;
  return (n + passes - 1) / passes;
}

template <int NT, int GP, bool STACK, bool BATCH>
__global__ void __launch_bounds__(P5_THREADS, 1)
pw_tc_kernel(const PWDev d0, float2* image0, float* weights0, const PWBatchDev B) {
  using C = P5Cfg<NT, GP>;
  extern __shared__ __align__(16) unsigned char dyn[];
  P5Shared& sh = *reinterpret_cast<P5Shared*>(dyn);
  float4* rho = reinterpret_cast<float4*>(dyn + ((sizeof(P5Shared) + 127) & ~(size_t)127));
  const uint32_t bbase = smem_u32(rho) + (uint32_t)C::RHO;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = (int)p5_uni((uint32_t)tid >> 5);
  volatile int* abort_flag = &sh.abort_flag;
  const uint32_t bar0 = smem_u32(sh.bars);
  auto s_full = [&](uint32_t s) { return bar0 + 8u * s; };
  auto s_empty = [&](uint32_t s) { return bar0 + 8u * (4u + s); };
  auto b_full = [&](uint32_t s) { return bar0 + 8u * (8u + s); };
  auto b_empty = [&](uint32_t s) { return bar0 + 8u * (10u + s); };
  auto d_full = [&](uint32_t s) { return bar0 + 8u * (12u + s); };
  auto d_empty = [&](uint32_t s) { return bar0 + 8u * (14u + s); };
  auto r_full = [&](uint32_t s) { return bar0 + 8u * (16u + s); };
  auto r_empty = [&](uint32_t s) { return bar0 + 8u * (16u + P5_NT + s); };

  if (tid == 0) {
    for (int s = 0; s < 4; ++s) {
      mbar_init(s_full(s), 4);
      mbar_init(s_empty(s), 2);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(b_full(s), 1);
      mbar_init(b_empty(s), 2);
      mbar_init(d_full(s), 2);
      mbar_init(d_empty(s), P5_CW);
    }
    for (int s = 0; s < P5_NT; ++s) {
      mbar_init(r_full(s), P5_CW);
      mbar_init(r_empty(s), 3);
    }
    sh.abort_flag = 0;
    sh.n_active = sh.n_empty = sh.n_exec = 0ull;
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

  // The next item (a tile and a range of its bins), drawn by thread 0 while the others wait.
  auto fetch = [&](int cur) {
    int item = -1, frame = 0;
    if (!*abort_flag) {
      if constexpr (BATCH) {
        const int t = (int)atomicAdd(B.counter, 1ull);
        if (t < B.tile_start[B.n_frames]) {
          int lo = 0, hi = B.n_frames - 1;   // the frame whose item range holds t
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (B.tile_start[mid] <= t) lo = mid; else hi = mid - 1;
          }
          frame = lo;
          item = t - B.tile_start[lo];
        }
      } else {
        const int t = (int)atomicAdd(&d0.counters[3], 1ull);
        if (t < ((d0.wt_nc + TILE_X - 1) / TILE_X) * ((d0.nz + TILE_Z - 1) / TILE_Z) * d0.split) item = t;
      }
    }
    if (cur >= 0 && (item < 0 || frame != cur)) {
      const PWDev& f = BATCH ? B.frames[cur] : d0;
      atomicAdd(&f.counters[0], sh.n_active * (unsigned long long)f.na);
      atomicAdd(&f.counters[1], sh.n_empty * (unsigned long long)f.na);
      atomicAdd(&f.counters[4], sh.n_exec);
      sh.n_active = sh.n_empty = sh.n_exec = 0ull;
    }
    sh.item = item;
    sh.frame = frame;
  };
  uint32_t a_ph = 0;               // phases of the slots' A tiles (bit per slot)
  uint32_t nd = 0;                 // bins with products so far
  uint32_t ns = 0;                 // aperture tables so far
  const uint32_t lead = lane == 0 ? 1u : 0u;

  if (warp >= P5_CW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P5_REGS_I));
    for (;;) {
      __syncthreads();
      const int item = sh.item;
      if (item < 0) break;
      const PWDev& d = BATCH ? B.frames[sh.frame] : d0;
      unsigned long long* err = &d.counters[2];
      const int part = item % d.split;
      const int kt = d.k_ub - part * d.split_bins;
      const int nb = min(d.split_bins, kt - d.k_lb + 1);
      __syncthreads();
      const unsigned un = p5_uni(p5_join(sh.un));
      const int E_lo = (int)(un & 0xffffu), E_hi = un == 0xffffffffu ? -1 : 0xffff - (int)(un >> 16);
      const int gp = p5_pass(BATCH ? min(p5_groups(d), GP) : GP, E_lo, E_hi);
      const int role = warp - P5_CW;       // 0, 1: products of the first, second bin of a pair; 2: copies
      if (lane == 0 && role < 3) {
        const int n_grp = d.ne_pad >> 3;                      // element groups of 8 in the spectra
        const uint32_t idesc = idesc_f16(P5_M, C::N);
        const int np = (nb + 1) >> 1;                         // pairs of bins
        unsigned long long exec = 0;
        bool ok = true;
        for (int a0 = 0; a0 < d.na; a0 += 4 * NT) {
          const unsigned char* Bsrc = (const unsigned char*)d.tc_B + (size_t)(a0 / (4 * NT)) * d.K * n_grp * C::GROUP;
          int eb = E_lo <= E_hi ? E_lo & ~7 : 0;
          do {
            const int g_max = min(gp - 1, n_grp - 1 - (eb >> 3));
            const size_t row = (size_t)n_grp * C::GROUP;      // a bin's B bytes
            const unsigned char* src = Bsrc + (size_t)(kt - d.k_lb) * row + (size_t)(eb >> 3) * C::GROUP;
            for (int b = 0; b < np && ok; ++b, src -= 2 * row) {
              const uint32_t ri = ns % P5_NT;
              if (b % P5_TP == 0) ok = p5_wait(r_full(ri), (ns / P5_NT) & 1u, 0u, abort_flag, err);
              const unsigned r = p5_join(sh.rng[ri][b % P5_TP]);
              // the last use of this table's ranges
              if (b % P5_TP == P5_TP - 1 || b == np - 1) {
                mbar_arrive(r_empty(ri));
                ++ns;
              }
              const int g_lo = max(((int)(r & 0xffffu) - eb) >> 3, 0);
              const int g_hi = r == 0xffffffffu ? -1 : min((0xffff - (int)(r >> 16) - eb) >> 3, g_max);
              if (g_lo > g_hi) continue;
              const uint32_t bs = nd & 1u, ph = (nd >> 1) & 1u;      // B and D buffers of the pair
              if (role == 2) {
                // both bins' B tiles (a band's odd last bin stands in for its missing partner, whose weights are 0)
                ok = ok && p5_wait(b_empty(bs), ph ^ 1u, 0u, abort_flag, err);
                if (ok) {
                  const uint32_t bytes = (uint32_t)(g_hi - g_lo + 1) * C::GROUP;
                  const uint32_t dst = bbase + bs * (2 * C::B_BIN) + (uint32_t)g_lo * C::GROUP;
                  const unsigned char* p = src + (size_t)g_lo * C::GROUP;
                  mbar_expect_tx(b_full(bs), 2 * bytes);
                  bulk_load(dst, p, bytes, b_full(bs));
                  bulk_load(dst + C::B_BIN, 2 * b + 1 < nb ? p - row : p, bytes, b_full(bs));
                }
                exec += (unsigned long long)P5_M * 16 * (g_hi - g_lo + 1) * min(4 * NT, d.na - a0);
              } else {
                const uint32_t ask_d = p5_ask(d_empty(bs), ph ^ 1u), ask_b = p5_ask(b_full(bs), ph);
                uint32_t ask_a = p5_ask(s_full((uint32_t)g_lo & 3u), (a_ph >> (g_lo & 3)) & 1u);
                ok = ok && p5_wait(d_empty(bs), ph ^ 1u, ask_d, abort_flag, err) &&
                     p5_wait(b_full(bs), ph, ask_b, abort_flag, err);
                const uint32_t dcol = tmem + (2 * bs + (uint32_t)role) * C::N;
                constexpr uint32_t LO = (32u * C::N) >> 4, GR = C::GROUP >> 4;   // descriptor steps: lo half, group
                constexpr uint64_t HI = smem_desc_plain_hi(256);
                uint32_t bd = (uint32_t)smem_desc_plain(bbase + (2 * bs + (uint32_t)role) * C::B_BIN, 128, 256) +
                              (uint32_t)g_lo * GR;
                const uint32_t abase = tmem + C::A0 + 16u * (uint32_t)role;
                uint32_t accum = 0u;
                for (int g = g_lo; g <= g_hi; ++g, bd += GR) {
                  const uint32_t sl = (uint32_t)g & 3u, a = abase + 32u * sl;
                  ok = ok && p5_wait(s_full(sl), (a_ph >> sl) & 1u, ask_a, abort_flag, err);
                  const uint32_t nx = (sl + 1u) & 3u;
                  ask_a = p5_ask(s_full(nx), (a_ph >> nx) & 1u);
                  fence_after_sync();
                  // the small cross products first, so that fewer steps round a full-size sum
                  mma_f16_ts(dcol, a, HI | (uint64_t)(bd + LO), idesc, accum);
                  mma_f16_ts(dcol, a + 8u, HI | (uint64_t)bd, idesc, 1u);
                  mma_f16_ts(dcol, a, HI | (uint64_t)bd, idesc, 1u);
                  accum = 1u;
                  mma_commit(s_empty(sl));
                  a_ph ^= 1u << sl;
                }
                mma_commit(b_empty(bs));
                mma_commit(d_full(bs));
              }
              ++nd;
            }
            eb += 8 * gp;
          } while (eb <= E_hi && ok);
        }
        if (role == 2) sh.n_exec += exec;
      }
      __syncwarp();
      __syncthreads();
    }
  } else {
    // ----------------------------------------------------------------------------------- A and D
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P5_REGS_C));
    const int q = warp & 3, slot = warp >> 2;         // lane quadrant (tile column), slot
    const int vb = 32 * q + lane;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    float4* us = (BATCH ? B.u_scr : d0.u_scr) + (size_t)blockIdx.x * (size_t)(P5_M * 4 * 12) + vb;
    int cur = -1;                    // frame of the last item
    for (;;) {
      if (tid == 0) fetch(cur);
      __syncthreads();
      const int item = sh.item;
      if (item < 0) break;
      cur = sh.frame;
      const PWDev& d = BATCH ? B.frames[sh.frame] : d0;
      float2* image = BATCH ? B.images[sh.frame] : image0;
      unsigned long long* err = &d.counters[2];
      const int ntx = (d.wt_nc + TILE_X - 1) / TILE_X, ntz = (d.nz + TILE_Z - 1) / TILE_Z;
      const int tile = item / d.split, part = item - tile * d.split;
      int tx, tz;
      tile_coords(tile, ntx, ntz, tx, tz);
      const int cw = tx * TILE_X + q;                       // column within the window table's slab
      const int j = tz * TILE_Z + lane;
      const bool valid = (cw < d.wt_nc) && (j < d.nz);
      const int cc = min(cw, d.wt_nc - 1), ic = d.wt_c0 + cc, jc = min(j, d.nz - 1);
      const int ne = d.ne;
      // this item's bins: kt down, nb of them
      const int kt = d.k_ub - part * d.split_bins;
      const int nb = min(d.split_bins, kt - d.k_lb + 1);
      const int emid = (int)p5_uni((uint32_t)d.col_emid[ic]), e0 = (int)p5_uni((uint32_t)d.col_e0[ic]);
      if (slot == 0) {
        // the tile's elements: its apertures at the band's smallest F
        int ilb, iub;
        aperture(d.col_p[ic], d.row_p[jc], d.gmax, ne, ilb, iub);
        const int lo = min(ilb, emid), hi = max(iub, emid - 1);
        const bool some = valid && lo <= hi;
        const unsigned mn = __reduce_min_sync(0xffffffffu, some ? (unsigned)lo : 0xffffu);
        const int mx = __reduce_max_sync(0xffffffffu, some ? hi : -1);
        if (lead) sh.un[q] = mx < 0 ? 0xffffffffu : (mn | ((unsigned)(0xffff - mx) << 16));
      }
      __syncthreads();
      const unsigned un = p5_uni(p5_join(sh.un));
      const int E_lo = (int)(un & 0xffffu), E_hi = un == 0xffffffffu ? -1 : 0xffff - (int)(un >> 16);
      const int gp = p5_pass(BATCH ? min(p5_groups(d), GP) : GP, E_lo, E_hi);
      const float inv_sigma = STACK ? 1.0f : 1.0f / tc_scale(*d.tc_max);
      const int n_grp = d.ne_pad >> 3;                      // element groups of 8 in the spectra
      const int tb = (d.tc_tb > 0 && d.tc_tb < 32) ? d.tc_tb : 32;   // bins between exact re-anchorings
      const int nstretch = (nb + P5_TT - 1) / P5_TT;
      float* weights = BATCH ? B.weights[sh.frame] : weights0;
      float2 acc = make_float2(0.0f, 0.0f), comp = make_float2(0.0f, 0.0f);
      unsigned c_act = 0, c_emp = 0;
      const int n_img = STACK ? d.na : 1;
      const size_t nvox = (size_t)d.nx * d.nz, vox = (size_t)ic * d.nz + jc;
      float2* out = d.split > 1 ? d.part + (size_t)part * n_img * nvox : image;

      for (int a0 = 0; a0 < d.na; a0 += 4 * NT) {
        // a tile without any aperture still runs one pass: its bins are counted and its weights written
        int eb = E_lo <= E_hi ? E_lo & ~7 : 0;
        bool first = a0 == 0;
        float2 sacc[STACK ? NT : 1];
        if constexpr (STACK) {
#pragma unroll
          for (int t = 0; t < NT; ++t) sacc[t] = make_float2(0.0f, 0.0f);
        }
        do {
          // Aperture table of stretch s: per bin and voxel the rows of the window table and n_k, per pair of bins
          // and column the element range; this warp takes its column's pair `slot`.
          auto build = [&](int s) {
            const uint32_t tbuf = (ns + (uint32_t)s) & 1u, ri = (ns + (uint32_t)s) % P5_NT;
            const uint32_t ask = p5_ask(r_empty(ri), (((ns + (uint32_t)s) / P5_NT) & 1u) ^ 1u);
            const dfl xp = d.col_p[ic], zp = d.row_p[jc];
            const P5Window wt = p5_window(d, cc, e0);
            int lo = 0xffff, hi = -1, rows[2];
            float inv[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int b = s * P5_TT + 2 * slot + t;
              const int kk = max(kt - b - d.k_lb, 0);
              int ilb, iub;
              p5_aperture(xp, zp, d.g[kk], ne, ilb, iub);
              // a side without elements takes the zero row
              const int row_l = ilb < emid ? ilb : wt.zero, row_r = iub >= emid ? iub : wt.zero;
              const float W = __ldg(wt.sum + row_l) + __ldg(wt.sum + row_r);
              inv[t] = W > 0.0f ? (d.norm ? __frcp_rn(W) : 1.0f) : 0.0f;
              const int a = min(ilb, emid), z = max(iub, emid - 1);
              const bool act = valid && b < nb && W > 0.0f && a <= z;
              if (first && valid && b < nb) {
                if (act) c_act += (unsigned)(z - a + 1); else ++c_emp;
                if (kk == d.K - 1 && weights) weights[vox] = W;
              }
              rows[t] = b < nb ? row_l | (row_r << 16) : wt.zero | (wt.zero << 16);   // beyond the band: weights 0
              if (act) {
                lo = min(lo, a);
                hi = max(hi, z);
              }
            }
            p5_wait(r_empty(ri), (((ns + (uint32_t)s) / P5_NT) & 1u) ^ 1u, ask, abort_flag, err);
            sh.tab[tbuf][slot][vb] = make_int4(rows[0], __float_as_int(inv[0]), rows[1], __float_as_int(inv[1]));
            const unsigned mn = __reduce_min_sync(0xffffffffu, (unsigned)lo);
            const int mx = __reduce_max_sync(0xffffffffu, hi);
            if (lead) sh.rng[ri][slot][q] = mx < 0 ? 0xffffffffu : (mn | ((unsigned)(0xffff - mx) << 16));
            __syncwarp();
            mbar_arrive_if(lead, r_full(ri));
          };
          build(0);
          const float* wcol = p5_window(d, cc, e0).tab + eb;
          const int g_max = min(gp - 1, n_grp - 1 - (eb >> 3));
          // phasor steps rho = e^{2 pi i u} into shared memory, by element pairs {Re, Re, Im, Im};
          // the delays u to scratch for the exact anchors
#pragma unroll 1
          for (int g = slot; g <= min(g_max, (E_hi - eb) >> 3); g += 4) {
#pragma unroll
            for (int j2 = 0; j2 < 4; ++j2) {
              dfl u[2];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int e = min(eb + 8 * g + 2 * j2 + h, ne - 1);
                u[h] = df_sqrt(df_add(df_sqr(df_sub(d.el_u[e], d.col_u[ic])), d.row_u2[jc]));
              }
              float2 r, m;
              p5_cis2(1.0f, make_float2(u[0].x, u[1].x), make_float2(u[0].y, u[1].y), r, m);
              rho[(4 * g + j2) * P5_M + vb] = make_float4(r.x, r.y, m.x, m.y);
              us[(size_t)(4 * g + j2) * P5_M] = make_float4(u[0].x, u[1].x, u[0].y, u[1].y);
            }
          }
          // transmit phasors of the thread's angles, by angle pairs
          float2 tr[NT / 2], ti[NT / 2], Hr[NT / 2], Hi[NT / 2];
          auto cis_tx = [&](float k, int p, float2& re, float2& im) {
            dfl u[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int a = min(a0 + 4 * (2 * p + h) + slot, d.na - 1);
              u[h] = df_add(d.tx_ax[(size_t)a * d.nx + ic], d.tx_az[(size_t)a * d.nz + jc]);
            }
            p5_cis2(k, make_float2(u[0].x, u[1].x), make_float2(u[0].y, u[1].y), re, im);
          };
#pragma unroll
          for (int p = 0; p < NT / 2; ++p) {
            cis_tx(1.0f, p, tr[p], ti[p]);
            Hr[p] = Hi[p] = make_float2(0.0f, 0.0f);
          }
          // the transmit recurrence H <- H t + n_k D for the two bins of a pair
          auto consume = [&](bool some, float iw0, float iw1, uint32_t ask) {
            float D[2][2 * NT];
            if (some) {
              const uint32_t db = nd & 1u;
              p5_wait(d_full(db), (nd >> 1) & 1u, ask, abort_flag, err);
              fence_after_sync();
              const uint32_t td = tl + (uint32_t)(2 * db * C::N + slot * C::SLOT);
              p5_ld_cols<2 * NT>(td, D[0]);
              p5_ld_cols<2 * NT>(td + C::N, D[1]);
              tmem_wait_ld();
              fence_before_sync();
              __syncwarp();
              mbar_arrive_if(lead, d_empty(db));
              ++nd;
            } else {
#pragma unroll
              for (int c = 0; c < 2 * NT; ++c) D[0][c] = D[1][c] = 0.0f;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const float2 w2 = p5_dup(x ? iw1 : iw0);
#pragma unroll
              for (int p = 0; p < NT / 2; ++p) {
                const float2 hr = Hr[p], hi = Hi[p], tn = p5_neg(ti[p]);
                const float2 dr = __fmul2_rn(make_float2(D[x][4 * p], D[x][4 * p + 1]), w2);
                const float2 di = __fmul2_rn(make_float2(D[x][4 * p + 2], D[x][4 * p + 3]), w2);
                Hr[p] = __ffma2_rn(hr, tr[p], __ffma2_rn(hi, tn, dr));
                Hi[p] = __ffma2_rn(hr, ti[p], __ffma2_rn(hi, tr[p], di));
              }
            }
          };
          // every tb bins (and at the end) the exact phase at the last bin consumed
          auto flush = [&](int k) {
            float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int p = 0; p < NT / 2; ++p) {
              float2 cr, ci;
              cis_tx((float)k, p, cr, ci);
              const float2 vr = __ffma2_rn(cr, Hr[p], p5_neg(__fmul2_rn(ci, Hi[p])));
              const float2 vi = __ffma2_rn(cr, Hi[p], __fmul2_rn(ci, Hr[p]));
              if constexpr (STACK) {
                sacc[2 * p].x += vr.x;
                sacc[2 * p].y += vi.x;
                sacc[2 * p + 1].x += vr.y;
                sacc[2 * p + 1].y += vi.y;
              } else {
                if (a0 + 8 * p + slot < d.na) {
                  sum.x += vr.x;
                  sum.y += vi.x;
                }
                if (a0 + 8 * p + 4 + slot < d.na) {
                  sum.x += vr.y;
                  sum.y += vi.y;
                }
              }
              Hr[p] = Hi[p] = make_float2(0.0f, 0.0f);
            }
            if constexpr (!STACK) {
              const float yx = sum.x - comp.x, sx = acc.x + yx;
              comp.x = (sx - acc.x) - yx;
              acc.x = sx;
              const float yy = sum.y - comp.y, sy = acc.y + yy;
              comp.y = (sy - acc.y) - yy;
              acc.y = sy;
            }
          };
          const uint32_t ta = tl + (uint32_t)(C::A0 + 32 * slot);     // the slot's A tiles
          const uint32_t sf = s_full((uint32_t)slot), se = s_empty((uint32_t)slot);
          const float4* rhov = rho + vb;
          unsigned live = 0u;     // groups whose phasors belong to the previous bin
          bool pend = false;      // the pair before has products
          float pend_iw0 = 0.0f, pend_iw1 = 0.0f;
#pragma unroll 1
          for (int s = 0; s < nstretch; ++s) {
            // table s is complete, and no warp reads the one before it any more
            p5_bar();
            if (s + 1 < nstretch) build(s + 1);
            const int npair = (min(P5_TT, nb - s * P5_TT) + 1) >> 1;
            const bool mark = (s & (tb / P5_TT - 1)) == 0;      // a re-anchoring
            if (mark) live = 0u;
            const int4* trow = &sh.tab[(ns + (uint32_t)s) & 1u][0][vb];
            const unsigned(*rrow)[4] = sh.rng[(ns + (uint32_t)s) % P5_NT];
#pragma unroll 1
            for (int t = 0; t < npair; ++t) {
              const unsigned r = p5_uni(p5_join(rrow[t]));
              const int4 te = trow[t * P5_M];
              // the pair's groups of 8 elements in this pass
              const int g_lo = max(((int)(r & 0xffffu) - eb) >> 3, 0);
              const int g_hi = r == 0xffffffffu ? -1 : min((0xffff - (int)(r >> 16) - eb) >> 3, g_max);
              const unsigned mask = g_lo <= g_hi ? (2u << g_hi) - (1u << g_lo) : 0u;
              const unsigned exact = mask & ~live;
              // rows of the window table (as offsets): left and right side of each bin
              const unsigned ol0 = (unsigned)(te.x & 0xffff) * (unsigned)d.wt_w, or0 = (unsigned)(te.x >> 16) * (unsigned)d.wt_w;
              const unsigned ol1 = (unsigned)(te.z & 0xffff) * (unsigned)d.wt_w, or1 = (unsigned)(te.z >> 16) * (unsigned)d.wt_w;
#pragma unroll 1
              for (int g = g_lo + ((slot - g_lo) & 3); g <= g_hi; g += 4) {
                const uint32_t tp = tl + (uint32_t)(C::PH + 16 * g);
                const int e8 = eb + 8 * g;
                const bool fresh = (exact >> g) & 1u;
                float p[16];
                if (!fresh) tmem_ld16_nowait(tp, p);
                const uint32_t ask_a = p5_ask(se, a_ph ^ 1u);
                const bool left = e8 + 8 <= emid;
                float4 w[2][2];
                {
                  const float4* w0 = reinterpret_cast<const float4*>(wcol + ((left ? ol0 : or0) + 8u * (unsigned)g));
                  const float4* w1 = reinterpret_cast<const float4*>(wcol + ((left ? ol1 : or1) + 8u * (unsigned)g));
                  w[0][0] = __ldg(w0);
                  w[0][1] = __ldg(w0 + 1);
                  w[1][0] = __ldg(w1);
                  w[1][1] = __ldg(w1 + 1);
                }
                float r4[16];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                  const float4 v = rhov[(4 * g + x) * P5_M];
                  r4[4 * x] = v.x;
                  r4[4 * x + 1] = v.y;
                  r4[4 * x + 2] = v.z;
                  r4[4 * x + 3] = v.w;
                }
                if (fresh) {
                  // exact phasors of the pair's first bin
                  const float kf = (float)(kt - s * P5_TT - 2 * t);
#pragma unroll
                  for (int x = 0; x < 4; ++x) {
                    const float4 u = us[(size_t)(4 * g + x) * P5_M];
                    float2 re, im;
                    p5_cis2(kf, make_float2(u.x, u.y), make_float2(u.z, u.w), re, im);
                    p[4 * x] = re.x;
                    p[4 * x + 1] = re.y;
                    p[4 * x + 2] = im.x;
                    p[4 * x + 3] = im.y;
                  }
                } else {
                  tmem_wait_ld();
                  p5_rotate(p, r4);
                }
                if (e8 < emid && !left) {
                  // the group around the voxel's column: the left side's values too
                  __syncwarp();
                  const float4* w0 = reinterpret_cast<const float4*>(wcol + (ol0 + 8u * (unsigned)g));
                  const float4* w1 = reinterpret_cast<const float4*>(wcol + (ol1 + 8u * (unsigned)g));
#pragma unroll
                  for (int x = 0; x < 2; ++x) {
                    const float4 v = __ldg((x ? w1 : w0)), z = __ldg((x ? w1 : w0) + 1);
                    w[x][0] = make_float4(w[x][0].x + v.x, w[x][0].y + v.y, w[x][0].z + v.z, w[x][0].w + v.w);
                    w[x][1] = make_float4(w[x][1].x + z.x, w[x][1].y + z.y, w[x][1].z + z.z, w[x][1].w + z.w);
                  }
                }
                uint32_t h[8], l[8];
                p5_operand(w[0][0], w[0][1], p, h, l);
                // the slot's A tiles are free once the products that read them last are complete
                p5_wait(se, a_ph ^ 1u, ask_a, abort_flag, err);
                fence_after_sync();
                tmem_st8(ta, h);
                tmem_st8(ta + 8u, l);
                p5_rotate(p, r4);
                tmem_st16(tp, p);
                p5_operand(w[1][0], w[1][1], p, h, l);
                tmem_st8(ta + 16u, h);
                tmem_st8(ta + 24u, l);
                tmem_wait_st();
                fence_before_sync();
                __syncwarp();
                mbar_arrive_if(lead, sf);
                a_ph ^= 1u;
              }
              live = mask;
              const uint32_t ask_d = pend ? p5_ask(d_full(nd & 1u), (nd >> 1) & 1u) : 0u;
              // the previous pair's products have had this pair's A to complete behind
              if (s + t > 0) {
                consume(pend, pend_iw0, pend_iw1, ask_d);
                if (mark && t == 0) flush(kt - s * P5_TT + 1);
              }
              pend = mask != 0u;
              pend_iw0 = __int_as_float(te.y);
              pend_iw1 = __int_as_float(te.w);
            }
          }
          consume(pend, pend_iw0, pend_iw1, 0u);
          flush(kt - ((nb + 1) & ~1) + 1);
          ns += (uint32_t)nstretch;
          first = false;
          eb += 8 * gp;
        } while (eb <= E_hi);
        if constexpr (STACK) {
          if (valid) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              const int a = a0 + 4 * t + slot;
              if (a < d.na) {
                const float is = 1.0f / tc_scale(d.tc_max[a]);
                out[(size_t)a * nvox + vox] = make_float2(sacc[t].x * d.scale * is, sacc[t].y * d.scale * is);
              }
            }
          }
        }
      }
      {
        const unsigned na = __reduce_add_sync(0xffffffffu, c_act), nm = __reduce_add_sync(0xffffffffu, c_emp);
        if (lead) {
          atomicAdd(&sh.n_active, (unsigned long long)na);
          atomicAdd(&sh.n_empty, (unsigned long long)nm);
        }
      }
      if constexpr (!STACK) {
        if (slot > 0) sh.red[slot - 1][vb] = acc;
        p5_bar();
        if (slot == 0 && valid) {
          float2 o = acc;
#pragma unroll
          for (int t = 0; t < 3; ++t) {
            o.x += sh.red[t][vb].x;
            o.y += sh.red[t][vb].y;
          }
          out[vox] = make_float2(o.x * d.scale * inv_sigma, o.y * d.scale * inv_sigma);
        }
      }
      if (valid && (STACK || slot == 0) && (d.counters[2] & FLAG_NONFINITE))
        p5_nonfinite(d, out + vox, STACK ? nvox : 0, cc, jc, kt, nb, STACK ? slot : 0, STACK ? 4 : 1);
      if (d.split > 1) {
        // the last of the tile's bin ranges to finish adds them up, in order
        unsigned* cnt = &d.tile_cnt[(size_t)(d.wt_c0 / TILE_X) * ntz + tile];
        __threadfence();
        p5_bar();
        if (tid == 0) sh.last = atomicAdd(cnt, 1u) == (unsigned)(d.split - 1);
        p5_bar();
        if (sh.last) {
          __threadfence();
          if (valid) {
            for (int a = slot; a < n_img; a += 4) {
              float2 s = make_float2(0.0f, 0.0f);
              for (int p = 0; p < d.split; ++p) {
                const float2 v = __ldcg(d.part + ((size_t)p * n_img + a) * nvox + vox);
                s.x += v.x;
                s.y += v.y;
              }
              image[(size_t)a * nvox + vox] = s;
            }
          }
        }
      }
      __syncthreads();
    }
  }
  // after a timeout, give the copies and products in flight time to land before the tensor
  // memory is freed (they take microseconds)
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

// ---------------------------------------------------------------------------
// operands
// ---------------------------------------------------------------------------
// Window values w_tab[column][row][e] and their sums w_sum[column][row] of the slab's columns, rows and
// elements counted from the column's first one e0.  A row is the aperture's outermost element of
// one side: row r < emid holds the left side's elements r .. emid - 1, row r >= emid the right
// side's emid .. r; the last row and the padding are zero.  The half-width, and so the window,
// depends on the column and that element alone.
__global__ void __launch_bounds__(128) pw_tc_window_kernel(const PWDev d, float* __restrict__ tab,
                                                           float* __restrict__ sum) {
  const int col = d.wt_c0 + blockIdx.x, ne = d.ne, e0 = d.col_e0 ? d.col_e0[col] : 0;
  const int row = (int)blockIdx.y < d.wt_rows ? e0 + (int)blockIdx.y : ne;
  const dfl xm = d.col_m[col];
  const int emid = d.col_emid[col];
  const bool left = row < emid;
  float L = 0.0f;
  if (row < ne) L = left ? half_left(d.el_lb, xm, row, ne) : half_right(d.el_ub, xm, row);
  const size_t line = (size_t)blockIdx.x * (d.wt_rows + 1) + blockIdx.y;
  float* o = tab + line * d.wt_w;
  for (int i = threadIdx.x; i < d.wt_w; i += blockDim.x) {
    const int e = e0 + i;
    float w = 0.0f;
    if (row < ne && L > 0.0f && (left ? (e >= row && e < emid) : (e >= emid && e <= row))) {
      const dfl c = d.el_m[e];
      w = win_apply(d.window_id, d.window_par, fabsf((c.x - xm.x) + (c.y - xm.y)), L);
    }
    o[i] = w;
  }
  if (threadIdx.x == 0) {
    float W = 0.0f;
    if (row < ne && L > 0.0f) {
      const float ip = (d.window_par > 0.0f) ? 1.0f / d.window_par : 0.0f;
      if (left) {
        const dfl c = d.el_m[emid - 1];
        W = win_sum_rt(d.window_id, (xm.x - c.x) + (xm.y - c.y), d.pitch_f, emid - row, 1.0f / L, d.window_par, ip);
      } else {
        const dfl c = d.el_m[emid];
        W = win_sum_rt(d.window_id, (c.x - xm.x) + (c.y - xm.y), d.pitch_f, row - emid + 1, 1.0f / L, d.window_par, ip);
      }
    }
    sum[line] = W;
  }
}

// largest |component| of the finite band spectra (float bits; >= 0 floats order as ints): of all the
// launch's angles into out[0], or with a column of blocks per angle (own) of each into out[angle]
__global__ void __launch_bounds__(256) pw_tc_absmax_kernel(const PWDev d, unsigned* out, int own) {
  const size_t na = own ? 1 : d.na, n = (size_t)d.ne * d.K * na;
  float m = 0.0f;
  for (size_t i = (size_t)blockIdx.y * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.y * blockDim.x) {
    const size_t ek = i / na, a = own ? blockIdx.x : i - ek * na;
    const float2 x = d.X[ek * d.x_na + d.x_a0 + a];
    if (p5_finite(x)) m = fmaxf(m, fmaxf(fabsf(x.x), fabsf(x.y)));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out + blockIdx.x, __float_as_uint(m));
}

// B tiles of the spectra, in the order the products read them: [angle pass][bin][element
// group of 8][hi, lo][8 columns n][K half][n][8 fp16].  Column n belongs to slot n / (N / 4);
// with c = n % (N / 4), it holds the real (c % 4 < 2) or imaginary part of G for the slot's
// angle j = 2 (c / 4) + c % 2.  Values that are not finite are left out (p5_nonfinite).  The fp16 scale
// is common to the angles of a compound, whose products share an accumulator, and each angle's own
// for images kept apart (own): what the loudest angle costs a quieter one in bits is lost in
// their sum, but not in its own image.
__global__ void __launch_bounds__(256) pw_tc_operand_kernel(const PWDev d, int n_ap, int nt, int N, int own) {
  const int G = d.ne_pad >> 3;
  const size_t n_all = (size_t)n_ap * d.K * G * N * 2;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (d.split > 1) {   // no bin range of a tile is done yet
    const size_t n_tiles = (size_t)((d.nx + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z);
    for (size_t t = i; t < n_tiles; t += (size_t)gridDim.x * blockDim.x) d.tile_cnt[t] = 0u;
  }
  if (i >= n_all) return;
  const int in_group = (int)(i % (2 * N));
  size_t r = i / (2 * N);
  const int g = (int)(r % G);
  r /= G;
  const int kk = (int)(r % d.K), ap = (int)(r / d.K);
  const int n = 8 * (in_group >> 4) + (in_group & 7), kc = (in_group >> 3) & 1;
  const int slot = n / (N / 4), c = n % (N / 4);
  const int j = 2 * (c >> 2) + (c & 1), imag = (c >> 1) & 1;
  const int a = ap * 4 * nt + 4 * j + slot;
  const float sigma = tc_scale(d.tc_max[own ? min(a, d.na - 1) : 0]);
  unsigned h[4], l[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int e = 8 * g + 4 * kc + t;
    float2 x = make_float2(0.0f, 0.0f);
    if (j < nt && a < d.na && e < d.ne) x = d.X[((size_t)e * d.K + kk) * d.x_na + d.x_a0 + a];
    if (!p5_finite(x)) {
      x = make_float2(0.0f, 0.0f);
      atomicOr(&d.counters[2], FLAG_NONFINITE);
    }
    x.x *= sigma;
    x.y *= sigma;
    tc_split_mx(imag ? x.y : x.x, imag ? x.x : -x.y, h[t], l[t]);
  }
  uint4* o = d.tc_B + (((size_t)ap * d.K + kk) * G + g) * (size_t)(4 * N) + in_group;
  o[0] = make_uint4(h[0], h[1], h[2], h[3]);
  o[2 * N] = make_uint4(l[0], l[1], l[2], l[3]);
}

typedef void (*p5_kernel_t)(const PWDev, float2*, float*, const PWBatchDev);

struct P5Choice {
  p5_kernel_t fn;
  int nt, n, smem;
};

template <int NT, int GP>
P5Choice p5_choice(bool stack, bool batch) {
  using C = P5Cfg<NT, GP>;
  P5Choice c{};
  c.fn = batch ? pw_tc_kernel<NT, GP, false, true> : (stack ? pw_tc_kernel<NT, GP, true, false>
                                                             : pw_tc_kernel<NT, GP, false, false>);
  c.nt = NT;
  c.n = C::N;
  c.smem = (int)sizeof(P5Shared) + 128 + C::SMEM;
  return c;
}

// Angles per thread and groups per element pass of a frame; of a batch, the angles of its class and
// room for either number of groups.
P5Choice p5_pick(int na, int groups, bool stack, bool batch) {
  if (na > 24) return p5_choice<8, 8>(stack, batch);
  if (na > 16) return p5_choice<6, 8>(stack, batch);
  if (na > 8) return groups > 8 ? p5_choice<4, 12>(stack, batch) : p5_choice<4, 8>(stack, batch);
  return groups > 8 ? p5_choice<2, 12>(stack, batch) : p5_choice<2, 8>(stack, batch);
}

int p5_sms() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm > 0 ? nsm : 1;
}

cudaError_t p5_smem_optin() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 64 && done[dev]) return cudaSuccess;
  for (int na : {8, 16, 24, 32})
    for (int v = 0; v < 5; ++v) {
      const P5Choice c = p5_pick(na, v < 3 ? 12 : 8, v == 1 || v == 4, v == 2);
      // the compute warps' register share needs the full allocation at launch
      cudaFuncAttributes a;
      if ((e = cudaFuncGetAttributes(&a, (const void*)c.fn)) != cudaSuccess) return e;
      if (a.numRegs != P5_REGS) return cudaErrorInvalidConfiguration;
      if ((e = cudaFuncSetAttribute((const void*)c.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, c.smem)) !=
          cudaSuccess)
        return e;
    }
  if (dev < 64) done[dev] = true;
  return cudaSuccess;
}

}  // namespace

int pw_tc_class(int na) { return na > 16 ? 1 : 0; }

size_t pw_tc_operand_bytes(int na, int K, int ne_pad) {
  const P5Choice c = p5_pick(na, 8, false, false);
  // a batch may run a frame with its class's widest passes
  const P5Choice w = p5_pick(pw_tc_class(na) ? 32 : 16, 8, false, false);
  const size_t g = (size_t)K * (ne_pad >> 3) * 64;
  return std::max((size_t)((na + 4 * c.nt - 1) / (4 * c.nt)) * c.n, (size_t)((na + 4 * w.nt - 1) / (4 * w.nt)) * w.n) * g;
}

size_t pw_tc_scratch_bytes(int grid) { return (size_t)grid * P5_M * 4 * 12 * sizeof(float4); }

int pw_tc_grid(const PWDev& d) {
  const int tiles = ((d.wt_nc + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z) * d.split;
  return std::max(1, std::min(tiles, p5_sms()));
}
int pw_tc_items(const PWDev& d) {
  return ((d.nx + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z) * d.split;
}
int pw_tc_batch_grid() { return p5_sms(); }

// Bin ranges per tile.  A tile is one block's work, so a launch of few tiles would leave most
// SMs idle: its band is split into ranges of at least 64 bins (each pays two exact anchors and
// the tile's set-up) until there are about six items per SM, so that the last wave costs a sixth.
// The kernel for one or two angles has a shorter set-up: at least 32 bins, or 16 while 32 would
// give fewer items than the blocks that fit the SMs, two each.  One angle, at least 64 | 32 | 16 bins:
// 48 x 57 voxels, 64 elements 128 | 97 | 87 us, 64 x 64, 128 elements 483 | 317 | 299 us,
// 128 x 128 581 | 580 | 599 us.
void pw_tc_pick_split(PWDev& d) {
  const int tiles = ((d.wt_nc + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z), nsm = p5_sms();
  int s = (6 * nsm + tiles - 1) / tiles;
  const int least = d.na > 2 ? 64 : (tiles * (d.K / 32) < 2 * nsm ? 16 : 32), unit = std::min(least, 32);
  s = std::max(1, std::min(s, d.K / least));
  d.split_bins = ((d.K + s - 1) / s + unit - 1) / unit * unit;
  d.split = (d.K + d.split_bins - 1) / d.split_bins;
}

cudaError_t launch_pw_tc_window(const PWDev& d, float* tab, float* sum, cudaStream_t s) {
  const dim3 grid(d.wt_nc, d.wt_rows + 1);   // columns in x: y holds 65535 blocks, elements are 4096 at most
  pw_tc_window_kernel<<<grid, 128, 0, s>>>(d, tab, sum);
  return cudaGetLastError();
}

cudaError_t launch_pw_tc_operand(const PWDev& d, int na_class, bool stack, cudaStream_t s) {
  if (!d.tc_B || !d.tc_max) return cudaErrorInvalidValue;
  const unsigned rows = stack ? (unsigned)d.na : 1u;
  cudaError_t e = cudaMemsetAsync(d.tc_max, 0, rows * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  pw_tc_absmax_kernel<<<dim3(rows, (304 + rows - 1) / rows), 256, 0, s>>>(d, d.tc_max, stack);
  const P5Choice c = p5_pick(na_class > 0 ? na_class : d.na, 8, false, false);
  const int n_ap = (d.na + 4 * c.nt - 1) / (4 * c.nt);
  const size_t n = (size_t)n_ap * d.K * (d.ne_pad >> 3) * c.n * 2;
  pw_tc_operand_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d, n_ap, c.nt, c.n, stack);
  return cudaGetLastError();
}

cudaError_t launch_pw_tc(const PWDev& d0, bool stack, float2* image, float* weights, cudaStream_t s) {
  if (d0.na <= 2) return launch_pw_few(d0, stack, image, weights, s);
  cudaError_t e = p5_smem_optin();
  if (e == cudaSuccess) e = launch_pw_tc_operand(d0, 0, stack, s);
  if (e != cudaSuccess) return e;
  const P5Choice c = p5_pick(d0.na, p5_groups(d0), stack, false);
  PWDev d = d0;
  const int slab = d0.wt_nc;
  for (int c0 = 0; c0 < d0.nx; c0 += slab) {
    d.wt_c0 = c0;
    d.wt_nc = std::min(slab, d0.nx - c0);
    // a window table that does not hold all columns is refilled for each slab of them
    if (slab < d0.nx && (e = launch_pw_tc_window(d, const_cast<float*>(d.w_tab), const_cast<float*>(d.w_sum), s)) !=
                            cudaSuccess)
      return e;
    if ((e = cudaMemsetAsync(d.counters + 3, 0, sizeof(unsigned long long), s)) != cudaSuccess) return e;
    c.fn<<<pw_tc_grid(d), P5_THREADS, c.smem, s>>>(d, image, weights, PWBatchDev{});
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_pw_tc_batch(const PWBatchDev& B, int na_class, int grid, cudaStream_t s) {
  cudaError_t e = p5_smem_optin();
  if (e == cudaSuccess) e = cudaMemsetAsync(B.counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  const P5Choice c = p5_pick(na_class, 12, false, true);
  c.fn<<<grid, P5_THREADS, c.smem, s>>>(PWDev{}, nullptr, nullptr, B);
  return cudaGetLastError();
}

}  // namespace fnum
