// The synthetic-aperture beamformer on the Blackwell tensor cores (tcgen05).
//
// Replaces the reference's per-bin, per-transmit phase matrices and cublasCgemm
// calls (+cuda/gpu_bf_saft_rf.cu:1144-1201, +cuda/saft_kernel_phase_shifts.cu:8-199).
// For a voxel v and band bin k the image term is a bilinear form in the
// transmit and receive phasors:
//     I_k(v) = n_k(v) sum_t a_t Y_t,   Y_t = sum_r X'_k(t, r) b_r,
//     a_t = w_tx(v, t, k) e^{2 pi i k u_t(v)},   b_r = w_rx(v, r, k) e^{2 pi i k u_r(v)},
// with X'_k(t, r) = X_k(t, r) e^{2 pi i k t0 / N} (the time offset folded into the
// spectra), n_k = 1 / (W_tx W_rx) of the normalisations that are on, and
// u_e(v) = |v - c_e| f_s / (N c) the one-way delay in cycles per bin.
//
// Y is a GEMM per bin: for a tile of 128 voxels (4 columns x 32 rows, a voxel per TMEM lane)
//     D[v][n(t, p)] = sum_{r, q} A[v][2r + q] B[n(t, p)][2r + q]
// with A = (Re b_r, Im b_r) and B the real form of X'_k,
//     B[(t, 0)][(r, .)] = Re X', -Im X',   B[(t, 1)][(r, .)] = Im X', Re X',
// so that D[v][(t, 0)] + i D[v][(t, 1)] = Y_t.  Both operands are split into fp16 hi + lo parts
// (the spectra scaled by a power of two into fp16 range) and the products hi.lo + lo.hi + hi.hi
// are accumulated in FP32 in tensor memory; the CUDA cores only form the phasors and the dot
// products with a (O(elements) work per voxel and bin, where the recurrence kernels do
// O(elements^2)).
//
// Kernel (persistent, one block per SM).  16 warps form A and take the dot products: warp w
// serves lane quadrant w % 4 (a tile column, a voxel per thread) and element slot w / 4 (the
// groups of 8 elements g with g % 4 = slot).  Per bin only the groups that the tile's apertures
// touch run, with N = 16 (groups).  Per group a warp steps its phasors p <- p conj(rho) (kept in
// tensor memory, 16 columns a group; exact every 16 bins and when a group comes back into
// range), multiplies them with the receive window and writes the split rows to its slot's A tile
// in shared memory.  Two threads issue the group's products (each for half of the transmit
// elements), two copy its B tiles in turn.  When a bin's D is complete every warp adds n_k sum_t w_tx p_t Y_t of its groups to its
// voxel (compensated sum).  The window of a voxel depends only on its column and the outermost
// element of each side, so its values come from a table built with the plan; per bin and voxel
// remain the table's rows and n_k, formed 4 bins ahead.
//
// What keeps the tensor cores busy is that a bin's products run beside the warps' work:
// - up to 64 elements the phasors of two bins fit tensor memory: a bin's A is formed before the
//   previous bin's dot products are taken;
// - beyond, each slot forms the A of its first group before them (those phasors are stepped back
//   for the dot product) and the others after them;
// - bins of up to 64 elements use the two halves of D in turn, wider ones all of it.
// A band of few tiles is split over the idle SMs.
//
// What bounds it: the latency of the chain from a bin's D over the dot products and the A of its
// successor back to D (issue slots 47 %, tensor cores 26 % busy); 128 elements leave no room for
// a second set of phasors, A tiles or accumulators that would cut it.
// 128 elements, boxcar, 2-7 MHz, 400 x 400 voxels: 34.1 ms with 16 warps that wrote 32-element A
// chunks, kept phasors in registers and searched segment lists; 18.8 ms here.  64 elements,
// Hann, whole band, 151 x 187: 11.9 and 3.6 ms (windows from the table, two bins in flight, the
// band in four ranges).  Fixed 16 KB B stages measured faster than a byte ring (20.3 and 23.7 ms
// at the time), one copy per group and two issuing threads 1 % better than two and one.
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

constexpr int ST_GMAX = 16;                 // element groups of 8: up to 128 elements
constexpr int ST_TT = 4;                    // bins per aperture table (one per slot)
// Bins between exact phasors.  Error against 64 bits and time at 128 elements, 400 x 400, with 32 | 16 | 8:
// 5.4e-7 | 4.3e-7 | 4.3e-7 and 18.70 | 18.84 | 19.09 ms; of nine other frames 4.0e-7 to 6.0e-7 with 32 (the
// kernel before, whose products truncate less often, 3.7e-7 to 5.1e-7), 2.7e-7 to 4.9e-7 with 16.
constexpr int ST_TB = 16;
constexpr int ST_NT = 4;                    // element ranges in flight (aperture tables: 2)
constexpr int ST_NB = 8;                    // B stages at most
constexpr int ST_A = 2 * P5_M * 32;         // a slot's A tile: hi, lo
constexpr int ST_PH = 256;                  // TMEM: D below, the phasors (16 columns a group) from here
constexpr int ST_NARROW = 128;              // D columns of a bin that fits half of D

struct StShared {
  uint2 tab[2][ST_TT][P5_M];         // per bin and voxel: rows tx left, right, rx left, right (8 bits each), n_k
  unsigned rng[ST_NT][ST_TT][4];     // per bin and column: element range lo | (0xffff - hi) << 16
  float2 red[3][P5_M];
  unsigned long long n_active, n_empty, n_exec;
  int item, last;
  int abort_flag;
  uint32_t tmem;
  uint64_t bars[4 + 4 + 2 * ST_NB + 4 + 2 * ST_NT];
};

// shared memory: StShared, A tiles, phasor steps, B stages
__host__ __device__ inline int st_sh_bytes() { return ((int)sizeof(StShared) + 127) / 128 * 128; }
__host__ __device__ inline int st_rho_bytes(int G) { return G * P5_M * 64; }
__host__ __device__ inline int st_b_bytes(int G) { return G * 1024; }        // 64 N at N = 16 G
constexpr int ST_SMEM_MAX = 232448;
__host__ __device__ inline int st_stages(int G) {
  const int n = (ST_SMEM_MAX - st_sh_bytes() - 4 * ST_A - st_rho_bytes(G)) / st_b_bytes(G);
  return n < ST_NB ? n : ST_NB;
}

// ---------------------------------------------------------------------------
// operands
// ---------------------------------------------------------------------------
// B tiles of X' scaled by the power of two sigma, in the order the products read them: [bin][rx
// group of 8][8 rows n][hi, lo][K half][n][8 fp16] (a group's row range is one copy), zero for t or r >= ne.  Row n holds transmit
// element t = 8 (n / 16) + 2 (n % 16 / 4) + n % 2, real part (n % 4 < 2) or imaginary part of Y.
// One block per (4 transmit elements, 32 receive elements, 8 bins): the spectra are read along
// bins into shared memory and written as 32-byte row pairs.
__global__ void __launch_bounds__(256) sa_tc_prep_kernel(const float2* __restrict__ X, int ne, int G, int K,
                                                         const float2* __restrict__ rot,
                                                         const unsigned* __restrict__ maxbits,
                                                         uint4* __restrict__ out) {
  __shared__ float2 tile[4][32][9];
  const int t0 = blockIdx.x * 4, r0 = blockIdx.y * 32, k0 = blockIdx.z * 8;
  for (int i = threadIdx.x; i < 4 * 32 * 8; i += 256) {
    const int kl = i & 7, rl = (i >> 3) & 31, tl = i >> 8;
    const int t = t0 + tl, r = r0 + rl, k = k0 + kl;
    tile[tl][rl][kl] = (t < ne && r < ne && k < K) ? X[((size_t)t * ne + r) * K + k] : make_float2(0.0f, 0.0f);
  }
  __syncthreads();
  const float sigma = tc_scale(*maxbits);
  // thread: transmit element t, receive elements r .. r + 3, bin k
  const int tl = threadIdx.x & 3, rq = (threadIdx.x >> 2) & 7, kl = threadIdx.x >> 5;
  const int t = t0 + tl, r = r0 + 4 * rq, k = k0 + kl;
  if (k >= K || r >= 8 * G) return;
  const float2 c = rot[k];
  unsigned h[2][4], l[2][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 x = tile[tl][4 * rq + i][kl];
    x = make_float2((x.x * c.x - x.y * c.y) * sigma, (x.x * c.y + x.y * c.x) * sigma);
    tc_split_mx(x.x, -x.y, h[0][i], l[0][i]);   // Re Y
    tc_split_mx(x.y, x.x, h[1][i], l[1][i]);    // Im Y
  }
  const int kh = (r >> 2) & 1, n0 = 16 * (t >> 3) + 4 * ((t & 7) >> 1) + (t & 1);
  uint4* o = out + ((size_t)k * G + (r >> 3)) * (size_t)(64 * G);   // a group: 2 G (8 rows) x 2 (hi, lo) x 16
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int n = n0 + 2 * p;
    uint4* q = o + (n >> 3) * 32 + kh * 8 + (n & 7);
    q[0] = make_uint4(h[p][0], h[p][1], h[p][2], h[p][3]);
    q[16] = make_uint4(l[p][0], l[p][1], l[p][2], l[p][3]);
  }
}

// ---------------------------------------------------------------------------
// the beamformer
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned st_range(const unsigned (&r)[4]) { return p5_uni(p5_join(r)); }

// Window values of a group's 8 elements by element pairs; false where every lane's are all 1.
// BOX: the elements of an interval.  Otherwise the table's left and right rows, which hold
// disjoint sides, so that only the group around the voxel's column needs both.
template <bool BOX>
__device__ __forceinline__ bool st_window(const float* wcol, unsigned row_l, unsigned row_r, int ne, int ne_pad, int g,
                                          int emid, float2 (&w)[4]) {
  const int e8 = 8 * g;
  if constexpr (BOX) {
    const int first = (int)row_l == ne ? emid : (int)row_l, last = (int)row_r == ne ? emid - 1 : (int)row_r;
    if (__all_sync(0xffffffffu, first <= e8 && last >= e8 + 7)) return false;
    const unsigned n = (unsigned)max(last - first + 1, 0), o = (unsigned)(e8 - first);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = make_float2(o + 2u * i < n ? 1.0f : 0.0f, o + 2u * i + 1u < n ? 1.0f : 0.0f);
  } else {
    const unsigned row = e8 + 8 <= emid ? row_l : row_r;
    const float4* r = reinterpret_cast<const float4*>(wcol + (row * (unsigned)ne_pad + (unsigned)e8));
    float4 a = __ldg(r), b = __ldg(r + 1);
    if (e8 < emid && e8 + 8 > emid) {
      const float4* v = reinterpret_cast<const float4*>(wcol + (row_l * (unsigned)ne_pad + (unsigned)e8));
      const float4 x = __ldg(v), y = __ldg(v + 1);
      a = make_float4(a.x + x.x, a.y + x.y, a.z + x.z, a.w + x.w);
      b = make_float4(b.x + y.x, b.y + y.y, b.z + y.z, b.w + y.w);
    }
    w[0] = make_float2(a.x, a.y);
    w[1] = make_float2(a.z, a.w);
    w[2] = make_float2(b.x, b.y);
    w[3] = make_float2(b.z, b.w);
  }
  return true;
}

// p <- w p
__device__ __forceinline__ void st_weigh(const float2 (&w)[4], const float (&pv)[16], float (&v)[16]) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const float2 re = __fmul2_rn(w[x], make_float2(pv[4 * x], pv[4 * x + 1]));
    const float2 im = __fmul2_rn(w[x], make_float2(pv[4 * x + 2], pv[4 * x + 3]));
    v[4 * x] = re.x;
    v[4 * x + 1] = re.y;
    v[4 * x + 2] = im.x;
    v[4 * x + 3] = im.y;
  }
}

// the phasor steps of a group, and p <- p rho
__device__ __forceinline__ void st_rho(const float4* rhov, int g, float (&r4)[16]) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const float4 v = rhov[(4 * g + x) * P5_M];
    r4[4 * x] = v.x;
    r4[4 * x + 1] = v.y;
    r4[4 * x + 2] = v.z;
    r4[4 * x + 3] = v.w;
  }
}
__device__ __forceinline__ void st_back(float (&pv)[16], const float (&rv)[16]) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 rr = make_float2(rv[4 * p], rv[4 * p + 1]), ri = make_float2(rv[4 * p + 2], rv[4 * p + 3]);
    const float2 a = make_float2(pv[4 * p], pv[4 * p + 1]), m = make_float2(pv[4 * p + 2], pv[4 * p + 3]);
    const float2 x = __ffma2_rn(p5_neg(m), ri, __fmul2_rn(a, rr));
    const float2 y = __ffma2_rn(m, rr, __fmul2_rn(a, ri));
    pv[4 * p] = x.x;
    pv[4 * p + 1] = x.y;
    pv[4 * p + 2] = y.x;
    pv[4 * p + 3] = y.y;
  }
}

// LAG: up to ST_GMAX / 2 groups, two bins' phasors in tensor memory; BOX: both windows boxcar
template <bool LAG, bool BOX>
__global__ void __launch_bounds__(P5_THREADS, 1)
sa_tc_kernel(const SADev d, const uint4* __restrict__ Bt, const unsigned* __restrict__ maxbits,
             float2* __restrict__ image, float* __restrict__ wtx_out, float* __restrict__ wrx_out) {
  extern __shared__ __align__(128) unsigned char dyn[];
  StShared& sh = *reinterpret_cast<StShared*>(dyn);
  const int G = (d.ne + 7) >> 3;                    // element groups
  const uint32_t NB = (uint32_t)st_stages(G), b_bytes = (uint32_t)st_b_bytes(G);
  unsigned char* abuf = dyn + st_sh_bytes();
  float4* rho = reinterpret_cast<float4*>(abuf + 4 * ST_A);
  const uint32_t abase = smem_u32(abuf), bbase = smem_u32(rho) + (uint32_t)st_rho_bytes(G);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = (int)p5_uni((uint32_t)tid >> 5);
  volatile int* abort_flag = &sh.abort_flag;
  unsigned long long* err = &d.counters[2];
  const uint32_t bar0 = smem_u32(sh.bars);
  auto s_full = [&](uint32_t s) { return bar0 + 8u * s; };
  auto s_empty = [&](uint32_t s) { return bar0 + 8u * (4u + s); };
  auto d_full = [&](uint32_t s) { return bar0 + 8u * (8u + s); };
  auto d_empty = [&](uint32_t s) { return bar0 + 8u * (10u + s); };
  auto r_full = [&](uint32_t s) { return bar0 + 8u * (12u + s); };
  auto r_empty = [&](uint32_t s) { return bar0 + 8u * (12u + ST_NT + s); };
  auto b_full = [&](uint32_t s) { return bar0 + 8u * (12u + 2 * ST_NT + s); };
  auto b_empty = [&](uint32_t s) { return bar0 + 8u * (12u + 2 * ST_NT + ST_NB + s); };

  if (tid == 0) {
    for (int s = 0; s < 4; ++s) {
      mbar_init(s_full(s), 4);
      mbar_init(s_empty(s), 2);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(d_full(s), 2);
      mbar_init(d_empty(s), P5_CW);
    }
    for (int s = 0; s < ST_NT; ++s) {
      mbar_init(r_full(s), P5_CW);
      mbar_init(r_empty(s), 4);
    }
    for (int s = 0; s < ST_NB; ++s) {
      mbar_init(b_full(s), 1);
      mbar_init(b_empty(s), 2);
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
  const int ntx = (d.wt_nc + TILE_X - 1) / TILE_X, ntz = (d.nz + TILE_Z - 1) / TILE_Z;
  const int n_items = ntx * ntz * d.split;
  uint32_t nd = 0;                 // bins with products so far
  uint32_t ns = 0;                 // aperture tables so far
  const uint32_t lead = lane == 0 ? 1u : 0u;

  if (warp >= P5_CW) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P5_REGS_I));
    const int role = warp - P5_CW;       // 0, 1: products of the first, second half of the transmit elements; 2, 3: copies
    uint32_t st = 0, st_ph = 0;          // B stage and its phase
    uint32_t turn = 0;                   // the copying threads take groups in turn
    uint32_t a_ph = 0;                   // phases of the slots' A tiles (bit per slot)
    bool prev_wide = false;
    for (;;) {
      __syncthreads();
      const int item = sh.item;
      if (item < 0) break;
      const int part = item % d.split;
      const int kt = d.k_ub - part * d.split_bins;
      const int nb = min(d.split_bins, kt - d.k_lb + 1);
      if (lane == 0) {
        unsigned long long exec = 0;
        bool ok = true;
        for (int b = 0; b < nb && ok; ++b) {
          const uint32_t ri = ns % ST_NT;
          if (b % ST_TT == 0) ok = p5_wait(r_full(ri), (ns / ST_NT) & 1u, 0u, abort_flag, err);
          const unsigned r = p5_join(sh.rng[ri][b % ST_TT]);
          // the last use of this table's ranges
          if (b % ST_TT == ST_TT - 1 || b == nb - 1) {
            mbar_arrive(r_empty(ri));
            ++ns;
          }
          if (r == 0xffffffffu) continue;
          const int g_lo = (int)(r & 0xffffu) >> 3, g_hi = (0xffff - (int)(r >> 16)) >> 3;
          const int ng = g_hi - g_lo + 1;
          if (role >= 2) {
            // per group: rows 16 g_lo .. 16 g_hi + 15
            const uint4* src = Bt + ((size_t)(kt - b - d.k_lb) * G + g_lo) * (size_t)(64 * G) + 64 * g_lo;
            for (int g = g_lo; g <= g_hi; ++g, src += 64 * G) {
              if (turn == ((uint32_t)role & 1u)) {
                ok = p5_wait(b_empty(st), st_ph ^ 1u, 0u, abort_flag, err);
                if (!ok) break;
                mbar_expect_tx(b_full(st), 1024u * (uint32_t)ng);
                bulk_load(bbase + st * b_bytes, src, 1024u * (uint32_t)ng, b_full(st));
              }
              turn ^= 1u;
              if (++st == NB) {
                st = 0;
                st_ph ^= 1u;
              }
            }
            if (role == 2) exec += (unsigned long long)P5_M * 64 * ng * ng;
          } else {
            // D: a half in turn for narrow bins; the bin before it must have been read where the two overlap
            const bool wide = 16 * ng > ST_NARROW;
            const uint32_t last = (wide || prev_wide) ? 1u : 2u;   // the bin read before this one writes: nd - last
            prev_wide = wide;
            uint32_t ask_a = p5_ask(s_full((uint32_t)g_lo & 3u), (a_ph >> (g_lo & 3)) & 1u);
            uint32_t ask_b = p5_ask(b_full(st), st_ph);
            // this thread's rows
            const int n0 = (ng + 1) >> 1;
            const uint32_t row0 = role ? (uint32_t)n0 : 0u, n = 16u * (uint32_t)(role ? ng - n0 : n0);
            const uint32_t dcol = tmem + (wide ? 0u : (nd & 1u) * ST_NARROW) + 16u * row0;
            const uint32_t idesc = idesc_f16(P5_M, (int)n);
            constexpr uint64_t HA = smem_desc_plain_hi(256), HB = smem_desc_plain_hi(512);
            const uint32_t b0 = (uint32_t)smem_desc_plain(bbase, 128, 512) + 64u * row0;
            const uint32_t a0 = (uint32_t)smem_desc_plain(abase, 128, 256);
            if (nd >= last)
              ok = p5_wait(d_empty((nd - last) & 1u), ((nd - last) >> 1) & 1u, 0u, abort_flag, err);
            uint32_t accum = 0u;
            for (int g = g_lo; g <= g_hi; ++g) {
              const uint32_t sl = (uint32_t)g & 3u;
              p5_wait(b_full(st), st_ph, ask_b, abort_flag, err);
              p5_wait(s_full(sl), (a_ph >> sl) & 1u, ask_a, abort_flag, err);
              const uint32_t bd = b0 + st * (b_bytes >> 4), ah = a0 + sl * (ST_A >> 4);
              const uint32_t be = b_empty(st), nx = (sl + 1u) & 3u;
              a_ph ^= 1u << sl;
              if (++st == NB) {
                st = 0;
                st_ph ^= 1u;
              }
              fence_after_sync();
              if (n) {
                // the small cross products first, so that fewer steps round a full-size sum
                mma_f16(dcol, HA | (uint64_t)ah, HB | (uint64_t)(bd + 16u), idesc, accum);
                mma_f16(dcol, HA | (uint64_t)(ah + (ST_A >> 5)), HB | (uint64_t)bd, idesc, 1u);
                mma_f16(dcol, HA | (uint64_t)ah, HB | (uint64_t)bd, idesc, 1u);
              }
              accum = 1u;
              mma_commit(s_empty(sl));
              mma_commit(be);
              ask_b = p5_ask(b_full(st), st_ph);
              ask_a = p5_ask(s_full(nx), (a_ph >> nx) & 1u);
            }
            mma_commit(d_full(nd & 1u));
            ok = ok && !*abort_flag;
          }
          ++nd;
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
    float4* us = d.u_scr + (size_t)blockIdx.x * (size_t)(P5_M * 4 * ST_GMAX) + vb;
    const uint32_t sf = s_full((uint32_t)slot), se = s_empty((uint32_t)slot);
    unsigned char* arow = abuf + slot * ST_A + (vb >> 3) * 256 + (vb & 7) * 16;
    const float4* rhov = rho + vb;
    const float inv_sigma = 1.0f / tc_scale(*maxbits);
    const int ne = d.ne;
    uint32_t a_ph = 0;                                // phase of the slot's A tile
    for (;;) {
      if (tid == 0) {
        const int t = *abort_flag ? n_items : (int)atomicAdd(&d.counters[3], 1ull);
        sh.item = t < n_items ? t : -1;
      }
      __syncthreads();
      const int item = sh.item;
      if (item < 0) break;
      const int tile = item / d.split, part = item - tile * d.split;
      int tx, tz;
      tile_coords(tile, ntx, ntz, tx, tz);
      const int cw = tx * TILE_X + q;                       // column within the window tables' slab
      const int j = tz * TILE_Z + lane;
      const bool valid = (cw < d.wt_nc) && (j < d.nz);
      const int cc = min(cw, d.wt_nc - 1), ic = d.wt_c0 + cc, jc = min(j, d.nz - 1);
      const size_t vox = (size_t)ic * d.nz + jc;
      const int kt = d.k_ub - part * d.split_bins;
      const int nb = min(d.split_bins, kt - d.k_lb + 1);
      const int emid = (int)p5_uni((uint32_t)d.col_emid[ic]);
      const float* wt_col = d.w_tab[0] + (size_t)cc * (size_t)(ne + 1) * d.ne_pad;
      const float* wr_col = d.w_tab[1] + (size_t)cc * (size_t)(ne + 1) * d.ne_pad;
      unsigned c_act = 0, c_emp = 0;
      // Aperture table of stretch s: per bin and voxel the rows of the window tables and n_k, per bin and column
      // the element range; this warp takes its column's bin `slot`.
      auto build = [&](int s) {
        const uint32_t tbuf = (ns + (uint32_t)s) & 1u, ri = (ns + (uint32_t)s) % ST_NT;
        const uint32_t rp = (((ns + (uint32_t)s) / ST_NT) & 1u) ^ 1u;
        const uint32_t ask = p5_ask(r_empty(ri), rp);
        const dfl xp = d.col_p[ic], zp = d.row_p[jc];
        const int b = s * ST_TT + slot;
        const int kk = max(kt - b - d.k_lb, 0);
        int tlb, tub, rlb, rub;
        p5_aperture(xp, zp, d.gtx[kk], ne, tlb, tub);
        rlb = tlb;
        rub = tub;
        if (!d.Xs) p5_aperture(xp, zp, d.grx[kk], ne, rlb, rub);
        // a side without elements takes the zero row
        const int t_l = tlb < emid ? tlb : ne, t_r = tub >= emid ? tub : ne;
        const int r_l = rlb < emid ? rlb : ne, r_r = rub >= emid ? rub : ne;
        const float* s0 = d.w_sum[0] + (size_t)cc * (size_t)(ne + 1);
        const float* s1 = d.w_sum[1] + (size_t)cc * (size_t)(ne + 1);
        const float Wt = __ldg(s0 + t_l) + __ldg(s0 + t_r);
        const float Wr = d.Xs ? Wt : __ldg(s1 + r_l) + __ldg(s1 + r_r);
        const float it = Wt > 0.0f ? (d.norm_tx ? __frcp_rn(Wt) : 1.0f) : 0.0f;
        const float ir = Wr > 0.0f ? (d.norm_rx ? __frcp_rn(Wr) : 1.0f) : 0.0f;
        const int t_n = max(tub, emid - 1) - min(tlb, emid) + 1, r_n = max(rub, emid - 1) - min(rlb, emid) + 1;
        const bool in = valid && b < nb;
        const bool act = in && Wt > 0.0f && Wr > 0.0f && t_n > 0 && r_n > 0;
        if (in) {
          if (act) c_act += (unsigned)(t_n * r_n); else ++c_emp;
          if (kk == d.K - 1) {
            if (wtx_out) wtx_out[vox] = Wt;
            if (wrx_out) wrx_out[vox] = Wr;
          }
        }
        const int lo = act ? min(min(tlb, rlb), emid) : 0xffff, hi = act ? max(max(tub, rub), emid - 1) : -1;
        p5_wait(r_empty(ri), rp, ask, abort_flag, err);
        sh.tab[tbuf][slot][vb] = make_uint2((unsigned)t_l | (unsigned)t_r << 8 | (unsigned)r_l << 16 | (unsigned)r_r << 24,
                                            __float_as_uint(act ? it * ir : 0.0f));
        const unsigned mn = __reduce_min_sync(0xffffffffu, (unsigned)lo);
        const int mx = __reduce_max_sync(0xffffffffu, hi);
        if (lead) sh.rng[ri][slot][q] = mx < 0 ? 0xffffffffu : (mn | ((unsigned)(0xffff - mx) << 16));
        __syncwarp();
        mbar_arrive_if(lead, r_full(ri));
      };
      build(0);
      // phasor steps rho = e^{2 pi i u} into shared memory, by element pairs {Re, Re, Im, Im}; the
      // delays u to scratch for the exact anchors
#pragma unroll 1
      for (int g = slot; g < G; g += 4) {
#pragma unroll
        for (int j2 = 0; j2 < 4; ++j2) {
          dfl u[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int e = min(8 * g + 2 * j2 + h, ne - 1);
            u[h] = df_sqrt(df_add(df_sqr(df_sub(d.el_u[e], d.col_u[ic])), d.row_u2[jc]));
          }
          float2 r, m;
          p5_cis2(1.0f, make_float2(u[0].x, u[1].x), make_float2(u[0].y, u[1].y), r, m);
          rho[(4 * g + j2) * P5_M + vb] = make_float4(r.x, r.y, m.x, m.y);
          us[(size_t)(4 * g + j2) * P5_M] = make_float4(u[0].x, u[1].x, u[0].y, u[1].y);
        }
      }
      float2 acc = make_float2(0.0f, 0.0f), comp = make_float2(0.0f, 0.0f);
      unsigned live = 0u;                 // groups whose phasors belong to the previous bin
      // the bin whose products are under way: its groups, transmit rows and n_k
      unsigned p_mask = 0u, p_rows = 0u;
      int p_glo = 0;
      float p_nrm = 0.0f;
      bool p_wide = false;
#pragma unroll 1
      for (int b = 0; b <= nb; ++b) {
        unsigned mask = 0u;
        uint2 te = make_uint2(0u, 0u);
        int g_lo = 0, g_hi = -1;
        if (b < nb) {
          const int s = b / ST_TT, t = b % ST_TT;
          if (t == 0) {
            // table s is complete, and no warp reads the one before it any more
            p5_bar();
            if (b + ST_TT < nb) build(s + 1);
          }
          const unsigned r = st_range(sh.rng[(ns + (uint32_t)s) % ST_NT][t]);
          if (b % ST_TB == 0) live = 0u;  // exact phasors
          // Without an aperture in the tile the bin has no groups, and the one under way is
          // finished below with its own phasors: the next one that has groups need not be its
          // neighbour, so its head's phasors stepped back would be another bin's.
          if (r != 0xffffffffu) {
            te = sh.tab[(ns + (uint32_t)s) & 1u][t][vb];
            g_lo = (int)(r & 0xffffu) >> 3;
            g_hi = (0xffff - (int)(r >> 16)) >> 3;
            mask = (2u << g_hi) - (1u << g_lo);
          }
        }
        const bool wide = 16 * (g_hi - g_lo + 1) > ST_NARROW;
        const unsigned exact = mask & ~live;
        const uint32_t cur = nd, prv = nd - 1u;          // counts of this bin and of the one under way
        const uint32_t ph_n = tl + ST_PH + (LAG ? (cur & 1u) * 128u : 0u);
        const uint32_t ph_o = tl + ST_PH + (LAG ? (prv & 1u) * 128u : 0u);
        const uint32_t td = tl + (p_wide ? 0u : (prv & 1u) * ST_NARROW);
        float2 sx = make_float2(0.0f, 0.0f), sy = make_float2(0.0f, 0.0f);
        const unsigned ms = mask & (0x1111u << slot);
        const unsigned head = LAG ? ms : ms & (0u - ms);
#pragma unroll 1
        for (int pass = 0; pass < (LAG ? 2 : 3); ++pass) {
          // A of the slot's first group (LAG: of all), the previous bin's dot products, the other groups' A
          const unsigned dots = pass == 1 ? p_mask : 0u;
          const unsigned gens = pass == 0 ? head : (pass == 2 ? ms & ~head : 0u);
          if (dots) {
            p5_wait(d_full(prv & 1u), (prv >> 1) & 1u, 0u, abort_flag, err);
            fence_after_sync();
          }
          const unsigned mine = (dots | gens) & (0x1111u << slot);
#pragma unroll 1
          for (unsigned m = mine; m; m &= m - 1u) {
            const int g = __ffs(m) - 1;
            if ((dots >> g) & 1u) {
              float y[16], p[16];
              tmem_ld16_nowait(td + (uint32_t)(16 * (g - p_glo)), y);
              tmem_ld16_nowait(ph_o + (uint32_t)(16 * g), p);
              float2 w[4];
              const bool weigh = st_window<BOX>(wt_col, p_rows & 0xffu, (p_rows >> 8) & 0xffu, ne, d.ne_pad, g, emid, w);
              tmem_wait_ld();
              if (!LAG && ((head >> g) & 1u)) {   // its phasors are this bin's

                float r4[16];
                st_rho(rhov, g, r4);
                st_back(p, r4);
              }
              if (weigh) st_weigh(w, p, p);
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const float2 ar = make_float2(p[4 * x], p[4 * x + 1]), ai = make_float2(p[4 * x + 2], p[4 * x + 3]);
                const float2 yr = make_float2(y[4 * x], y[4 * x + 1]), yi = make_float2(y[4 * x + 2], y[4 * x + 3]);
                sx = __ffma2_rn(ar, yr, __ffma2_rn(p5_neg(ai), yi, sx));
                sy = __ffma2_rn(ar, yi, __ffma2_rn(ai, yr, sy));
              }
            }
            if ((gens >> g) & 1u) {
              const bool fresh = (exact >> g) & 1u;
              float p[16];
              if (!fresh) tmem_ld16_nowait(ph_o + (uint32_t)(16 * g), p);
              const uint32_t ask_a = p5_ask(se, a_ph ^ 1u);
              float2 w[4];
              const bool weigh = st_window<BOX>(wr_col, (te.x >> 16) & 0xffu, te.x >> 24, ne, d.ne_pad, g, emid, w);
              if (fresh) {
                const float kf = (float)(kt - b);
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
                float r4[16];
                st_rho(rhov, g, r4);
                tmem_wait_ld();
                p5_rotate(p, r4);
              }
              tmem_st16(ph_n + (uint32_t)(16 * g), p);
              uint32_t h[8], l[8];
              if (weigh) st_weigh(w, p, p);
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                tc_split_mx(p[4 * x], p[4 * x + 2], h[2 * x], l[2 * x]);
                tc_split_mx(p[4 * x + 1], p[4 * x + 3], h[2 * x + 1], l[2 * x + 1]);
              }
              // the slot's A tile is free once the products that read it last are complete
              p5_wait(se, a_ph ^ 1u, ask_a, abort_flag, err);
              uint4* o = reinterpret_cast<uint4*>(arow);
              o[0] = make_uint4(h[0], h[1], h[2], h[3]);
              o[8] = make_uint4(h[4], h[5], h[6], h[7]);
              o[ST_A / 32] = make_uint4(l[0], l[1], l[2], l[3]);
              o[ST_A / 32 + 8] = make_uint4(l[4], l[5], l[6], l[7]);
              fence_proxy_async_smem();
              __syncwarp();
              mbar_arrive_if(lead, sf);
              a_ph ^= 1u;
              tmem_wait_st();
            }
          }
          if (dots) {
            fence_before_sync();
            __syncwarp();
            mbar_arrive_if(lead, d_empty(prv & 1u));
          }
        }
        // n_k Y of the previous bin into the voxel, compensated
        if (p_mask) {
          const float yx = p_nrm * (sx.x + sx.y) - comp.x, nx = acc.x + yx;
          comp.x = (nx - acc.x) - yx;
          acc.x = nx;
          const float yy = p_nrm * (sy.x + sy.y) - comp.y, ny = acc.y + yy;
          comp.y = (ny - acc.y) - yy;
          acc.y = ny;
        }
        live = mask;
        p_mask = mask;
        p_rows = te.x;
        p_nrm = __uint_as_float(te.y);
        p_glo = g_lo;
        p_wide = wide;
        if (mask) ++nd;
      }
      ns += (uint32_t)((nb + ST_TT - 1) / ST_TT);
      {
        const unsigned na = __reduce_add_sync(0xffffffffu, c_act), nm = __reduce_add_sync(0xffffffffu, c_emp);
        if (lead) {
          atomicAdd(&sh.n_active, (unsigned long long)na);
          atomicAdd(&sh.n_empty, (unsigned long long)nm);
        }
      }
      const size_t nvox = (size_t)d.nx * d.nz;
      float2* out = d.split > 1 ? d.part + (size_t)part * nvox : image;
      if (slot > 0) sh.red[slot - 1][vb] = acc;
      p5_bar();
      if (slot == 0 && valid) {
        float2 o = acc;
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          o.x += sh.red[t][vb].x;
          o.y += sh.red[t][vb].y;
        }
        const float f = d.scale * inv_sigma;
        out[vox] = make_float2(o.x * f, o.y * f);
      }
      if (d.split > 1) {
        // the last of the tile's bin ranges to finish adds them up, in order
        __threadfence();
        p5_bar();
        if (tid == 0)
          sh.last = atomicAdd(&d.tile_cnt[(size_t)(d.wt_c0 / TILE_X) * ntz + tile], 1u) == (unsigned)(d.split - 1);
        p5_bar();
        if (sh.last && slot == 0 && valid) {
          __threadfence();
          float2 s = make_float2(0.0f, 0.0f);
          for (int p = 0; p < d.split; ++p) {
            const float2 v = __ldcg(d.part + (size_t)p * nvox + vox);
            s.x += v.x;
            s.y += v.y;
          }
          image[vox] = s;
        }
      }
      __syncthreads();
    }
  }
  // after a timeout, give the copies and products in flight time to land before the tensor
  // memory is freed (they take microseconds)
  if (tid == 0) {
    atomicAdd(&d.counters[0], sh.n_active);
    atomicAdd(&d.counters[1], sh.n_empty);
    atomicAdd(&d.counters[4], sh.n_exec);
    if (*abort_flag) {
      const unsigned long long t0 = global_ns();
      while (global_ns() - t0 < 20000000ull) {
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

typedef void (*st_kernel_t)(const SADev, const uint4*, const unsigned*, float2*, float*, float*);
st_kernel_t st_pick(const SADev& d) {
  const bool lag = (d.ne + 7) / 8 <= ST_GMAX / 2, box = d.wtx_id == 0 && d.wrx_id == 0;
  return lag ? (box ? sa_tc_kernel<true, true> : sa_tc_kernel<true, false>)
             : (box ? sa_tc_kernel<false, true> : sa_tc_kernel<false, false>);
}
int st_smem(int G) { return st_sh_bytes() + 4 * ST_A + st_rho_bytes(G) + st_stages(G) * st_b_bytes(G); }

int st_sms() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm > 0 ? nsm : 1;
}

}  // namespace

bool sa_tc_supported(const SADev& d) { return d.ne >= 1 && d.ne <= 8 * ST_GMAX && d.last_bin_only == 0; }

size_t sa_tc_bytes(int ne, int K) {
  const size_t G = (size_t)((ne + 7) / 8);
  return (size_t)K * G * G * 1024;
}

size_t sa_tc_scratch_bytes(const SADev& d) {
  return (size_t)sa_tc_grid(d) * P5_M * 4 * ST_GMAX * sizeof(float4);
}

// Bin ranges per tile.  A tile is one block's work, so a launch of few tiles would leave SMs idle
// in its last wave: its band is split into ranges of at least 64 bins (each pays the tile's
// set-up) until there are about six items per SM.
void sa_tc_pick_split(SADev& d) {
  const int tiles = ((d.wt_nc + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z);
  int s = (6 * st_sms() + tiles - 1) / tiles;
  s = std::max(1, std::min(s, d.K / 64));
  d.split_bins = ((d.K + s - 1) / s + 31) / 32 * 32;
  d.split = (d.K + d.split_bins - 1) / d.split_bins;
}

cudaError_t sa_tc_setup(SaTc& t, const SADev& d, void* planes, unsigned* maxbits, const float2* rot) {
  t.planes = planes;
  t.maxbits = maxbits;
  t.rot = rot;
  // the compute warps' register share needs the full allocation at launch
  cudaFuncAttributes a;
  const void* fn = (const void*)st_pick(d);
  cudaError_t e = cudaFuncGetAttributes(&a, fn);
  if (e != cudaSuccess) return e;
  if (a.numRegs != P5_REGS) return cudaErrorInvalidConfiguration;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM_MAX);
}

int sa_tc_grid(const SADev& d) {
  const int tiles = ((d.wt_nc + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z) * d.split;
  return std::max(1, std::min(tiles, st_sms()));
}

// one window table per side for the columns wt_c0 .. wt_c0 + wt_nc - 1
cudaError_t launch_sa_tc_window(const SADev& d, cudaStream_t s) {
  PWDev w{};
  w.ne = d.ne;
  w.wt_rows = d.ne;
  w.wt_w = d.ne_pad;
  w.wt_c0 = d.wt_c0;
  w.wt_nc = d.wt_nc;
  w.col_m = d.col_m;
  w.col_emid = d.col_emid;
  w.el_m = d.el_m;
  w.el_lb = d.el_lb;
  w.el_ub = d.el_ub;
  w.pitch_f = d.pitch_f;
  for (int i = 0; i < (d.w_tab[0] == d.w_tab[1] ? 1 : 2); ++i) {
    w.window_id = i ? d.wrx_id : d.wtx_id;
    w.window_par = i ? d.wrx_par : d.wtx_par;
    const cudaError_t e = launch_pw_tc_window(w, const_cast<float*>(d.w_tab[i]), const_cast<float*>(d.w_sum[i]), s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_sa_tc(const SADev& d0, const SaTc& t, float2* image, float* wtx, float* wrx, cudaStream_t s) {
  cudaError_t e = launch_absmax((const float*)d0.X, (size_t)d0.ne * d0.ne * d0.K * 2, t.maxbits, s);
  if (e != cudaSuccess) return e;
  const int G = (d0.ne + 7) / 8;
  const dim3 pg(2 * G, (G + 3) / 4, (d0.K + 7) / 8);
  sa_tc_prep_kernel<<<pg, 256, 0, s>>>(d0.X, d0.ne, G, d0.K, t.rot, t.maxbits, (uint4*)t.planes);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  SADev d = d0;
  if (d.split > 1) {
    const size_t tiles = (size_t)((d.nx + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z);
    if ((e = cudaMemsetAsync(d.tile_cnt, 0, tiles * sizeof(unsigned), s)) != cudaSuccess) return e;
  }
  for (int c0 = 0; c0 < d0.nx; c0 += d0.wt_nc) {
    d.wt_c0 = c0;
    d.wt_nc = std::min(d0.wt_nc, d0.nx - c0);
    // window tables that do not hold all columns are refilled for each slab of them
    if (d0.wt_nc < d0.nx && (e = launch_sa_tc_window(d, s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(d.counters + 3, 0, sizeof(unsigned long long), s)) != cudaSuccess) return e;
    st_pick(d)<<<sa_tc_grid(d), P5_THREADS, st_smem(G), s>>>(d, (const uint4*)t.planes, t.maxbits, image, wtx, wrx);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace fnum
