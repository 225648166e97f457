// The plane-wave beamformer for one or two angles, in FP32 with the window table (variant 9).
//
// A voxel's image is I(v) = s sum_a sum_e sum_k n_k w_k(v, e) X_k(e, a) z^k, z = e^{2 pi i (u_e + u_a)}:
// the terms of fnum_pw_tc.cu's product, where one or two angles fill 2 or 4 of the 16 columns that
// a tensor-core product has at least.  Here each (voxel, element, angle) runs a Horner recurrence
// over the bins from the top down, A <- A z + n_k w_k X_k, 4 FMA and the two products with the
// weight a term, and stretches of 32 (or 16) bins are added with the exact phase of their last bin.
//
// A block serves a tile of 128 voxels (4 columns x 32 rows, a voxel per lane) with two element
// slots of 4 warps and, for a frame of few tiles, a range of its bins.  Per chunk of bins the
// threads form the window table's rows and n_k of every (bin, voxel) and the chunk's spectra are
// copied to shared memory as element pairs {Re, Re, Im, Im}, the operands of packed FP32x2
// instructions.  Then every warp takes its slot's groups of 8 elements within its column's
// apertures, with the group's recurrences in registers.  Where F is the same at all bins of a chunk
// (constant, or at its bound) so are the apertures: the chunk then has one row per voxel and
// its weights multiply the sums over the bins, not each term.
//
// What bounds it: issue slots and the FMA pipe (54 % busy each where F varies) at four warps a
// scheduler: about 100 instructions per 8 elements and bin with chunks of 32 bins, of which 41 are
// the recurrence, and 85 with 64; chunks of one F need half of those.  One angle, 128 elements,
// 256 x 256, F partly at its upper bound: 4.55 ms with the segment-list kernel (its weights change
// at nearly every bin, and a tile's boundaries are resolved serially), 4.13 ms on the tensor cores,
// 2.05 ms here with chunks of 32 bins, 1.93 ms with 64 and 1.67 ms with one weight for chunks of one F.
// Constant F 1.5, 128 elements, 512 x 512, one | two angles: 2.23 | 3.72 ms with the segment-list
// kernel (one segment a voxel), 2.71 | 4.32 ms with a weight a term, 1.43 | 2.75 ms with one a chunk.
// Two blocks an SM: three spill (2.19 ms).  One angle, 64 elements, 48 x 57: 1005, 185 and 82 us
// (the band in ranges of 16 bins).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "fnum_tc_beam.cuh"

namespace fnum {

namespace {

using namespace tcx;

constexpr int FW_THREADS = 256;
constexpr int FW_BC = 64;          // bins of a chunk: a group's delays and steps are formed once per chunk
__host__ __device__ constexpr int fw_ep(int na) { return 32 / na; }   // element pairs whose spectra shared memory holds

struct FwShared {
  uint2 tab[FW_BC][P5_M];          // per bin and voxel: row left | row right << 16, n_k
  unsigned lo[TILE_X];             // the chunk's elements by column
  int hi[TILE_X];
  float2 red[2][P5_M];
  unsigned long long n_active, n_empty, n_exec;
  int last;
};
constexpr int fw_smem(int na) { return ((int)sizeof(FwShared) + 127) / 128 * 128 + FW_BC * fw_ep(na) * na * 16; }
constexpr int FW_BLOCKS = 2;             // resident per SM
constexpr int FW_SMEM_ONE = 120 * 1024;  // more than half of an SM's shared memory: one resident block
static_assert(fw_smem(1) <= FW_SMEM_ONE && fw_smem(2) <= FW_SMEM_ONE, "shared memory");

// spectra as element pairs [bin][pair][angle] {Re, Re, Im, Im}, zero beyond the last element and for
// values that are not finite; and no bin range of a tile is done yet
__global__ void __launch_bounds__(256) fw_pairs_kernel(const PWDev d, float4* __restrict__ out) {
  const int np = d.ne_pad >> 1;
  const size_t n = (size_t)d.K * np * d.na;
  const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  if (d.split > 1) {
    const size_t n_tiles = (size_t)((d.nx + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z);
    for (size_t t = t0; t < n_tiles; t += step) d.tile_cnt[t] = 0u;
  }
  for (size_t i = t0; i < n; i += step) {
    const int a = (int)(i % d.na);
    const size_t r = i / d.na;
    const int p = (int)(r % np), kk = (int)(r / np);
    float2 x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 2 * p + h;
      x[h] = e < d.ne ? d.X[((size_t)e * d.K + kk) * d.x_na + d.x_a0 + a] : make_float2(0.0f, 0.0f);
      if (!p5_finite(x[h])) {
        x[h] = make_float2(0.0f, 0.0f);
        atomicOr(&d.counters[2], FLAG_NONFINITE);
      }
    }
    out[i] = make_float4(x[0].x, x[1].x, x[0].y, x[1].y);
  }
}

template <int NA, bool STACK>
__global__ void __launch_bounds__(FW_THREADS, FW_BLOCKS)
pw_few_kernel(const PWDev d, float2* __restrict__ image, float* __restrict__ weights) {
  extern __shared__ __align__(128) unsigned char dyn[];
  FwShared& sh = *reinterpret_cast<FwShared*>(dyn);
  float4* xs = reinterpret_cast<float4*>(dyn + (sizeof(FwShared) + 127) / 128 * 128);
  const float4* Xp = reinterpret_cast<const float4*>(d.tc_B);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = warp & 3, slot = warp >> 2, vb = 32 * q + lane;
  const int ntx = (d.wt_nc + TILE_X - 1) / TILE_X, ntz = (d.nz + TILE_Z - 1) / TILE_Z;
  const int item = blockIdx.x, tile = item / d.split, part = item - tile * d.split;
  int tx, tz;
  tile_coords(tile, ntx, ntz, tx, tz);
  const int cw = tx * TILE_X + q, j = tz * TILE_Z + lane;
  const bool valid = cw < d.wt_nc && j < d.nz;
  const int cc = min(cw, d.wt_nc - 1), ic = d.wt_c0 + cc, jc = min(j, d.nz - 1);
  const int ne = d.ne, np = d.ne_pad >> 1;
  const int kt = d.k_ub - part * d.split_bins;
  const int nb = min(d.split_bins, kt - d.k_lb + 1);
  const int emid = d.col_emid[ic];
  const dfl xp = d.col_p[ic], zp = d.row_p[jc], xu = d.col_u[ic], zu2 = d.row_u2[jc];
  dfl ua[NA];
#pragma unroll
  for (int a = 0; a < NA; ++a) ua[a] = df_add(d.tx_ax[(size_t)a * d.nx + ic], d.tx_az[(size_t)a * d.nz + jc]);
  const P5Window wt = p5_window(d, cc, (int)p5_uni((uint32_t)d.col_e0[ic]));
  const size_t nvox = (size_t)d.nx * d.nz, vox = (size_t)ic * d.nz + jc;
  const int tb = (d.tc_tb > 0 && d.tc_tb < 32) ? d.tc_tb : 32;   // bins between exact phases
  unsigned c_act = 0, c_emp = 0;
  unsigned long long c_exec = 0;
  constexpr int NO = STACK ? NA : 1, FW_EP = fw_ep(NA);
  float2 acc[NO], comp[NO];
#pragma unroll
  for (int o = 0; o < NO; ++o) acc[o] = comp[o] = make_float2(0.0f, 0.0f);
  if (tid == 0) sh.n_active = sh.n_empty = sh.n_exec = 0ull;

  for (int b0 = 0; b0 < nb; b0 += FW_BC) {
    const int n = min(FW_BC, nb - b0), k_hi = kt - b0;
    __syncthreads();                 // the previous chunk's tables are consumed
    if (tid < TILE_X) {
      sh.lo[tid] = 0xffffu;
      sh.hi[tid] = -1;
    }
    // one F for all the chunk's bins: one aperture and one weight per voxel and element
    bool same = true;
    if (tid < n) {
      const dfl g0 = d.g[k_hi - d.k_lb], g1 = d.g[k_hi - tid - d.k_lb];
      same = g0.x == g1.x && g0.y == g1.y;
    }
    const bool steady = __syncthreads_and(same);
    {
      unsigned lo = 0xffffu;
      int hi = -1;
      const int nt = steady ? 1 : n;             // table entries, each of n / nt bins
      for (int b = slot; b < nt; b += 2) {
        const int kk = k_hi - b - d.k_lb;
        int ilb, iub;
        p5_aperture(xp, zp, d.g[kk], ne, ilb, iub);
        // a side without elements takes the zero row
        const int row_l = ilb < emid ? ilb : wt.zero, row_r = iub >= emid ? iub : wt.zero;
        const float W = __ldg(wt.sum + row_l) + __ldg(wt.sum + row_r);
        const int a = min(ilb, emid), z = max(iub, emid - 1);
        const bool act = valid && W > 0.0f && a <= z;
        if (valid) {
          const unsigned m = steady ? (unsigned)n : 1u;
          if (act) c_act += m * (unsigned)(z - a + 1); else c_emp += m;
          if (kk == d.K - 1 && weights) weights[vox] = W;
        }
        sh.tab[b][vb] = make_uint2((unsigned)row_l | (unsigned)row_r << 16,
                                   __float_as_uint(act ? (d.norm ? __frcp_rn(W) : 1.0f) : 0.0f));
        if (act) {
          lo = min(lo, (unsigned)a);
          hi = max(hi, z);
        }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lane == 0 && hi >= 0) {
        atomicMin(&sh.lo[q], lo);
        atomicMax(&sh.hi[q], hi);
      }
    }
    __syncthreads();
    const int g_lo = sh.hi[q] < 0 ? 1 : (int)sh.lo[q] >> 3, g_hi = sh.hi[q] < 0 ? 0 : sh.hi[q] >> 3;
    unsigned u_lo = 0xffffu;
    int u_hi = -1;
#pragma unroll
    for (int c = 0; c < TILE_X; ++c) {
      u_lo = min(u_lo, sh.lo[c]);
      u_hi = max(u_hi, sh.hi[c]);
    }
    if (u_hi < 0) continue;
    // passes of FW_EP element pairs from the first group of the tile
    for (int p0 = (int)(u_lo >> 3) * 4; 2 * p0 <= u_hi; p0 += FW_EP) {
      const int pn = min(FW_EP, (u_hi >> 3) * 4 + 4 - p0);      // pairs of the pass
      if (p0 != (int)(u_lo >> 3) * 4) __syncthreads();           // the previous pass is consumed
      for (int i = tid; i < n * pn * NA; i += FW_THREADS) {
        const int b = i / (pn * NA), r = i - b * (pn * NA);
        xs[b * (FW_EP * NA) + r] = __ldg(Xp + ((size_t)(k_hi - b - d.k_lb) * np + p0) * NA + r);
      }
      __syncthreads();
      const int first = max(g_lo, p0 >> 2), last = min(g_hi, (p0 + pn - 1) >> 2);
      float2 sum[NO];
#pragma unroll
      for (int o = 0; o < NO; ++o) sum[o] = make_float2(0.0f, 0.0f);
#pragma unroll 1
      for (int g = first + ((slot - first) & 1); g <= last; g += 2) {
        float2 zr[NA][4], zi[NA][4], zn[NA][4], Ar[NA][4], Ai[NA][4];   // zn = -zi
        float2 uh[4], ul[4];           // receive delays of the group's element pairs
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          dfl u[2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            u[h] = df_sqrt(df_add(df_sqr(df_sub(d.el_u[min(8 * g + 2 * x + h, ne - 1)], xu)), zu2));
          if constexpr (NA == 1) {   // with the transmit delay
            u[0] = df_add(u[0], ua[0]);
            u[1] = df_add(u[1], ua[0]);
          }
          uh[x] = make_float2(u[0].x, u[1].x);
          ul[x] = make_float2(u[0].y, u[1].y);
#pragma unroll
          for (int a = 0; a < NA; ++a) {
            const dfl v0 = NA == 1 ? u[0] : df_add(u[0], ua[a]), v1 = NA == 1 ? u[1] : df_add(u[1], ua[a]);
            p5_cis2(1.0f, make_float2(v0.x, v1.x), make_float2(v0.y, v1.y), zr[a][x], zi[a][x]);
            zn[a][x] = p5_neg(zi[a][x]);
            Ar[a][x] = Ai[a][x] = make_float2(0.0f, 0.0f);
          }
        }
        const int e8 = 8 * g;
        const bool left = e8 + 8 <= emid, mixed = e8 < emid && !left;
        const float4* xg = xs + (4 * g - p0) * NA;
        const uint2* tg = &sh.tab[0][vb];
        const float* wg = wt.tab + e8;
        // n_k w of the group's element pairs at table entry te
        auto weigh = [&](uint2 te, float2 (&w)[4]) {
          const unsigned row = left ? te.x & 0xffffu : te.x >> 16;
          const float4* wr = reinterpret_cast<const float4*>(wg + row * (unsigned)d.wt_w);
          float4 w0 = __ldg(wr), w1 = __ldg(wr + 1);
          if (mixed) {
            // the group around the voxel's column: the left side's values too
            const float4* wl = reinterpret_cast<const float4*>(wg + (te.x & 0xffffu) * (unsigned)d.wt_w);
            const float4 v = __ldg(wl), z = __ldg(wl + 1);
            w0 = make_float4(w0.x + v.x, w0.y + v.y, w0.z + v.z, w0.w + v.w);
            w1 = make_float4(w1.x + z.x, w1.y + z.y, w1.z + z.z, w1.w + z.w);
          }
          const float2 nk = p5_dup(__uint_as_float(te.y));
          w[0] = __fmul2_rn(nk, make_float2(w0.x, w0.y));
          w[1] = __fmul2_rn(nk, make_float2(w0.z, w0.w));
          w[2] = __fmul2_rn(nk, make_float2(w1.x, w1.y));
          w[3] = __fmul2_rn(nk, make_float2(w1.z, w1.w));
        };
        // the bins of the chunk; ONE: with the weights of a steady chunk after the sum
        auto bins = [&](auto one) {
          constexpr bool ONE = decltype(one)::value;
          float2 w[4];
          if constexpr (ONE) weigh(tg[0], w);
#pragma unroll 1
          for (int bs = 0; bs < n; bs += tb) {
            const int be = min(bs + tb, n);
#pragma unroll 4
            for (int b = bs; b < be; ++b) {
              if constexpr (!ONE) weigh(tg[b * P5_M], w);
#pragma unroll
              for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                  const float4 X = xg[b * (FW_EP * NA) + x * NA + a];
                  float2 xr = make_float2(X.x, X.y), xi = make_float2(X.z, X.w);
                  if constexpr (!ONE) {
                    xr = __fmul2_rn(w[x], xr);
                    xi = __fmul2_rn(w[x], xi);
                  }
                  const float2 hr = Ar[a][x], hi = Ai[a][x];
                  Ar[a][x] = __ffma2_rn(hr, zr[a][x], __ffma2_rn(hi, zn[a][x], xr));
                  Ai[a][x] = __ffma2_rn(hr, zi[a][x], __ffma2_rn(hi, zr[a][x], xi));
                }
            }
            // the exact phase at the stretch's last bin
            const float kf = (float)(k_hi - be + 1);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
              for (int a = 0; a < NA; ++a) {
                dfl v0 = make_float2(uh[x].x, ul[x].x), v1 = make_float2(uh[x].y, ul[x].y);
                if constexpr (NA > 1) {
                  v0 = df_add(v0, ua[a]);
                  v1 = df_add(v1, ua[a]);
                }
                float2 cr, ci;
                p5_cis2(kf, make_float2(v0.x, v1.x), make_float2(v0.y, v1.y), cr, ci);
                float2 vr = __ffma2_rn(cr, Ar[a][x], p5_neg(__fmul2_rn(ci, Ai[a][x])));
                float2 vi = __ffma2_rn(cr, Ai[a][x], __fmul2_rn(ci, Ar[a][x]));
                if constexpr (ONE) {
                  vr = __fmul2_rn(w[x], vr);
                  vi = __fmul2_rn(w[x], vi);
                }
                float2& s = sum[STACK ? a : 0];
                s.x += vr.x + vr.y;
                s.y += vi.x + vi.y;
                Ar[a][x] = Ai[a][x] = make_float2(0.0f, 0.0f);
              }
          }
        };
        if (steady) bins(std::true_type{}); else bins(std::false_type{});
        if (lane == 0) c_exec += (unsigned long long)(n * 8 * 32) * NA;
      }
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        const float yx = sum[o].x - comp[o].x, sx = acc[o].x + yx;
        comp[o].x = (sx - acc[o].x) - yx;
        acc[o].x = sx;
        const float yy = sum[o].y - comp[o].y, sy = acc[o].y + yy;
        comp[o].y = (sy - acc[o].y) - yy;
        acc[o].y = sy;
      }
    }
  }
  {
    const unsigned na = __reduce_add_sync(0xffffffffu, c_act), nm = __reduce_add_sync(0xffffffffu, c_emp);
    if (lane == 0) {
      atomicAdd(&sh.n_active, (unsigned long long)na);
      atomicAdd(&sh.n_empty, (unsigned long long)nm);
      atomicAdd(&sh.n_exec, c_exec);
    }
  }
  if (slot == 1) {
#pragma unroll
    for (int o = 0; o < NO; ++o) sh.red[o][vb] = acc[o];
  }
  __syncthreads();
  float2* out = d.split > 1 ? d.part + (size_t)part * NO * nvox : image;
  if (slot == 0 && valid) {
#pragma unroll
    for (int o = 0; o < NO; ++o)
      out[(size_t)o * nvox + vox] =
          make_float2((acc[o].x + sh.red[o][vb].x) * d.scale, (acc[o].y + sh.red[o][vb].y) * d.scale);
    if (d.counters[2] & FLAG_NONFINITE)
      p5_nonfinite(d, out + vox, STACK ? nvox : 0, cc, jc, kt, nb, 0, 1);
  }
  if (tid == 0) {
    atomicAdd(&d.counters[0], sh.n_active * (unsigned long long)NA);
    atomicAdd(&d.counters[1], sh.n_empty * (unsigned long long)NA);
    atomicAdd(&d.counters[4], sh.n_exec);
  }
  if (d.split > 1) {
    // the last of the tile's bin ranges to finish adds them up, in order
    __threadfence();
    __syncthreads();
    if (tid == 0)
      sh.last = atomicAdd(&d.tile_cnt[(size_t)(d.wt_c0 / TILE_X) * ntz + tile], 1u) == (unsigned)(d.split - 1);
    __syncthreads();
    if (sh.last && slot == 0 && valid) {
      __threadfence();
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        float2 s = make_float2(0.0f, 0.0f);
        for (int p = 0; p < d.split; ++p) {
          const float2 v = __ldcg(d.part + ((size_t)p * NO + o) * nvox + vox);
          s.x += v.x;
          s.y += v.y;
        }
        image[(size_t)o * nvox + vox] = s;
      }
    }
  }
}

typedef void (*fw_kernel_t)(const PWDev, float2*, float*);
fw_kernel_t fw_pick(int na, bool stack) {
  if (na == 1) return pw_few_kernel<1, false>;
  return stack ? pw_few_kernel<2, true> : pw_few_kernel<2, false>;
}

}  // namespace

int pw_few_grid(const PWDev& d) {
  return ((d.wt_nc + TILE_X - 1) / TILE_X) * ((d.nz + TILE_Z - 1) / TILE_Z) * d.split;
}

int pw_few_blocks(const PWDev& d) { return d.blocks_per_sm > 0 ? std::min(d.blocks_per_sm, FW_BLOCKS) : FW_BLOCKS; }

cudaError_t launch_pw_few(const PWDev& d0, bool stack, float2* image, float* weights, cudaStream_t s) {
  if (!d0.tc_B || d0.na < 1 || d0.na > 2) return cudaErrorInvalidValue;
  const fw_kernel_t fn = fw_pick(d0.na, stack);
  const int smem = pw_few_blocks(d0) < FW_BLOCKS ? FW_SMEM_ONE : fw_smem(d0.na);
  cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, FW_SMEM_ONE);
  if (e != cudaSuccess) return e;
  fw_pairs_kernel<<<608, 256, 0, s>>>(d0, (float4*)d0.tc_B);
  PWDev d = d0;
  for (int c0 = 0; c0 < d0.nx; c0 += d0.wt_nc) {
    d.wt_c0 = c0;
    d.wt_nc = std::min(d0.wt_nc, d0.nx - c0);
    // a window table that does not hold all columns is refilled for each slab of them
    if (d0.wt_nc < d0.nx && (e = launch_pw_tc_window(d, const_cast<float*>(d.w_tab), const_cast<float*>(d.w_sum), s)) !=
                                cudaSuccess)
      return e;
    fn<<<pw_few_grid(d), FW_THREADS, smem, s>>>(d, image, weights);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace fnum
