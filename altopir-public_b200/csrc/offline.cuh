// offline.cuh -- the scheme's offline set-up on the device, for an engine whose database is resident: the hint's
// ring multiply kept in NTT form, the InspiRING precomputation of every output, the packing matrix, bold_t_hat and
// the row-0 prefixes (Prepared::new, src/service.rs:127-157; YServer::perform_offline_precomputation_simplepir,
// src/server.rs:947-1021; full_packing_with_preprocessing_offline, src/packing.rs:2260-2359).
//
// Ring Z_Q[X]/(X^n + 1).  NTT form: slot s holds the evaluation at psi^(2 brv(s) + 1) (Longa-Naehrig transforms of
// hint.cuh over the tables psi^brv, psi^-brv), the slot order of the reference's automorphism tables, under which
// tau_t acts as the permutation table_t[s] = brv(((t (2 brv(s) + 1)) mod 2n - 1) / 2).
//
// Per output o (n database columns, n = 2048 in the scheme) the reference computes
//   act[j]  = NTT(perm(hint column o n + j))                       prep_pack_lwes (src/packing.rs:910-942)
//   ev[v]   = NTT over j of act[j][v]                               precompute_aggregates_ntt (:2260-2291)
//   r_i     = n^-1 ev[table_(g^i)[s]][s],  rbar_i the same with 2n - g^i,  g = 5, i < n / 2
//   walk i = n/2 - 2 .. 0:  bold_t[i] = NTT(G^-1(r_(i+1))),  r_i += sum_k tau_(g^i)(w)[k] bold_t[i][k]
//                          (and the bar chain with tau_(2n - g^i) and w)          full_packing_offline_mode (:2301-2359)
//   bold_t_hat = NTT(G^-1(rbar_0)),  a_hat = r_0 + sum_k v[k] bold_t_hat[k] in coefficient form
// with G^-1 the base-2^b digits (b = floor(32 / tg) + 1, gadget_invert_transposed_alloc, :1468-1493).
//
// Two identities let the device skip work the reference does literally:
//   * perm (util.rs negacyclic_perm, shift 0) is the automorphism X -> X^-1, whose slot table is s -> n - 1 - s;
//     NTT(hint column) is the hint's accumulator before its inverse transform, so act[j][s] = acc_j[n - 1 - s];
//   * the packing-matrix fold (sw_pack_build) writes every (column z, slot s, digit k) once: the automorphism that
//     carries z to s is e = (2 brv(s) + 1) (2 brv(z) + 1)^-1 mod 2n, e = g^i or 2n - g^i, so each byte of the
//     matrix is a gather from bold_t or bold_t_bar instead of a scatter-add.
#pragma once
#include <cooperative_groups.h>
#include <cstdint>
#include "hint.cuh"
#include "kernels.cuh"
#include "modq.cuh"
#include "sm100.cuh"
#include "waits.cuh"

namespace alto {

constexpr int kActSmemCols = 8;  // database columns per CTA of the shared-memory act kernel: one 32-byte sector per slot

__device__ __forceinline__ int brv_bits(int x, int logn) { return (int)(__brev((unsigned)x) >> (32 - logn)); }

// table_t[s] of the automorphism tau_t (t odd, < 2n)
__device__ __forceinline__ int auto_slot(int t, int s, int n, int logn) {
  const int e = (t * (2 * brv_bits(s, logn) + 1)) & (2 * n - 1);
  return brv_bits((e - 1) >> 1, logn);
}

// g^i mod 2n, or 2n - g^i for the bar chain (g = 5)
__device__ __forceinline__ int gen_pow(int i, int bar, int n) {
  int r = 1, b = 5;
  for (int k = i; k; k >>= 1) {
    if (k & 1) r = (r * b) & (2 * n - 1);
    b = (b * b) & (2 * n - 1);
  }
  return bar ? 2 * n - r : r;
}

// Forward transforms of `cnt` polynomials stored back to back in shared memory.
__device__ __forceinline__ void ntt_fwd_multi(uint32_t *a, int n, int cnt, const uint32_t *__restrict__ psi) {
  const int half = n >> 1;
  for (int m = 1, t = half; m < n; m <<= 1, t >>= 1) {
    for (int b = threadIdx.x; b < cnt * half; b += blockDim.x) {
      const int p = b / half, bb = b - p * half;
      const int i = bb / t, j = p * n + 2 * i * t + (bb - i * t);
      const uint32_t u = a[j], v = mul_q(a[j + t], __ldg(psi + m + i));
      a[j] = add_q(u, v);
      a[j + t] = sub_q(u, v);
    }
    __syncthreads();
  }
}

// acc = INTT(acc) (times n^-1), then its tg base-2^bits digits into dig[k n + s], all in shared memory.
__device__ __forceinline__ void digits_of(uint32_t *acc, uint32_t *dig, int n, int tg, int bits,
                                         const uint32_t *__restrict__ psi_inv, uint32_t n_inv) {
  hint_ntt_inv(acc, n, psi_inv);
  const uint32_t mask = bits >= 32 ? 0xffffffffu : (1u << bits) - 1u;
  for (int s = threadIdx.x; s < n; s += blockDim.x) {
    const uint32_t x = mul_q(acc[s], n_inv);
    for (int k = 0; k < tg; ++k) dig[k * n + s] = bits * k >= 32 ? 0u : (x >> (bits * k)) & mask;
  }
  __syncthreads();
}

// act, one CTA per kActSmemCols consecutive database columns: acc_c = sum_p NTT(D_(p,c)) . qhat_p (qhat = NTT(perm(q_p))),
// stored as actT[o][s][j] = acc_c[n - 1 - s] for column c = o n + j.  Database columns come from the engine's tile
// layout as in hint_ring_kernel.
__global__ void __launch_bounds__(256) offline_act_kernel(const uint8_t *__restrict__ db, size_t kbs, int n,
                                                          int polys, const uint32_t *__restrict__ qhat,
                                                          const uint32_t *__restrict__ psi, uint32_t *__restrict__ act) {
  extern __shared__ uint32_t osm[];
  uint32_t *a = osm, *acc = osm + n;
  const size_t col0 = (size_t)blockIdx.x * kActSmemCols;
  for (int i = threadIdx.x; i < kActSmemCols * n; i += blockDim.x) acc[i] = 0;
  for (int c = 0; c < kActSmemCols; ++c) {
    const size_t col = col0 + c;
    const uint8_t *row = db + (col / 128) * kbs * 16384 + (col % 128) * 128;
    for (int p = 0; p < polys; ++p) {
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const size_t rec = (size_t)p * n + i;
        a[i] = row[(rec >> 7) * 16384 + (rec & 127)];
      }
      __syncthreads();
      hint_ntt_fwd(a, n, psi);
      const uint32_t *qh = qhat + (size_t)p * n;
      for (int i = threadIdx.x; i < n; i += blockDim.x) acc[c * n + i] = add_q(acc[c * n + i], mul_q(a[i], __ldg(qh + i)));
    }
  }
  __syncthreads();
  const size_t o = col0 / n, j0 = col0 % n;  // kActSmemCols divides n: the CTA's columns share their output
  for (int idx = threadIdx.x; idx < n * kActSmemCols; idx += blockDim.x) {
    const int s = idx / kActSmemCols, c = idx - s * kActSmemCols;
    act[(o * n + s) * n + j0 + c] = acc[c * n + (n - 1 - s)];
  }
}

// ------------------------------------------------------------------------------------ the hint on the tensor cores
// acc_c = sum_p NTT(D_(p,c)) . qhat_p for n = 2048, the first seven of the transform's eleven stages as one byte-limb
// product.  With index i = 16 j + r, block i' of 128 after those stages is the residue of D modulo X^16 - zeta_i',
// zeta_i' = psi[128 + i']^2 (Cooley-Tukey stages over psi^brv), so its coefficient r is sum_j W[i'][j] x[16 j + r] with
// W[i'][j] = zeta_i'^j: a 128 x 128 matrix of four byte limbs times the records' bytes, exact in int32 (128 x 255 x 255 <
// 2^23).  A thread then holds the 16 coefficients of one block of one column, so the other four stages, the product with
// qhat and the sum over p are that thread's own and nothing is exchanged.
//
// Operands.  A = the limbs of W, 128 rows x 128 bytes K-major with 128-byte swizzling, resident in shared memory.  B =
// kActCols columns of the database for one p, N = (column, r), K = j: a tile row (one column, 128 records) holds eight j
// of 16 r each, which is one 8 x 16-byte core matrix of an MN-major operand without swizzling; the next column is 128
// bytes on (stride byte offset) and the next eight j the next tile (leading byte offset).  So the database tiles
// are loaded as they are, 16 tiles x kActCols rows a box.  One accumulator of kActCols x 16 columns per limb, two
// buffers: all of TMEM.
//
// Persistent, one CTA an SM: warps 0..15 transform (warp w: TMEM lanes 32 (w & 3).., column w >> 2), warp 16 loads, warp
// 17 issues the MMAs.  Bound by the 16 warps' integer work (53 instructions a record byte, the multiplier pipe 78 %
// busy; the tensor pipe 10 %).  18 warps leave 96 registers a thread, a few short: ptxas spills 132 bytes.  Measured: 2.2 ms a GiB of database, against 8.9 with all eleven stages in registers and
// one shared-memory exchange every three of them.
constexpr int kActCols = 4;                            // database columns of a unit
constexpr int kActStageBytes = 16 * kActCols * 128;    // one p of a unit: 16 tiles x kActCols rows
constexpr int kActStages = 8;
constexpr int kActWBytes = 4 * 128 * 128;
constexpr int kActThreads = 18 * 32;
constexpr int kActTwBytes = 15 * 128 * 4, kActOutBytes = 2048 * kActCols * 4;
constexpr int kActSmem = 1024 + kActWBytes + kActStages * kActStageBytes + kActTwBytes + kActOutBytes + 256;

// The byte limbs of W: w[(l 128 + i') 128 + j] = byte l of zeta_i'^j mod Q.
__global__ void offline_dft_kernel(const uint32_t *__restrict__ psi, uint8_t *__restrict__ w) {
  const int i = blockIdx.x, j = threadIdx.x;
  uint32_t b = __ldg(psi + 128 + i), r = 1;
  b = mul_q(b, b);
  for (int k = j; k; k >>= 1) {
    if (k & 1) r = mul_q(r, b);
    b = mul_q(b, b);
  }
  for (int l = 0; l < 4; ++l) w[(l * 128 + i) * 128 + j] = (uint8_t)(r >> (8 * l));
}

// (a0, a1, a2) += x y as a 96-bit sum
__device__ __forceinline__ void mac96(uint32_t &a0, uint32_t &a1, uint32_t &a2, uint32_t x, uint32_t y) {
  const uint64_t p = (uint64_t)x * y;
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
      : "+r"(a0), "+r"(a1), "+r"(a2)
      : "r"((uint32_t)p), "r"((uint32_t)(p >> 32)));
}

// Cooley-Tukey butterfly on 32-bit representatives (lazy_add), Gentleman-Sande on residues; twiddles in Montgomery form.
__device__ __forceinline__ void bf_ct(uint32_t &x, uint32_t &y, uint32_t wm) {
  const uint32_t v = mont_q(y, wm);
  y = lazy_sub(x, v);
  x = lazy_add(x, v);
}
__device__ __forceinline__ void bf_gs(uint32_t &x, uint32_t &y, uint32_t wm) {
  const uint32_t s = add_q(x, y);
  y = mont_q(sub_q(x, y), wm);
  x = s;
}

// qhat in the order the transform threads read it: word (p 4 + v) 512 + 4 i' + u is slot 16 i' + 4 v + u (hint_query_kernel
// with BLOCKED).  act[(o n + s) n + j] = acc_c[n - 1 - s], c = o n + j, as offline_act_kernel writes it.
__global__ void __launch_bounds__(kActThreads, 1)
    offline_act_mma_kernel(const __grid_constant__ CUtensorMap map_db, const __grid_constant__ CUtensorMap map_w,
                           int polys, int groups, const uint4 *__restrict__ qhat, const uint32_t *__restrict__ psi,
                           uint32_t *__restrict__ act, uint32_t *err) {
  constexpr int n = 2048, N = 16 * kActCols;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw);
  const uint32_t ring = base + kActWBytes;
  uint32_t *tw = reinterpret_cast<uint32_t *>(smem + kActWBytes + kActStages * kActStageBytes);
  uint32_t *stage_out = tw + 15 * 128;
  uint64_t *bars = reinterpret_cast<uint64_t *>(stage_out + 2048 * kActCols);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * kActStages, accf0 = empty0 + 8 * kActStages,
                 acce0 = accf0 + 16, wbar = acce0 + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kActStages + 5);
  volatile int *bail = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kActStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accf0 + 8 * b, 1);
      mbar_init(acce0 + 8 * b, 16);
    }
    mbar_init(wbar, 1);
    *bail = 0;
    fence_barrier_init();
  }
  if (warp == 16 && lane == 0) {
    tma_prefetch_desc(&map_db);
    tma_prefetch_desc(&map_w);
  }
  if (warp == 17) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  // twiddles of the last four stages, [stage and block][i']: psi[128 + i'], psi[256 + 2 i' + h], ...
  for (int x = tid; x < 15 * 128; x += kActThreads) {
    const int t = x >> 7, i = x & 127, st = t < 1 ? 0 : t < 3 ? 1 : t < 7 ? 2 : 3, h = t - ((1 << st) - 1);
    tw[x] = to_mont(__ldg(psi + (128 << st) + (i << st) + h));
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Every wait is bounded; after a timeout (recorded in *err, with the bail flag) the later ones fail within a few polls, the
  // loaders and the MMA issuer stop, and the transform warps run on to the end, so that they meet their barriers.
  if (warp == 16) {
    if (lane == 0) {
      mbar_arrive_expect_tx(wbar, kActWBytes);
      for (int l = 0; l < 4; ++l) tma_load_2d(base + l * 16384, &map_w, wbar, 0, 128 * l, policy_evict_normal());
      const uint64_t pol = policy_evict_first();
      int g = 0;
      bool stop = false;
      for (int u = blockIdx.x; u < groups && !stop; u += gridDim.x) {
        const int col = u * kActCols, mt = col >> 7, row = col & 127;
        for (int p = 0; p < polys; ++p, ++g) {
          const int s = g % kActStages, round = g / kActStages;
          if (round > 0 && !mbar_wait(empty0 + 8 * s, (round - 1) & 1, err, ALTO_ERR_WAIT_EMPTY, bail)) {
            stop = true;
            break;
          }
          mbar_arrive_expect_tx(full0 + 8 * s, kActStageBytes);
          tma_load_rows(ring + s * kActStageBytes, &map_db, full0 + 8 * s, row, 16 * p, mt, pol);
        }
      }
      if (stop) {  // loads already issued land within microseconds
        const uint64_t t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 17) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_u8u8_s32(N) | (1u << 16);  // B is MN-major
      int g = 0;
      bool stop = !mbar_wait(wbar, 0, err, ALTO_ERR_WAIT_FULL, bail);
      for (int u = blockIdx.x; u < groups && !stop; u += gridDim.x) {
        for (int p = 0; p < polys; ++p, ++g) {
          const int s = g % kActStages, round = g / kActStages, b = g & 1, use = g >> 1;
          if (use > 0 && !mbar_wait(acce0 + 8 * b, (use - 1) & 1, err, ALTO_ERR_WAIT_ACCUM, bail)) stop = true;
          if (stop || !mbar_wait(full0 + 8 * s, round & 1, err, ALTO_ERR_WAIT_FULL, bail)) {
            stop = true;
            break;
          }
          tc_fence_after();
          const uint32_t sb = ring + s * kActStageBytes;
#pragma unroll
          for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)  // 32 j: four tiles
              mma_i8(tmem + (uint32_t)((b * 4 + l) * N), desc_sw128(base + l * 16384 + kk * 32),
                     desc_mn_plain(sb + kk * 4 * (kActCols * 128), kActCols * 128, 128), idesc, kk != 0);
          mma_commit(empty0 + 8 * s);
          mma_commit(accf0 + 8 * b);
        }
      }
      if (*bail) {  // MMAs issued so far complete before TMEM and shared memory go away
        const uint64_t t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) {
        }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, c = warp >> 2, i = q * 32 + lane;  // block i' of column c
    int g = 0;
    for (int u = blockIdx.x; u < groups; u += gridDim.x) {
      uint32_t a0[16], a1[16], a2[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) a0[k] = a1[k] = a2[k] = 0;
      for (int p = 0; p < polys; ++p, ++g) {
        const int b = g & 1, use = g >> 1;
        mbar_wait_warp(accf0 + 8 * b, use & 1, err, ALTO_ERR_WAIT_ACCUM, bail);
        tc_fence_after();
        const uint32_t ta = tmem + (uint32_t)(b * 4 * N + 16 * c) + ((uint32_t)(q * 32) << 16);
        uint32_t x[16];
        {
          uint32_t hi[16], lo[16];
          tmem_ld16(ta + 2 * N, x);
          tmem_ld16(ta + 3 * N, hi);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; ++k) x[k] += hi[k] << 8;  // < 2^32
          tmem_ld16(ta, lo);
          tmem_ld16(ta + N, hi);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acce0 + 8 * b);
          // lo + 2^8 hi + 2^16 x: the high half of x folds to 12287 (x >> 16) < 2^30, so that sum stays below 2^32 - 12287
#pragma unroll
          for (int k = 0; k < 16; ++k) x[k] = lazy_add(x[k] << 16, lo[k] + (hi[k] << 8) + (x[k] >> 16) * kFold);
        }
        const uint32_t *t = tw + i;
#pragma unroll
        for (int st = 0; st < 4; ++st) {
          const int h = 8 >> st;
#pragma unroll
          for (int blk = 0; blk < (1 << st); ++blk) {
            const uint32_t wm = t[((1 << st) - 1 + blk) * 128];
#pragma unroll
            for (int r = 0; r < h; ++r) bf_ct(x[blk * 2 * h + r], x[blk * 2 * h + h + r], wm);
          }
        }
        const uint4 *qp = qhat + (size_t)p * 512 + i;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 y = __ldg(qp + 128 * v);
          mac96(a0[4 * v], a1[4 * v], a2[4 * v], x[4 * v], y.x);
          mac96(a0[4 * v + 1], a1[4 * v + 1], a2[4 * v + 1], x[4 * v + 1], y.y);
          mac96(a0[4 * v + 2], a1[4 * v + 2], a2[4 * v + 2], x[4 * v + 2], y.z);
          mac96(a0[4 * v + 3], a1[4 * v + 3], a2[4 * v + 3], x[4 * v + 3], y.w);
        }
      }
      // 2^32 = 12287 and 2^64 = 12287^2 (mod Q).  a2 counts at most one carry a product (polys < 2^31 of them), so the sum
      // stays below 2^59
#pragma unroll
      for (int k = 0; k < 16; ++k)
        stage_out[(k * 128 + i) * kActCols + c] =
            red_q64((uint64_t)a1[k] * kFold + a0[k] + (uint64_t)a2[k] * ((uint64_t)kFold * kFold));
      asm volatile("bar.sync 1, 512;" ::: "memory");
      const size_t col = (size_t)u * kActCols, o = col / n, j0 = col % n;
      for (int y = tid; y < 2048; y += 512) {
        const int s = 16 * (y & 127) + (y >> 7);
        *reinterpret_cast<uint4 *>(act + (o * n + (n - 1 - s)) * n + j0) =
            *reinterpret_cast<const uint4 *>(stage_out + y * kActCols);
      }
      asm volatile("bar.sync 1, 512;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ev: forward transform of every row of act in place (one CTA per row of n).
__global__ void __launch_bounds__(256) offline_rows_kernel(uint32_t *__restrict__ rows, int n,
                                                           const uint32_t *__restrict__ psi) {
  extern __shared__ uint32_t osm[];
  uint32_t *r = rows + (size_t)blockIdx.x * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) osm[i] = r[i];
  __syncthreads();
  hint_ntt_fwd(osm, n, psi);
  for (int i = threadIdx.x; i < n; i += blockDim.x) r[i] = osm[i];
}

// The backward walk, one CTA per (output o, chain bar): bar 0 walks r with tau_(g^i)(w), bar 1 walks rbar with
// tau_(2n - g^i)(w).  bt[((o 2 + bar) (n/2 - 1) + i) tg + k][s] = bold_t (bar 0) or bold_t_bar (bar 1); the chain's
// final r_0 (rbar_0) goes to last[(o 2 + bar) n + s].
__global__ void __launch_bounds__(1024) offline_walk_kernel(const uint32_t *__restrict__ ev, int n, int logn, int tg,
                                                            int bits, const uint32_t *__restrict__ w,
                                                            const uint32_t *__restrict__ psi,
                                                            const uint32_t *__restrict__ psi_inv, uint32_t n_inv,
                                                            uint32_t *__restrict__ bt, uint32_t *__restrict__ last) {
  extern __shared__ uint32_t osm[];
  uint32_t *cur = osm, *dig = osm + n;
  const int o = blockIdx.x >> 1, bar = blockIdx.x & 1, half = n >> 1;
  const uint32_t *evo = ev + (size_t)o * n * n;
  int e = gen_pow(half - 1, bar, n);
  for (int s = threadIdx.x; s < n; s += blockDim.x) cur[s] = mul_q(evo[(size_t)auto_slot(e, s, n, logn) * n + s], n_inv);
  __syncthreads();
  for (int i = half - 2; i >= 0; --i) {
    digits_of(cur, dig, n, tg, bits, psi_inv, n_inv);
    ntt_fwd_multi(dig, n, tg, psi);
    e = gen_pow(i, bar, n);
    uint32_t *out = bt + (((size_t)(o * 2 + bar) * (half - 1) + i) * tg) * n;
    for (int s = threadIdx.x; s < n; s += blockDim.x) {
      const int ts = auto_slot(e, s, n, logn);
      uint32_t acc = mul_q(evo[(size_t)ts * n + s], n_inv);
      for (int k = 0; k < tg; ++k) {
        const uint32_t d = dig[k * n + s];
        out[k * n + s] = d;
        acc = add_q(acc, mul_q(__ldg(w + k * n + ts), d));
      }
      cur[s] = acc;
    }
    __syncthreads();
  }
  for (int s = threadIdx.x; s < n; s += blockDim.x) last[(size_t)(o * 2 + bar) * n + s] = cur[s];
}

// The same walk with one thread-block cluster of C CTAs per (output, chain): every CTA runs the step's inverse
// transform (the same values in each), takes the digits k = c, c + C, ... of its rank c, transforms them and forms
// its part of sum_k tau(w)[k] bold_t[i][k]; the parts are summed through distributed shared memory.  A step costs
// two transforms instead of 1 + tg.  Launched with cluster dimensions (C, 1, 1): CTAs C q .. C q + C - 1 are chain q.
__global__ void __launch_bounds__(1024) offline_walk_cluster_kernel(const uint32_t *__restrict__ ev, int n, int logn,
                                                                    int tg, int bits, const uint32_t *__restrict__ w,
                                                                    const uint32_t *__restrict__ psi,
                                                                    const uint32_t *__restrict__ psi_inv,
                                                                    uint32_t n_inv, uint32_t *__restrict__ bt,
                                                                    uint32_t *__restrict__ last) {
  namespace cg = cooperative_groups;
  extern __shared__ uint32_t osm[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), c = (int)cl.block_rank();
  const int chain = blockIdx.x / C, o = chain >> 1, bar = chain & 1, half = n >> 1;
  const int kper = (tg + C - 1) / C;
  uint32_t *cur = osm, *part = osm + n, *dig = osm + 2 * n;
  const uint32_t mask = bits >= 32 ? 0xffffffffu : (1u << bits) - 1u;
  const uint32_t *evo = ev + (size_t)o * n * n;
  int e = gen_pow(half - 1, bar, n);
  for (int s = threadIdx.x; s < n; s += blockDim.x) cur[s] = mul_q(evo[(size_t)auto_slot(e, s, n, logn) * n + s], n_inv);
  __syncthreads();
  constexpr int kAgg = 4;  // slots a thread gathers ahead (n <= kAgg blockDim.x)
  for (int i = half - 2; i >= 0; --i) {
    // this step's aggregate r_i, loaded before the transforms so that its latency hides behind them
    e = gen_pow(i, bar, n);
    uint32_t agg[kAgg];
#pragma unroll
    for (int j = 0; j < kAgg; ++j) {
      const int s = threadIdx.x + j * (int)blockDim.x;
      agg[j] = s < n ? evo[(size_t)auto_slot(e, s, n, logn) * n + s] : 0u;
    }
    hint_ntt_inv(cur, n, psi_inv);
    for (int s = threadIdx.x; s < n; s += blockDim.x) {
      const uint32_t x = mul_q(cur[s], n_inv);
      for (int j = 0; j < kper; ++j) {
        const int k = c + C * j;
        dig[j * n + s] = (k < tg && bits * k < 32) ? (x >> (bits * k)) & mask : 0u;
      }
    }
    __syncthreads();
    ntt_fwd_multi(dig, n, kper, psi);
    uint32_t *out = bt + (((size_t)chain * (half - 1) + i) * tg) * n;
    for (int s = threadIdx.x; s < n; s += blockDim.x) {
      const int ts = auto_slot(e, s, n, logn);
      uint32_t p = 0;
      for (int j = 0; j < kper; ++j) {
        const int k = c + C * j;
        if (k < tg) {
          const uint32_t d = dig[j * n + s];
          out[k * n + s] = d;
          p = add_q(p, mul_q(__ldg(w + k * n + ts), d));
        }
      }
      part[s] = p;
    }
    cl.sync();  // every CTA's part is written
#pragma unroll
    for (int j = 0; j < kAgg; ++j) {
      const int s = threadIdx.x + j * (int)blockDim.x;
      if (s >= n) break;
      uint32_t acc = mul_q(agg[j], n_inv);
      for (int r = 0; r < C; ++r) acc = add_q(acc, cl.map_shared_rank(part, r)[s]);
      cur[s] = acc;
    }
    cl.sync();  // every CTA has read the parts (they are rewritten next step) and holds the whole new r_i
  }
  if (c == 0)
    for (int s = threadIdx.x; s < n; s += blockDim.x) last[(size_t)chain * n + s] = cur[s];
}

// ------------------------------------------------------------------------------------ register transforms, n = 2048
// 512 threads hold 4 values each.  Layout s: index i = (g >> s) << (s + 2) | m << s | (g & (2^s - 1)), so a thread's four
// values differ in bits s and s + 1.  The inverse transform runs two stages in each of the layouts 0, 2, 4, 6, 8 and the
// last one (t = 1024) in layout 9; the forward transform the same backwards.  Between layouts the values go through
// shared memory, padded against bank conflicts (reg_pad).  0 <-> 2 <-> 4 stay inside a warp, 4 <-> 6 inside
// two warps and 6 <-> 8 inside eight, so that only 8 <-> 9 needs a barrier of the whole block.  Twiddles are in
// Montgomery form.
struct RegTwiddles {
  uint32_t c[5], a[5][2], d;  // per layout: the stage of bit s + 1, the two of bit s; the last stage
};
__device__ __forceinline__ void load_tw(RegTwiddles &t, const uint32_t *__restrict__ psi, int g) {
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int base = (2048 >> (2 * q + 2)) + (g >> (2 * q));
    t.c[q] = to_mont(__ldg(psi + base));
    t.a[q][0] = to_mont(__ldg(psi + 2 * base));
    t.a[q][1] = to_mont(__ldg(psi + 2 * base + 1));
  }
  t.d = to_mont(__ldg(psi + 1));
}

template <int S>
__device__ __forceinline__ int reg_index(int g, int m) {
  return ((g >> S) << (S + 2)) | (m << S) | (g & ((1 << S) - 1));
}
// Every exchange (layouts S and S + 2; 8 and 9 for S = 8) has a buffer of its own, so that a thread only ever overwrites
// words that it read itself the last time.  Index i lies there at reg_pad(i), padded so that both layouts' accesses are
// free of bank conflicts; the padding adds, so that the four values of a thread lie at fixed distances from its first.
template <int S>
__device__ __forceinline__ constexpr int reg_pad(int i) {
  return S == 0 ? i + 4 * (i >> 5) : S == 2 ? 2304 + i + 20 * (i >> 4) : S == 4 ? 6912 + i + 16 * (i >> 6) : 9472 + (S - 6) * 1024 + i;
}
constexpr int kRegWords = 13568;  // of the five buffers
// Layout A's value m in the buffer of exchange S, relative to value 0: bits A and A + 1 of the other index bits are zero.
template <int S, int A>
__device__ __forceinline__ constexpr int reg_step(int m) {
  return reg_pad<S>(m << A) - reg_pad<S>(0);
}
__device__ __forceinline__ void sync_warps(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Moves the values from layout A to layout B through `buf`, behind a barrier of the threads that share words.
template <int A, int B>
__device__ __forceinline__ void relayout(uint32_t (&x)[4], uint32_t *buf, int g) {
  constexpr int S = A < B ? A : B;
  uint32_t *to = buf + reg_pad<S>(reg_index<A>(g, 0));
  const uint32_t *from = buf + reg_pad<S>(reg_index<B>(g, 0));
  if constexpr (A == 0) {
    *reinterpret_cast<uint4 *>(to) = make_uint4(x[0], x[1], x[2], x[3]);
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) to[reg_step<S, A>(m)] = x[m];
  }
  if constexpr (S < 4) __syncwarp();
  else if constexpr (S == 4) sync_warps(1 + (g >> 6), 64);
  else if constexpr (S == 6) sync_warps(9 + (g >> 8), 256);
  else __syncthreads();
  if constexpr (B == 0) {
    const uint4 u = *reinterpret_cast<const uint4 *>(from);
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) x[m] = from[reg_step<S, B>(m)];
  }
}
__device__ __forceinline__ void round_gs(uint32_t (&x)[4], const RegTwiddles &t, int q) {
  bf_gs(x[0], x[1], t.a[q][0]);
  bf_gs(x[2], x[3], t.a[q][1]);
  bf_gs(x[0], x[2], t.c[q]);
  bf_gs(x[1], x[3], t.c[q]);
}
__device__ __forceinline__ void round_ct(uint32_t (&x)[4], const RegTwiddles &t, int q) {
  bf_ct(x[0], x[2], t.c[q]);
  bf_ct(x[1], x[3], t.c[q]);
  bf_ct(x[0], x[1], t.a[q][0]);
  bf_ct(x[2], x[3], t.a[q][1]);
}

// Residues in layout 0 in, residues in layout 9 out (without n^-1).  `buf`: kRegWords; the two transforms in turn need no
// barrier between them, two of the same do.
__device__ __forceinline__ void intt_regs(uint32_t (&x)[4], uint32_t *buf, const RegTwiddles &t, int g) {
  round_gs(x, t, 0);
  relayout<0, 2>(x, buf, g);
  round_gs(x, t, 1);
  relayout<2, 4>(x, buf, g);
  round_gs(x, t, 2);
  relayout<4, 6>(x, buf, g);
  round_gs(x, t, 3);
  relayout<6, 8>(x, buf, g);
  round_gs(x, t, 4);
  relayout<8, 9>(x, buf, g);
  bf_gs(x[0], x[2], t.d);
  bf_gs(x[1], x[3], t.d);
}
// 32-bit representatives in layout 9 in, the same in layout 0 out.
__device__ __forceinline__ void ntt_regs(uint32_t (&x)[4], uint32_t *buf, const RegTwiddles &t, int g) {
  bf_ct(x[0], x[2], t.d);
  bf_ct(x[1], x[3], t.d);
  relayout<9, 8>(x, buf, g);
  round_ct(x, t, 4);
  relayout<8, 6>(x, buf, g);
  round_ct(x, t, 3);
  relayout<6, 4>(x, buf, g);
  round_ct(x, t, 2);
  relayout<4, 2>(x, buf, g);
  round_ct(x, t, 1);
  relayout<2, 0>(x, buf, g);
  round_ct(x, t, 0);
}

// offline_rows_kernel for n = 2048: the transform of every row in place, in registers; the next row's loads run ahead.
// 32,768 rows: 0.28 ms against 0.73 with shared-memory stages (0.08 at the copy rate; bound by integer instructions).
__global__ void __launch_bounds__(512, 2) offline_rows8_kernel(uint32_t *__restrict__ rows, int count,
                                                               const uint32_t *__restrict__ psi) {
  constexpr int n = 2048;
  extern __shared__ __align__(16) uint32_t buf[];
  const int g = threadIdx.x;
  RegTwiddles t;
  load_tw(t, psi, g);
  uint32_t x[4], next[4] = {0, 0, 0, 0};
  int r = blockIdx.x;
  if (r < count)
#pragma unroll
    for (int m = 0; m < 4; ++m) next[m] = rows[(size_t)r * n + reg_index<9>(g, m)];
  for (; r < count; r += gridDim.x) {
#pragma unroll
    for (int m = 0; m < 4; ++m) x[m] = next[m];
    if (r + (int)gridDim.x < count)
#pragma unroll
      for (int m = 0; m < 4; ++m) next[m] = rows[(size_t)(r + gridDim.x) * n + reg_index<9>(g, m)];
    ntt_regs(x, buf, t, g);
    *reinterpret_cast<uint4 *>(rows + (size_t)r * n + 4 * g) =
        make_uint4(canon_q(x[0]), canon_q(x[1]), canon_q(x[2]), canon_q(x[3]));
    __syncthreads();  // the buffers are free for the next row
  }
}

// The cluster walk for n = 2048, tg CTAs a cluster (one digit each), both transforms in registers.  A chain is 1022
// dependent steps, so a step's time is its instructions and barriers in a row: the twiddles stay in registers for the
// whole walk, the coefficients leave the inverse transform in the layout that the forward one starts from, and n^-1 is
// folded into w and the aggregates (x holds n^-1 times the reference's r_i, so the inverse transform gives its
// coefficients themselves).  Every CTA runs the inverse transform, transforms its own digit, and copies its share of the
// next r_i -- its digit's product with the rotated w, plus the aggregate of the slots that are its own modulo C -- into
// every other CTA's shared memory (a 512-byte bulk copy a warp, counted on the receiver's barrier).  The share buffers
// and their barriers alternate by step: a warp sends its share of step i + 2 after every share of step i + 1 has arrived,
// which the others' same warps sent after they had received and read step i's.
// Measured for one walk of 1022 steps (the set-up of 2,048 records x 2,048 bytes): 15.6 ms with twiddles loaded from
// global memory by 256 threads of 8 values and shares pushed by remote stores before a cluster barrier, 6.7 with the
// twiddles in registers, Montgomery products and no exchange between the transforms, 6.2 with bulk copies for the
// remote stores, 4.7 with 512 threads of 4 values (two warps a scheduler left most of the fixed latencies exposed).
__global__ void __launch_bounds__(512, 1) offline_walk8_kernel(const uint32_t *__restrict__ ev, int bits,
                                                               const uint32_t *__restrict__ w,
                                                               const uint32_t *__restrict__ psi,
                                                               const uint32_t *__restrict__ psi_inv, uint32_t n_inv,
                                                               uint32_t *__restrict__ bt, uint32_t *__restrict__ last,
                                                               uint32_t *err) {
  namespace cg = cooperative_groups;
  constexpr int n = 2048, half = n / 2;
  extern __shared__ __align__(16) uint32_t osm[];
  __shared__ __align__(8) uint64_t arrived[2];
  __shared__ int bail;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), k = (int)cl.block_rank();  // one CTA per gadget digit; this CTA's digit
  const int chain = blockIdx.x / C, o = chain >> 1, bar = chain & 1, g = threadIdx.x;
  uint32_t *buf = osm, *wk = osm + kRegWords, *parts = wk + n;  // parts[buffer][rank][slot]
  const int shift = bits * k < 32 ? bits * k : 0;
  const uint32_t mask = bits * k < 32 ? (bits >= 32 ? 0xffffffffu : (1u << bits) - 1u) : 0u;
  const uint32_t *evo = ev + (size_t)o * n * n;
  RegTwiddles fw, iv;
  load_tw(fw, psi, g);
  load_tw(iv, psi_inv, g);
  for (int s = g; s < n; s += 512) wk[s] = to_mont(mul_q(__ldg(w + k * n + s), n_inv));
  const uint32_t agg_scale = to_mont(mul_q(n_inv, n_inv));
  uint32_t odd[4], own = 0;  // 2 brv(slot) + 1; the thread's slots whose aggregate this CTA adds
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    odd[m] = 2u * (__brev((uint32_t)(4 * g + m)) >> 21) + 1u;
    if ((4 * g + m) % C == k) own |= 1u << m;
  }
  auto slot_of = [&](uint32_t e, int m) { return __brev(((e * odd[m]) & (2 * n - 1)) >> 1) >> 21; };
  uint32_t x[4], e = (uint32_t)gen_pow(half - 1, bar, n);
#pragma unroll
  for (int m = 0; m < 4; ++m) x[m] = mont_q(evo[(size_t)slot_of(e, m) * n + 4 * g + m], agg_scale);
  const uint32_t bar0 = smem_u32(arrived);
  if (g == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar0 + 8, 1);
    bail = 0;
    fence_barrier_init();
  }
  uint32_t *out = bt + (((size_t)chain * (half - 1) + (half - 2)) * C + k) * n + 4 * g;
  cluster_sync_all();  // w is in shared memory, and every CTA's barriers are ready for the others' shares
  ShareTurns turn;  // the same in all threads of a warp
  for (int i = half - 2; i >= 0; --i) {
    if (g == 0) turn.arm([&](int b) { mbar_arrive_expect_tx(bar0 + 8 * b, (uint32_t)((C - 1) * n * 4)); });
    // the aggregates are gathered now, so that their latency hides behind the transforms
    e = (e * 0xcccccccdu) & (2 * n - 1);  // times 5^-1 mod 2n
    uint32_t agg[4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
      agg[m] = (own >> m) & 1u ? __ldg(evo + (size_t)slot_of(e, m) * n + 4 * g + m) : 0u;
    intt_regs(x, buf, iv, g);
#pragma unroll
    for (int m = 0; m < 4; ++m) x[m] = (x[m] >> shift) & mask;
    ntt_regs(x, buf, fw, g);
    uint32_t v[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      x[m] = canon_q(x[m]);
      v[m] = mont_q(x[m], wk[slot_of(e, m)]);
      if ((own >> m) & 1u) v[m] = add_q(v[m], mont_q(agg[m], agg_scale));
    }
    uint32_t *mine = parts + (size_t)(turn.buf * C + k) * n;
    reinterpret_cast<uint4 *>(mine)[g] = make_uint4(v[0], v[1], v[2], v[3]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((g & 31) < C && (g & 31) != k)  // each warp sends its 128 words as soon as they are written
      turn.send([&](int b) {
        const uint32_t src = smem_u32(mine + 4 * (g & ~31)), r = (uint32_t)(g & 31);
        bulk_copy_to_cta(map_to_rank(src, r), src, 512, map_to_rank(bar0 + 8 * b, r));
      });
    *reinterpret_cast<uint4 *>(out) = make_uint4(x[0], x[1], x[2], x[3]);
    out -= (size_t)C * n;
    // after a timeout (recorded in *err) the walk goes on by itself, so that every barrier of the block is met by all its
    // threads
    turn.wait([&](int b, uint32_t parity) {
      return mbar_wait_warp<true>(bar0 + 8 * b, parity, err, ALTO_ERR_WAIT_FULL, &bail);
    });
    const uint4 *p = reinterpret_cast<const uint4 *>(parts + (size_t)turn.buf * C * n) + g;
    uint4 u = p[0];
    x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
    for (int r = 1; r < C; ++r) {
      u = p[r * (n / 4)];
      x[0] = lazy_add(x[0], u.x); x[1] = lazy_add(x[1], u.y); x[2] = lazy_add(x[2], u.z); x[3] = lazy_add(x[3], u.w);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) x[m] = canon_q(x[m]);
    turn.next();
  }
  if (!turn.live) {  // copies already issued land within microseconds; no CTA is gone before
    const uint64_t t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) {
    }
  }
  __syncwarp();
  cluster_sync_all();  // no CTA exits while another may still copy into its shared memory
  if (k == 0)
#pragma unroll
    for (int m = 0; m < 4; ++m) last[(size_t)chain * n + 4 * g + m] = mul_q(x[m], n);
}

// Per output (one CTA each): bold_t_hat = NTT(G^-1(rbar_0)); a_hat = INTT(r_0 + sum_k v[k] bold_t_hat[k]).  Writes
// the engine's bold_t_hat (times the tail's scale 2^-log2 n), the row-0 prefix (a_hat rescaled to 2^q2_bits, packed
// LSB first, the rest of the part zero: switch_prefix_row0, src/modulus_switch.rs:136-147) and, for callers that
// ask, the plain bold_t_hat and a_hat.
__global__ void __launch_bounds__(1024) offline_finish_kernel(const uint32_t *__restrict__ last, int n, int tg,
                                                              int bits, const uint32_t *__restrict__ v,
                                                              const uint32_t *__restrict__ psi,
                                                              const uint32_t *__restrict__ psi_inv, uint32_t n_inv,
                                                              uint32_t tail_scale, uint32_t *__restrict__ that_eng,
                                                              uint8_t *__restrict__ prefix, size_t part_len,
                                                              int q2_bits, uint32_t *__restrict__ that_out,
                                                              uint32_t *__restrict__ a_hat_out) {
  extern __shared__ uint32_t osm[];
  uint32_t *cur = osm, *dig = osm + n;
  const int o = blockIdx.x;
  const size_t count = (size_t)tg * n;
  for (int s = threadIdx.x; s < n; s += blockDim.x) cur[s] = last[(size_t)(o * 2 + 1) * n + s];
  __syncthreads();
  digits_of(cur, dig, n, tg, bits, psi_inv, n_inv);
  ntt_fwd_multi(dig, n, tg, psi);
  for (int s = threadIdx.x; s < n; s += blockDim.x) {
    uint32_t acc = last[(size_t)(o * 2) * n + s];
    for (int k = 0; k < tg; ++k) {
      const uint32_t t = dig[k * n + s];
      acc = add_q(acc, mul_q(__ldg(v + k * n + s), t));
      that_eng[o * count + k * n + s] = mul_q(t, tail_scale);
      if (that_out) that_out[o * count + k * n + s] = t;
    }
    cur[s] = acc;
  }
  __syncthreads();
  hint_ntt_inv(cur, n, psi_inv);
  for (int s = threadIdx.x; s < n; s += blockDim.x) {
    cur[s] = mul_q(cur[s], n_inv);
    if (a_hat_out) a_hat_out[(size_t)o * n + s] = cur[s];
  }
  __syncthreads();
  // rescale(a, Q, 2^q2_bits): centre, round half away from zero, reduce (src/modulus_switch.rs:116-130)
  const int64_t q = kQ32, half = kQ32 / 2, q2 = int64_t(1) << q2_bits;
  uint8_t *pre = prefix + (size_t)o * part_len;
  const size_t row0_bytes = ((size_t)q2_bits * n + 7) / 8;
  for (size_t b = row0_bytes + threadIdx.x; b < part_len; b += blockDim.x) pre[b] = 0;
  // 8 values of q2_bits bits fill q2_bits whole bytes: thread g packs values 8 g .. 8 g + 7
  for (int g = threadIdx.x; g < n / 8; g += blockDim.x) {
    uint8_t bytes[64] = {};
    for (int u = 0; u < 8; ++u) {
      const int64_t a = cur[8 * g + u];
      const int64_t c = a >= half ? a - q : a;
      int64_t t = (c * q2 + (c >= 0 ? half : -half)) / q;
      t = ((t % q2) + q2) % q2;
      for (int bit = 0; bit < q2_bits; ++bit)
        if ((t >> bit) & 1) bytes[(u * q2_bits + bit) >> 3] |= (uint8_t)(1u << ((u * q2_bits + bit) & 7));
    }
    for (int k = 0; k < q2_bits; ++k) pre[(size_t)g * q2_bits + k] = bytes[k];
  }
}

// The packing matrix in the engine's tile layout: U[col][k n + s] = bold_t[o][i][k][z] (or bold_t_bar), col = o n + z, for
// the automorphism t = g^i (or 2n - g^i) that carries z to s, zero for the two slots that no step of the walk reaches;
// times tail_scale; byte j of it goes to row 4 col + j, byte kk of the row, of tile (row / 128, kk / 128) at (mt kbs +
// kb) 16 KB.  A CTA takes kPlaneCols columns of one digit k: it reads their words of every bold_t row (32 bytes a row),
// scatters each to its slot s in shared memory, then writes 32 rows of the matrix, 4 KB together in every tile.  Bound by
// HBM and the scattered shared-memory stores: the 1 GiB matrix takes 0.61 ms (1 GiB read, 1 GiB written; 0.33 at the copy
// rate) against 2.47 with one thread per value, a 32-byte sector read for each and four byte stores.
// It writes 16 slots at a time, so n is at least 16 (a multiple of it, being a power of two).
constexpr int kPlaneCols = 8, kPlaneMinN = 16;
__global__ void __launch_bounds__(256) offline_planes_kernel(const uint32_t *__restrict__ bt, int n, int logn, int tg,
                                                             const uint16_t *__restrict__ gen, uint32_t tail_scale,
                                                             uint8_t *__restrict__ ub, size_t kbs) {
  extern __shared__ __align__(16) uint32_t osm[];  // [column][slot], rows padded by 4 words
  const int half = n >> 1, ld = n + 4, k = blockIdx.y, hz = threadIdx.x & 1;
  const size_t col0 = (size_t)blockIdx.x * kPlaneCols;
  const int o = (int)(col0 / n), z0 = (int)(col0 % n) + 4 * hz;
  const uint32_t scale = to_mont(tail_scale);
  int odd[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) odd[v] = 2 * brv_bits(z0 + v, logn) + 1;
  uint32_t *mine = osm + 4 * hz * ld;
  const uint32_t *src = bt + (size_t)o * 2 * (half - 1) * tg * n + (size_t)k * n + z0;
#pragma unroll 4
  for (int r = threadIdx.x >> 1; r < n; r += 128) {  // rows of both chains, the last one of each all zero
    const int bar = r >= half, i = r - bar * half, t = bar ? 2 * n - __ldg(gen + i) : __ldg(gen + i);
    uint4 x = make_uint4(0, 0, 0, 0);
    if (i < half - 1) x = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)(bar * (half - 1) + i) * tg * n));
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int v = 0; v < 4; ++v)
      mine[v * ld + brv_bits(((t * odd[v]) & (2 * n - 1)) >> 1, logn)] = mont_q(w[v], scale);
  }
  __syncthreads();
  for (int y = threadIdx.x; y < kPlaneCols * (n / 16); y += 256) {  // 16 slots of a column: 16 bytes in each plane
    // consecutive threads take the eight 16-byte pieces of a row, then the next columns (n < 128 has fewer pieces a row)
    const int pieces = n < 128 ? n / 16 : 8, per = pieces * kPlaneCols;
    const int tile = y / per, rest = y - tile * per, c = rest / pieces, s = tile * 128 + (rest - c * pieces) * 16;
    uint32_t p[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 u = *reinterpret_cast<const uint4 *>(osm + c * ld + s + 4 * q);
      const uint32_t l01 = __byte_perm(u.x, u.y, 0x5140), l23 = __byte_perm(u.z, u.w, 0x5140);
      const uint32_t h01 = __byte_perm(u.x, u.y, 0x7362), h23 = __byte_perm(u.z, u.w, 0x7362);
      p[0][q] = __byte_perm(l01, l23, 0x5410);
      p[1][q] = __byte_perm(l01, l23, 0x7632);
      p[2][q] = __byte_perm(h01, h23, 0x5410);
      p[3][q] = __byte_perm(h01, h23, 0x7632);
    }
    const size_t row = 4 * (col0 + c), kk = (size_t)k * n + s;
    uint8_t *dst = ub + ((row >> 7) * kbs + (kk >> 7)) * 16384 + (row & 127) * 128 + (kk & 127);
#pragma unroll
    for (int b = 0; b < 4; ++b) *reinterpret_cast<uint4 *>(dst + 128 * b) = make_uint4(p[b][0], p[b][1], p[b][2], p[b][3]);
  }
}

}  // namespace alto
