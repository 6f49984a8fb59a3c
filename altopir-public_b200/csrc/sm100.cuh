// sm100.cuh -- thin inline-PTX layer for the Blackwell (sm_100a) primitives the answer engine uses:
// mbarriers with bounded waits, TMA tiled loads, tcgen05 TMEM allocation, tcgen05.mma kind::i8, tcgen05.commit
// and tcgen05.ld.  Every wait in this file gives up after ALTO_WAIT_NS nanoseconds of wall time, records an error
// code in the batch's error word (waits.cuh) and returns false, so that a lost arrival can never hang the GPU.
#pragma once
#include <cuda.h>
#include <cstdint>

#include "waits.cuh"

#ifndef ALTO_WAIT_NS
#define ALTO_WAIT_NS 2000000000ull  // 2 s: far above any legitimate wait (a whole batch takes milliseconds)
#endif

namespace alto {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// True in one lane of a converged warp, the same one every time: the MMAs and the commits that track them are one
// thread's.  The issuing warps loop and wait as a whole and issue behind this test, so that descriptors, coordinates and
// barrier addresses stay uniform; issued from a `lane == 0` branch, an MMA cost 88 cycles of the warp instead of at most
// 45, and the 1 GiB pack of 128 clients took 507 us in wide units instead of 383.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// ------------------------------------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// CLUSTER: acquire what other CTAs of the cluster stored before their arrivals.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
// Waits for the phase with the given parity to complete.  Returns false (and records `code` in *err) after
// ALTO_WAIT_NS of wall time, or at once when another role of this CTA has already recorded an error.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t *err, uint32_t code,
                                          volatile int *bail) {
  if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
  const uint64_t t0 = globaltimer();
  for (uint32_t it = 0;; ++it) {
    if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
    if ((it & 63u) == 63u) {
      if (*bail) return false;
      if (globaltimer() - t0 > ALTO_WAIT_NS) {
        record_error(err, code);
        *bail = 1;
        return false;
      }
    }
  }
}

// The same for a converged warp, which waits and goes on as one: false for every lane when any lane gave up, so that no
// lane is left at a warp-wide instruction after a timeout.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, uint32_t *err, uint32_t code,
                                               volatile int *bail) {
  return __all_sync(0xffffffffu, mbar_wait<CLUSTER>(bar, parity, err, code, bail));
}

// ------------------------------------------------------------------------------------------------ TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
// 2-D tiled load of a box into shared memory; completion is signalled on `bar` as transaction bytes.
// x (the innermost coordinate, in bytes for u8 data) is always a multiple of 128 here.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x, int32_t y,
                                            uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "l"(cache_hint)
      : "memory");
}
// 3-D tiled load (x innermost, in bytes; z selects a record chunk of the scan operands).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x, int32_t y,
                                            int32_t z, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z), "l"(cache_hint)
      : "memory");
}
// 4-D tiled load of one tile of a tile-contiguous operand: coordinates (0, 0, k block, 128-row tile), the box being
// the whole 128 x 128-byte tile (16 KB contiguous in global memory).
__device__ __forceinline__ void tma_load_tile(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t kb,
                                              int32_t mt, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(kb), "r"(mt), "l"(cache_hint)
      : "memory");
}
// 4-D load of a few rows of consecutive tiles: coordinates (0, first row in the tile, first k block, 128-row tile).
__device__ __forceinline__ void tma_load_rows(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t row, int32_t kb,
                                              int32_t mt, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], %7;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(kb), "r"(mt), "l"(cache_hint)
      : "memory");
}
// L2 cache policies for the loads (createpolicy fractions of 1.0).
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// ------------------------------------------------------------------------------------------------ tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major operand tile written by TMA with 128-byte swizzling: rows of 128
// bytes, 8-row swizzle atoms of 1024 bytes stacked at a 1024-byte stride.  Fields: start address >> 4 in bits
// [0,14), leading byte offset >> 4 in [16,30) (unused by swizzled K-major layouts, set to 1), stride byte offset
// >> 4 in [32,46), descriptor version 1 in [46,48), base offset 0 (tiles are 1024-byte aligned), layout type 2
// (128-byte swizzle) in [61,64).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) |
         ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

// Shared-memory matrix descriptor of an MN-major operand without swizzling: core matrices of 8 (K) x 16 bytes (M or N), 128
// bytes each, the next 16 along M or N at `stride` bytes and the next 8 along K at `leading` bytes.  Layout type 0.
__device__ __forceinline__ uint64_t desc_mn_plain(uint32_t smem_addr, uint32_t leading, uint32_t stride) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(leading >> 4) << 16) | ((uint64_t)(stride >> 4) << 32) |
         ((uint64_t)1u << 46);
}

// Instruction descriptor of tcgen05.mma kind::i8 with unsigned 8-bit A and B (both K-major), signed 32-bit
// accumulator, no saturation, M = 128: D format S32 in bits [4,6), A/B formats 0 (u8) in [7,10) and [10,13),
// N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t idesc_u8u8_s32(uint32_t n) {
  return (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, 128 x N x 32 per instruction; issued by one thread.
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once every tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// Loads 16 consecutive 32-bit TMEM columns of this warp's 32 lanes (lane i of the warp reads TMEM lane
// base_lane + i).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 32 lanes x 32 columns: column j of this thread's lane into r[j].
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

}  // namespace alto

// ------------------------------------------------------------------------------------------------ CTA pairs
namespace alto {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The shared::cluster address of the same shared-memory object in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on an mbarrier of this CTA.
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Arrive on an mbarrier given by its shared::cluster address (possibly in the peer CTA).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Copies `bytes` (a multiple of 16, 16-byte aligned) of this CTA's shared memory to another CTA's (a shared::cluster
// address); their arrival counts as transaction bytes on that CTA's mbarrier.
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// TMA load into this CTA's shared memory whose completion is counted on the pair leader's mbarrier
// (bar_cluster is a shared::cluster address).  No multicast: each CTA loads only its own tile.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster, int32_t x,
                                                 int32_t y, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(x), "r"(y), "l"(cache_hint)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster, int32_t x,
                                                 int32_t y, int32_t z, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(x), "r"(y), "r"(z), "l"(cache_hint)
      : "memory");
}
__device__ __forceinline__ void tma_load_tile_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster,
                                                   int32_t kb, int32_t mt, uint64_t cache_hint) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(0), "r"(kb), "r"(mt), "l"(cache_hint)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Instruction descriptor of the pair MMA: u8 x u8 -> s32, both K-major, M = 256 (128 rows per CTA), N = n.
__host__ __device__ constexpr uint32_t idesc_pair_u8u8_s32(uint32_t n) {
  return (2u << 4) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}
// D[tmem of both CTAs] (+)= A[128 rows in each CTA] x B[n/2 rows in each CTA]^T, 256 x n x 32; leader thread only.
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the mbarrier at the same shared-memory offset in both CTAs of the pair once the leader's MMAs issued so
// far have completed.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  const uint16_t both = 0x3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::
                   "r"(bar),
               "h"(both)
               : "memory");
}

// The low word of desc_sw128 (address and leading offset); the high word is the same for every tile.
__device__ __forceinline__ uint32_t desc_lo_sw128(uint32_t smem_addr) { return (smem_addr >> 4) | (1u << 16); }
constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint64_t desc_of(uint32_t lo) {
  return (uint64_t)lo | ((uint64_t)kDescHiSw128 << 32);
}
// One 128-byte block of K: four pair MMAs on the tiles whose descriptors start at a_lo and b_lo; `accumulate` 0 clears D
// with the first.
__device__ __forceinline__ void mma_block_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                               uint32_t accumulate) {
  mma_i8_pair(d_tmem, desc_of(a_lo), desc_of(b_lo), idesc, accumulate);
#pragma unroll
  for (uint32_t kk = 1; kk < 4; ++kk) mma_i8_pair(d_tmem, desc_of(a_lo + 2 * kk), desc_of(b_lo + 2 * kk), idesc, 1u);
}

}  // namespace alto
