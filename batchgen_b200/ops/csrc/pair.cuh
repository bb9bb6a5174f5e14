// Two CTAs of a cluster on one product: tcgen05 with cta_group::2 (each CTA holds half of M in its TMEM, half of A and half of B in its
// shared memory), and an epilogue that stores D^T tiles as rows of D.
//
// A K step of 128 bytes of a 256 x 256 product stages 32 KB in each CTA, 48 KB where one CTA works on 128 x 256: operands cross the L2 -> SM
// fabric and shared memory that much less often.  Loads are plain per-CTA tile loads whose bytes count on the leader's barrier.
#pragma once
#include "common.cuh"

namespace bg {
namespace pair {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// all threads of both CTAs
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the leader's copy of a shared-memory object of this CTA
__device__ __forceinline__ uint32_t leader_addr(const void* p) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(out) : "r"(smem_u32(p)));
  return out;
}
// Arrive on a barrier in either CTA, for a thread there that waits with wait_cluster.  At cluster scope, for the waiter is in another CTA; relaxed, for what
// is handed over is TMEM, whose reads tcgen05.fence::before_thread_sync orders before the arrival, and nothing that this thread stored: a release
// would also wait for the tile's stores to land (64 matrices of 2,304 x 512 with 300 rows 84 us, 66 so).
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// mbar_wait for a barrier of this CTA on which the other CTA's threads, loads or products arrive too
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int why) {
  uint64_t t0 = 0;
  for (uint32_t i = 0;; ++i) {
    if (try_wait_cluster(bar, parity)) return true;
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      if ((i & 0xFFFFu) == 0xFFFFu) {
        const uint64_t t = global_timer_ns();
        if (t0 == 0) t0 = t;
        else if (t - t0 > kWaitBudgetNs) break;
      }
    }
  }
  if (*abort_flag == 0) *abort_flag = why;
  return false;
}

// a tile load into this CTA whose bytes count on the barrier at shared::cluster address `bar`, in either CTA
__device__ __forceinline__ void load_2d(void* smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ void alloc(uint32_t* smem_holder, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_holder)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrive on the barrier at this offset in both CTAs once the products issued so far have completed
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 16 lanes x 32 columns: v[4 j + e] is lane t / 4, column 8 j + 2 (t % 4) + e for e < 2, and lane t / 4 + 8, the same columns, for e - 2
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&b);
}
// eight outputs of a row, `left` of them at most, in one piece where `wide` (rows on 16-byte boundaries)
__device__ __forceinline__ void store_8(__nv_bfloat16* dst, const uint32_t (&w)[4], int left, bool wide) {
  if (wide && left >= 8) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < left) reinterpret_cast<uint16_t*>(dst)[i] = static_cast<uint16_t>(w[i / 2] >> (16 * (i & 1)));
  }
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
// 32 outputs x 8 tokens of a warp, x[b] the outputs 8 b + t / 4 of tokens 2 (t % 4) and the next: thread t stores the outputs 8 (t % 4) .. of
// token t / 4 at row[0 .. 8) as store_8 does (row: the thread's token, its first output; null: token not present)
__device__ __forceinline__ void store_32x8(const uint32_t (&x)[4], __nv_bfloat16* row, int left, bool wide) {
  const bool e = threadIdx.x & 1, f = threadIdx.x & 2;
  uint32_t m[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) m[b] = transpose_8x8(x[b]);          // token t / 4, outputs 8 b + 2 (t % 4) and the next
  // block t % 4 from all four threads of the token
  const uint32_t a0 = e ? m[1] : m[0], a1 = e ? m[3] : m[2];
  const uint32_t r0 = __shfl_xor_sync(0xffffffffu, e ? m[0] : m[1], 1), r1 = __shfl_xor_sync(0xffffffffu, e ? m[2] : m[3], 1);
  const uint32_t k0 = f ? a1 : a0, k1 = f ? r1 : r0;
  const uint32_t t0 = __shfl_xor_sync(0xffffffffu, f ? a0 : a1, 2), t1 = __shfl_xor_sync(0xffffffffu, f ? r0 : r1, 2);
  const uint32_t x0 = e ? k1 : k0, x1 = e ? k0 : k1, y0 = e ? t1 : t0, y1 = e ? t0 : t1;
  const uint4 o = f ? make_uint4(y0, y1, x0, x1) : make_uint4(x0, x1, y0, y1);
  if (row == nullptr) return;
  const uint32_t w[4] = {o.x, o.y, o.z, o.w};
  store_8(row, w, left, wide);
}

}  // namespace pair
}  // namespace bg
