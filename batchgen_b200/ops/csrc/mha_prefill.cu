// Varlen causal multi-head attention for MLA prefill in the expanded (non-absorbed) form, on tcgen05.
//
// For long prompts the absorbed form (queries projected into the 576-wide latent space) costs 3.4x the
// FLOPs of plain attention over up-projected keys and values (192-wide keys = 128 nope + 64 rope, 128-wide
// values).  This kernel is the flash-attention forward for that shape:
//
//   S[q, k] = Q[q, 0:192] . K[k, 0:192]          (M = 128 queries, N = 64 keys; both K-major via TMA)
//   O[q, :] += P[q, k] . V[k, 0:128]             (M = 128, N = 128; V read N-major, P from TMEM)
//
// One CTA = one (256-query tile, head): two halves of 128 queries with softmax warps of their own, so that the tensor cores work for one half
// while the other's softmax runs, and each key / value tile is loaded once for both.  Query row i of the tile sees the first kv0 + i
// keys of its sequence's key range, which covers causal masking, cached context (kv0 > 1 for the first query) and the boundary to
// the next sequence in the packed batch with a single comparison.  A thread owns a query row (TMEM lane), so the online softmax
// needs no cross-thread reduction; the accumulator is rescaled only when the running maximum grew by more than 2^8.  P goes back over
// S in TMEM (two bf16 to a column) as the A operand of P.V.  K/V tiles flow through a 3-stage TMA ring; S of tile t+1 is issued before P.V of
// tile t.
//
// The warps of a half wait for nothing but their own tiles, so a fast one is up to a tile ahead of a slow one: it may store P of t+1 while the
// other still rescales O for t.  So P has a barrier for each S buffer: a warp's next arrival there needs S of t+2, which follows P.V of t and
// with it all four arrivals for t.  The end of P.V likewise: a warp that does not rescale waits for none but the last, two phases after what its
// last scores say is complete, where one barrier's parity is the same again.
//
// With one 128-query tile a CTA and P through shared memory, the product of S, the softmax and P.V took turns.  One softmax warp's exponentials
// take 512 of the tensor cores' 640 clocks for 128 queries x 64 keys.  128 heads: prompts of 2,048, 1,461, 874 and 1,000 tokens 654 -> 408 us
// (813 TFLOP/s), 1,536 tokens behind 5,000 1,023 -> 654 (1,110); 32 heads, 4,096 tokens 293 -> 195.  What is left is each CTA's start and end,
// some 4 us a tile, and the diagonal.
//
// Where the halves of all tiles find an SM each, a half is a CTA by itself (grid z): two in one CTA would take turns beside idle SMs.  Heads x
// tokens, one half a CTA / two / the kernel of one 128-query tile: 8 x 2,048 39 / 46 / 44 us, 1 x 4,096 59 / 77 / 72, 16 x 140 behind 4,000 66 / 80 / 78; past
// one round two halves win, 64 x 300 23 / 18 / 20, 8 x 4,096 92 / 84 / 94.
//
// Roles (384 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 4..7 and 8..11 softmax / epilogue of a half.
// All waits are bounded (common.cuh).
//
// Replaces (by behaviour): FA2/FA3 varlen prefill as dispatched by batchgen/attention/varlen_dispatch.py and
// prefill_attn_w8a16_prepacked (batchgen/models/deepseek/deepseekv3/wrappers.py:251-303).
#include "common.cuh"

namespace bg {
namespace mha {

constexpr int kDqk = 192, kDv = 128;
constexpr int kKvRow = 256;                      // per head in the kv_b projection output: 128 key-nope dims | 128 value dims
constexpr int BM = 128, BN = 64;
constexpr int kStages = 3;
constexpr int kThreads = 384;
constexpr int kQBytes = 3 * BM * 128;            // 48 KB, twice
constexpr int kKBytes = 3 * BN * 128;            // 24 KB
constexpr int kVBytes = 2 * BN * 128;            // 16 KB
constexpr int kTmemCols = 512;                   // each half: S (and P over it) 2 x 64, O 128
constexpr int kHalfCols = 256;

struct Work {
  int q_row0;    // first query row of the tile (rows of Q / out)
  int n_q;       // queries in the tile (<= 256)
  int k_row0;    // first key row of the sequence (rows of K / V)
  int kv0;       // keys visible to query 0 of the tile (>= 1)
};

struct Shared {
  uint64_t q_full;
  uint64_t kv_full[kStages];
  uint64_t kv_empty[kStages];
  uint64_t s_full[2][2];     // [half][buffer]
  uint64_t p_full[2][2];
  uint64_t o_done[2][2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(lbo >> 4) << 16;
  d |= static_cast<uint64_t>(sbo >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
__device__ __forceinline__ bool mbar_probe(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
  tmem_ld_32x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(v));
}
__global__ void __launch_bounds__(kThreads, 1)
mha_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                   const __grid_constant__ CUtensorMap tm_kpe, const Work* __restrict__ work,
                   __nv_bfloat16* __restrict__ out, int H, float scale_log2, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_buf = smem;
  uint8_t* k_buf = q_buf + 2 * kQBytes;
  uint8_t* v_buf = k_buf + kStages * kKBytes;
  Shared& ss = *reinterpret_cast<Shared*>(v_buf + kStages * kVBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ss.abort_flag;
  Work w = work[blockIdx.x];
  const int h = blockIdx.y;
  if (gridDim.z > 1) {                    // one half of the tile
    if (blockIdx.z > 0) {
      w.q_row0 += BM;
      w.kv0 += BM;
      w.n_q -= BM;
    }
    w.n_q = min(w.n_q, BM);
    if (w.n_q <= 0) return;
  }
  // key tiles that a half sees: up to its last query's
  const int tiles0 = (w.kv0 + min(w.n_q, BM) - 1 + BN - 1) / BN, tiles1 = w.n_q > BM ? (w.kv0 + w.n_q - 1 + BN - 1) / BN : 0;
  const int n_tiles = max(tiles0, tiles1);

  if (threadIdx.x == 0) {
    mbar_init(&ss.q_full, 1);
    for (int s = 0; s < kStages; ++s) { mbar_init(&ss.kv_full[s], 1); mbar_init(&ss.kv_empty[s], 1); }
    for (int x = 0; x < 2; ++x) {
      mbar_init(&ss.s_full[x][0], 1);
      mbar_init(&ss.s_full[x][1], 1);
      mbar_init(&ss.p_full[x][0], 4);
      mbar_init(&ss.p_full[x][1], 4);
      mbar_init(&ss.o_done[x][0], 1);
      mbar_init(&ss.o_done[x][1], 1);
    }
    ss.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&ss.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(&ss.q_full, tiles1 > 0 ? 2 * kQBytes : kQBytes);
      for (int x = 0; x < (tiles1 > 0 ? 2 : 1); ++x)
        for (int c = 0; c < 3; ++c)
          tma_load_2d(q_buf + x * kQBytes + c * BM * 128, &tm_q, &ss.q_full, h * kDqk + c * 64, w.q_row0 + x * BM);
      bool ok = true;
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t % kStages;
        if (!mbar_wait(&ss.kv_empty[s], ((t / kStages) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
        mbar_expect_tx(&ss.kv_full[s], kKBytes + kVBytes);
        const int krow = w.k_row0 + t * BN;
        // keys: 128 "nope" dims of this head out of the kv_b projection + the 64 roped dims shared by all heads
        for (int c = 0; c < 2; ++c) tma_load_2d(k_buf + s * kKBytes + c * BN * 128, &tm_kv, &ss.kv_full[s], h * kKvRow + c * 64, krow);
        tma_load_2d(k_buf + s * kKBytes + 2 * BN * 128, &tm_kpe, &ss.kv_full[s], 0, krow);
        for (int c = 0; c < 2; ++c) tma_load_2d(v_buf + s * kVBytes + c * BN * 128, &tm_kv, &ss.kv_full[s], h * kKvRow + 128 + c * 64, krow);
      }
      if (ok) {
        const int n = n_tiles < kStages ? n_tiles : kStages;
        for (int j = n_tiles - n; j < n_tiles; ++j)
          if (!mbar_wait(&ss.kv_empty[j % kStages], (j / kStages) & 1, abort_flag, kTimeoutProducer)) break;
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = idesc_bf16(BM, BN, 0);
      constexpr uint32_t idesc_pv = idesc_bf16(BM, kDv, 1);
      bool ok = mbar_wait(&ss.q_full, 0, abort_flag, kTimeoutMma);
      auto keys = [&](int t) { return mbar_wait(&ss.kv_full[t % kStages], (t / kStages) & 1, abort_flag, kTimeoutMma); };
      auto issue_s = [&](int x, int t) {
        tc_fence_after();
        const int s = t % kStages;
        const uint32_t tm_s = tmem_base + x * kHalfCols + (t & 1) * BN;
        for (int c = 0; c < 3; ++c) {
          const uint64_t adesc = make_smem_desc_sw128(smem_u32(q_buf + x * kQBytes + c * BM * 128));
          const uint64_t bdesc = make_smem_desc_sw128(smem_u32(k_buf + s * kKBytes + c * BN * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16(tm_s, adesc + 2 * k, bdesc + 2 * k, idesc_s, (c | k) ? 1u : 0u);
        }
        tc_commit(&ss.s_full[x][t & 1]);
      };
      ok = ok && keys(0);
      if (ok) issue_s(0, 0);
      if (ok && tiles1 > 0) issue_s(1, 0);
      for (int t = 0; ok && t < n_tiles; ++t) {
        // S of a half's next tile before its P.V of this one, unless the keys are still on their way
        const bool ready = t + 1 < n_tiles && mbar_probe(&ss.kv_full[(t + 1) % kStages], ((t + 1) / kStages) & 1);
        const int s = t % kStages;
        const uint32_t v_base = smem_u32(v_buf + s * kVBytes);
        for (int x = 0; ok && x < 2; ++x) {
          const int mine = x ? tiles1 : tiles0;
          if (t >= mine) continue;
          if (ready && t + 1 < mine) issue_s(x, t + 1);
          if (!mbar_wait(&ss.p_full[x][t & 1], (t >> 1) & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tm_p = tmem_base + x * kHalfCols + (t & 1) * BN, tm_o = tmem_base + x * kHalfCols + 2 * BN;
#pragma unroll
          for (int j = 0; j < BN / 16; ++j)
            mma_f16_ta(tm_o, tm_p + 8 * j, desc_mn_sw128(v_base + j * 2048, BN * 128, 1024), idesc_pv, (t > 0 || j > 0) ? 1u : 0u);
          tc_commit(&ss.o_done[x][t & 1]);
        }
        if (!ok) break;
        tc_commit(&ss.kv_empty[s]);
        if (!ready && t + 1 < n_tiles) {
          ok = keys(t + 1);
          for (int x = 0; ok && x < 2; ++x)
            if (t + 1 < (x ? tiles1 : tiles0)) issue_s(x, t + 1);
        }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ softmax / correction / epilogue of a half: thread = query row
    const int quad = warp & 3, x = (warp - 4) >> 2, mine = x ? tiles1 : tiles0;
    const int r = x * BM + quad * 32 + lane;
    const uint32_t base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + x * kHalfCols, tm_o = base + 2 * BN;
    const int visible = w.kv0 + r, all_see = w.kv0 + x * BM + quad * 32;      // keys this row may see, keys every row of the warp may see
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int t = 0; ok && t < mine; ++t) {
      if (!__all_sync(0xffffffffu, mbar_wait(&ss.s_full[x][t & 1], (t >> 1) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
      tc_fence_after();
      const uint32_t tm_s = base + (t & 1) * BN;
      uint32_t sv[64];
      tmem_ld32(tm_s, sv);
      tmem_ld32(tm_s + 32, sv + 32);
      tmem_ld_wait();
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (all_see < (t + 1) * BN) {             // masked after the scale, which may be zero or negative
        const int n_ok = visible - t * BN;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const float v = j < n_ok ? __uint_as_float(sv[j]) * scale_log2 : -INFINITY;
          sv[j] = __float_as_uint(v);
          mx[j & 3] = fmaxf(mx[j & 3], v);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          const float2 v = __fmul2_rn(make_float2(__uint_as_float(sv[j]), __uint_as_float(sv[j + 1])), make_float2(scale_log2, scale_log2));
          sv[j] = __float_as_uint(v.x);
          sv[j + 1] = __float_as_uint(v.y);
          mx[j & 2] = fmaxf(mx[j & 2], v.x);
          mx[(j & 2) + 1] = fmaxf(mx[(j & 2) + 1], v.y);
        }
      }
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const bool grow = mt > m_run + 8.f;
      const float m_new = grow ? mt : m_run;
      const float alpha = (grow && m_run != -INFINITY) ? ex2(m_run - m_new) : 1.f;
      if (t > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // P.V of the tile before this one (that of earlier ones was complete when S of this tile was)
        if (!__all_sync(0xffffffffu, mbar_wait(&ss.o_done[x][(t - 1) & 1], ((t - 1) >> 1) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t ov[32];
          tmem_ld_32x32(tm_o + c * 32, ov);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * alpha);
          tmem_st_32x32(tm_o + c * 32, ov);
        }
      }
      float lsum = 0.f;
      const float neg_m = (m_new == -INFINITY) ? 0.f : -m_new;
      uint32_t pk[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float2 e = __fadd2_rn(make_float2(__uint_as_float(sv[2 * j]), __uint_as_float(sv[2 * j + 1])), make_float2(neg_m, neg_m));
        const __nv_bfloat162 o = __floats2bfloat162_rn(ex2(e.x), ex2(e.y));
        pk[j] = *reinterpret_cast<const uint32_t*>(&o);
        lsum += __uint_as_float(pk[j] << 16) + __uint_as_float(pk[j] & 0xffff0000u);
      }
      tmem_st_32x32(tm_s, pk);
      tmem_st_wait();
      l_run = l_run * alpha + lsum;
      m_run = m_new;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ss.p_full[x][t & 1]);
    }
    if (ok && mine > 0) ok = __all_sync(0xffffffffu, mbar_wait(&ss.o_done[x][(mine - 1) & 1], ((mine - 1) >> 1) & 1, abort_flag, kTimeoutEpilogue));
    if (ok && mine > 0) {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      __nv_bfloat16* orow = out + ((size_t)(w.q_row0 + r) * H + h) * kDv;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32(tm_o + c * 32, ov);
        tmem_ld_wait();
        if (r < w.n_q) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            __align__(16) __nv_bfloat162 o[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              o[q] = __floats2bfloat162_rn(__uint_as_float(ov[j + 2 * q]) * inv, __uint_as_float(ov[j + 2 * q + 1]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + j) = *reinterpret_cast<const uint4*>(o);
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
  if (threadIdx.x == 0 && ss.abort_flag != 0 && status != nullptr) atomicMax(status, ss.abort_flag);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}
static int make_map(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t row_stride,
                    uint32_t box_rows) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {row_stride * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

}  // namespace mha
}  // namespace bg

extern "C" {

// q [Tq, H, 192] (nope | roped pe), kv [Tk, H, 256] (key nope | value: the kv_b projection of the latent rows),
// kpe [Tk, kpe_stride] (roped shared key part in the first 64 columns), out [Tq, H, 128]: bf16.
// work: n_work x 4 ints (q_row0, n_q, k_row0, kv0), one CTA per work item and head, or two where all of them fit the SMs at once.
int bg_mha_prefill(const void* q, const void* kv, const void* kpe, long long kpe_stride, void* out, const int* work,
                   int n_work, int Tq, int Tk, int H, float scale, int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::mha;
  if (n_work <= 0 || H <= 0) return 0;
  if (kpe_stride % 8 != 0) return -1;
  CUtensorMap tq, tk, tv;
  if (make_map(&tq, q, (uint64_t)H * kDqk, (uint64_t)Tq, (uint64_t)H * kDqk, BM) != 0) return -10;
  if (make_map(&tk, kv, (uint64_t)H * kKvRow, (uint64_t)Tk, (uint64_t)H * kKvRow, BN) != 0) return -11;
  if (make_map(&tv, kpe, 64, (uint64_t)Tk, (uint64_t)kpe_stride, BN) != 0) return -12;
  static bg::DeviceOnce attr_set;
  const size_t smem = 2 * kQBytes + kStages * (kKBytes + kVBytes) + sizeof(Shared) + 1024;
  if (!bg::ensure_dynamic_smem(mha_prefill_kernel, smem, attr_set)) return -13;
  dim3 grid(n_work, H, 2ll * n_work * H <= num_sms ? 2 : 1);
  mha_prefill_kernel<<<grid, kThreads, smem, stream>>>(tq, tk, tv, reinterpret_cast<const Work*>(work),
                                                       reinterpret_cast<__nv_bfloat16*>(out), H,
                                                       scale * 1.4426950408889634f, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -14;
}

}  // extern "C"
