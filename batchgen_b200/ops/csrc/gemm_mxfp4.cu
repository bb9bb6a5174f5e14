// 4-bit-weight GEMM (W4A16): bf16 activations x e2m1 weights with one e8m0 scale per 32 (MXFP4), or x offset-binary int4 weights with
// one bf16 scale per 32 (INT4); dense and ragged grouped (per-expert), on tcgen05 tensor cores.
//
//   D[m, n] = sum_k A[m, k] * ( e2m1(Wq[n, k]) * 2^(Ws[n, k / 32] - 127) )
//
// The packed weights stay 4-bit all the way from HBM into shared memory (decode is bound by weight bytes).  Weights are the MMA's M side
// and its operand in TMEM (D^T = W . X^T): a thread owns a weight row, expands 64 weights of it in registers and stores them to its TMEM
// lane, 32 columns a K step, so the expanded weights take no shared memory, no swizzle and no proxy fence.  Tokens are the N side, in
// tiles of up to 192 rows cut evenly from a segment and rounded up to 16: a decode step's dozen tokens cost a 16-wide product
// instead of a 128-row one, and a prompt expert's 150 tokens meet each weight once.
//
// A pair of nibbles becomes a pair of bf16 by a byte selection, one product for both shifts, a mask and one packed product: e2m1 bits placed
// at bit 6 of a bf16 are the value times 2^-126, subnormals included, and the product with 2^126 times the scale is exact.  128 experts of
// 6,144 x 2,880 and of 2,880 x 3,072, four a token, cold weights, against four warps that converted, multiplied in fp32 and rounded, with
// shared-memory operands and 128-row token tiles: one token 59 and 36 us -> 35 and 21, 160 tokens 997 and 504 -> 546 and 286 (184 and 92 at copy
// bandwidth), 4,650 tokens 1,864 and 945 -> 731 and 374.  Bound by the latency of a step's chain (expansion, TMEM store, product): some 520
// clocks at 160 tokens, issue slots 59 % and the integer pipe 54 % busy.
// MXFP4 products of up to 80 rows a segment without the fused SiLU go to gemm_mxfp4_block.cu (160 tokens 287 and 176 us); from there on the expanded
// form is ahead, and int4 weights, whose scales are not powers of two, stay here.
//
// Roles (736 threads, one CTA per SM, persistent over tiles):
//   warp 0       TMA producer of the token tiles (swizzled), 6 stages
//   warp 1       TMEM allocator + tcgen05.mma issuer
//   warps 2..5   epilogue (thread = weight row), optional SiLU(gate) * up on interleaved rows
//   warps 6..21  weight expansion, four groups of four warps on K steps in turn, a TMEM slot each (two groups: 15 % slower)
//   warp 22      TMA producer of the packed weights, 4 stages of 256 columns (whole 128-byte lines of a row)
//
// Replaces (by behaviour): the Marlin-tile MXFP4 grouped kernels
// batchgen_kernels/src/moe/mxfp4/marlin_grouped_gemm.cu (v1/v2/v3), the LUT-dequant WGMMA kernels of
// GPT-OSS, and the load-time dequantisers batchgen_kernels/src/moe/mxfp4/mxfp4_dequant*.cu; weight
// layout per batchgen/models/moonshotai/kimi_linear/k3/mxfp4_layout.py:37-38,179-182 (e2m1 pairs,
// low nibble first, e8m0 per 32).
#include <cuda_fp4.h>

#include "common.cuh"
#include "token_tiles.cuh"
#include "w4_steps.h"

namespace bg {
namespace mx {

constexpr int BW = 128;                   // weight rows of a tile (MMA M)
constexpr int BT = 192;                   // most tokens of a tile (MMA N)
constexpr int kBox = 32;                  // token rows of one TMA box
constexpr int BK = 64;                    // elements of K per step (one 128-byte swizzle atom of bf16)
constexpr int kXStages = 6, kQStages = 4;
constexpr int kThreads = 32 * (7 + 4 * kGroups);
constexpr int kTmemCols = 512;            // two accumulators of BT columns, kGroups weight operands of 32
constexpr int kSlotCol = 2 * BT;
constexpr int kMaxGroups = 1024;
constexpr int kXBytes = BT * BK * 2;      // 24 KB
constexpr int kQBytes = BW * 128;         // 16 KB packed: 128 bytes of every row, a step for each group
constexpr int EPI_STORE = 0;
constexpr int EPI_SILU_MUL = 1;
constexpr int QMODE_MXFP4 = 0;            // e2m1 values, one e8m0 scale per 32
constexpr int QMODE_INT4 = 1;             // offset-binary int4 (value = q - 8), one bf16 scale per 32

struct Params {
  const uint8_t* ws;     // [groups * N, K / 32] e8m0, or bf16
  __nv_bfloat16* D;      // [M, ldd]
  int ldd;
  const int* offsets;    // [groups + 1] segment starts; null = dense
  const int* counts;     // [groups] rows present in a segment, or null: all of it
  int groups, M, N, K;
  int* status;
};

struct Shared {
  uint64_t x_full[kXStages], x_empty[kXStages];
  uint64_t q_full[kQStages], q_empty[kQStages];      // empty: every expansion warp has read its part of the stage
  uint64_t w_full[kGroups], w_empty[kGroups];        // weight operands in TMEM, one of each group
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  Segments<kMaxGroups> seg;
  float xch[2][32][32];                              // SiLU epilogue: the up rows' values of 32 tokens
};

__device__ __forceinline__ float e8m0_to_float(uint32_t e) {
  // 2^(e - 127); e = 0 is 2^-127 (a subnormal float), e = 255 is NaN in the format and never stored
  return e == 0u ? __uint_as_float(0x00400000u) : __uint_as_float(e << 23);
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// bytes of {a: 0 .. 3, b: 4 .. 7}; a selector with its top bit set repeats the byte's sign bit (zero here: nibbles in bytes)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// 8 weights of one 32-bit word (low nibble first) -> 4 pairs of bf16, times f (both halves; FOLDED: MXFP4 scales times 2^126).
// The integer pipe is the limit (two clocks an instruction): a selection and a mask a pair, three more a word; both shifts are one product.
template <int QMODE, bool FOLDED>
__device__ __forceinline__ void expand8(uint32_t w, uint32_t f, uint32_t* o) {
  const uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const uint32_t y = prmt(lo, hi, b | ((8 | b) << 4) | ((4 + b) << 8) | ((8 | b) << 12));      // a weight's nibble in each half
    if (QMODE == QMODE_INT4) {
      o[b] = mul_bf16x2(sub_bf16x2(y | 0x43004300u, 0x43084308u), f);                    // 128 + q, less 136: both exact
    } else {
      uint32_t v = (y * 0x1040u) & 0x81C081C0u;                                          // magnitude at bit 6 up, sign at bit 15
      if (!FOLDED) v = mul_bf16x2(v, 0x7E807E80u);                                       // 2^126: the e2m1 value itself
      o[b] = mul_bf16x2(v, f);
    }
  }
}

template <int EPI, int QMODE>
__global__ void __launch_bounds__(kThreads, 1)
w4_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmQ, Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x_tiles = smem;
  uint8_t* q_tiles = smem + kXStages * kXBytes;
  Shared& ss = *reinterpret_cast<Shared*>(q_tiles + kQStages * kQBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
  const int KB = p.K / BK;
  const int n_tiles = (p.N + BW - 1) / BW;
  volatile int* abort_flag = &ss.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kXStages; ++s) { mbar_init(&ss.x_full[s], 1); mbar_init(&ss.x_empty[s], 1); }
    for (int s = 0; s < kQStages; ++s) { mbar_init(&ss.q_full[s], 1); mbar_init(&ss.q_empty[s], 4 * kGroups); }
    for (int s = 0; s < kGroups; ++s) { mbar_init(&ss.w_full[s], 4); mbar_init(&ss.w_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ss.tmem_full[b], 1); mbar_init(&ss.tmem_empty[b], 4); }
    ss.abort_flag = 0;
    mbar_fence_init();
  }
  if (p.offsets != nullptr) load_segments<BT>(ss.seg, p.offsets, p.counts, p.groups);
  if (warp == 1) {
    tmem_alloc(&ss.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;
  TokenWalker<BT, BW, kMaxGroups> walk(p.offsets != nullptr ? &ss.seg : nullptr, p.groups, n_tiles, p.M);
  TokenTile t;
  uint32_t it = 0, acc = 0;
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------ token tiles
    if (elect_one()) {
      tma_prefetch_desc(&tmX);
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x) {
        const int boxes = (tile_cols(t) + kBox - 1) / kBox;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kXStages;
          if (!mbar_wait(&ss.x_empty[s], ((it / kXStages) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
          mbar_expect_tx(&ss.x_full[s], boxes * kBox * BK * 2);
          for (int b = 0; b < boxes; ++b)
            tma_load_2d(x_tiles + s * kXBytes + b * kBox * BK * 2, &tmX, &ss.x_full[s], kb * BK, t.m0 + b * kBox);
        }
      }
      if (ok) {
        const uint32_t n = it < (uint32_t)kXStages ? it : (uint32_t)kXStages;
        for (uint32_t j = it - n; j < it; ++j)
          if (!mbar_wait(&ss.x_empty[j % kXStages], (j / kXStages) & 1, abort_flag, kTimeoutProducer)) break;
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
      }
    }
  } else if (warp == 6 + 4 * kGroups) {
    // ------------------------------------------------------------ packed weights
    if (elect_one()) {
      tma_prefetch_desc(&tmQ);
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x) {
        const int row = t.g * p.N + t.n0;
        for (int kb = 0; kb < KB; kb += kGroups, ++it) {             // columns past K / 2 are filled with zeros
          const int s = it % kQStages;
          if (!mbar_wait(&ss.q_empty[s], ((it / kQStages) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
          mbar_expect_tx(&ss.q_full[s], kQBytes);
          tma_load_2d(q_tiles + s * kQBytes, &tmQ, &ss.q_full[s], kb * (BK / 2), row);
        }
      }
      if (ok) {
        const uint32_t n = it < (uint32_t)kQStages ? it : (uint32_t)kQStages;
        for (uint32_t j = it - n; j < it; ++j)
          if (!mbar_wait(&ss.q_empty[j % kQStages], (j / kQStages) & 1, abort_flag, kTimeoutProducer)) break;
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
        const int buf = acc & 1;
        const uint32_t idesc = make_idesc(BW, tile_cols(t), 1, 1);   // bf16 x bf16 -> fp32
        if (!mbar_wait(&ss.tmem_empty[buf], ((acc >> 1) & 1) ^ 1, abort_flag, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kXStages, slot = step_group(kb);
          if (!mbar_wait(&ss.x_full[s], (it / kXStages) & 1, abort_flag, kTimeoutMma) ||
              !mbar_wait(&ss.w_full[slot], slot_use(KB, acc, kb) & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          const uint64_t bdesc = make_smem_desc_sw128(smem_u32(x_tiles + s * kXBytes));
          const uint32_t w = tmem_base + kSlotCol + slot * 32;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            mma_f16_ta(tmem_base + buf * BT, w + 8 * k, bdesc + 2 * k, idesc, (kb | k) ? 1u : 0u);
          tc_commit(&ss.x_empty[s]);
          tc_commit(&ss.w_empty[slot]);
        }
        if (ok) tc_commit(&ss.tmem_full[buf]);
      }
    }
  } else if (warp >= 6) {
    // ------------------------------------------------------------ weight expansion: groups of 128 threads take steps in turn
    const int group = (warp - 6) >> 2;
    const int r = quad * 32 + lane;          // weight row within the tile
    constexpr int kScaleBytes = QMODE == QMODE_INT4 ? 2 : 1;
    const int sk = (p.K / 32) * kScaleBytes;                     // scale bytes per weight row
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint32_t stage = 0;                      // stages of packed weights so far
    for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
      const uint8_t* srow = p.ws + (size_t)(t.g * p.N + min(t.n0 + r, p.N - 1)) * sk;
      // the two scales of a 64-wide K step: 2 bytes (e8m0) or 4 bytes (bf16)
      auto load_scales = [&](int kb) -> uint32_t {
        if (kb >= KB) return 0u;
        return QMODE == QMODE_INT4 ? *reinterpret_cast<const uint32_t*>(srow + 4 * kb)
                                   : static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(srow + 2 * kb));
      };
      uint32_t sc[3];                                                // three own steps ahead
#pragma unroll
      for (int i = 0; i < 3; ++i) sc[i] = load_scales(group + kGroups * i);
      for (int kb = group; kb < KB + group; kb += kGroups, ++stage) {
        const uint32_t s2 = sc[0];
        sc[0] = sc[1]; sc[1] = sc[2];
        sc[2] = load_scales(kb + 3 * kGroups);
        const int qs = stage % kQStages;
        if (!__all_sync(0xffffffffu, mbar_wait(&ss.q_full[qs], (stage / kQStages) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
        const uint8_t* q = q_tiles + qs * kQBytes + r * 128;          // 16-byte chunk c of row r lies at c ^ (r & 7)
        const uint4 q0 = *reinterpret_cast<const uint4*>(q + (((2 * group) ^ (r & 7)) << 4));
        const uint4 q1 = *reinterpret_cast<const uint4*>(q + (((2 * group + 1) ^ (r & 7)) << 4));
        __syncwarp();
        if (lane == 0) mbar_arrive(&ss.q_empty[qs]);
        if (kb >= KB) continue;                                      // the last stage may have steps past K
        uint32_t o[32];
        const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        if (QMODE == QMODE_INT4) {
          const uint32_t f0 = __byte_perm(s2, 0, 0x1010), f1 = __byte_perm(s2, 0, 0x3232);
#pragma unroll
          for (int c = 0; c < 8; ++c) expand8<QMODE, false>(words[c], c < 4 ? f0 : f1, o + 4 * c);
        } else {
          const uint32_t e0 = s2 & 0xFFu, e1 = s2 >> 8;
          // 2^(e - 1) is a bf16 up to e = 128 (a scale of 2); larger scales take the 2^126 by itself
          const bool folded = __all_sync(0xffffffffu, max(e0, e1) <= 128u);
          if (folded) {
            const uint32_t f0 = (e0 + 126u) << 7, f1 = (e1 + 126u) << 7;      // exponent field of 2^(e - 1)
#pragma unroll
            for (int c = 0; c < 8; ++c) expand8<QMODE, true>(words[c], c < 4 ? f0 | f0 << 16 : f1 | f1 << 16, o + 4 * c);
          } else {
            const uint32_t f0 = e0 == 0u ? 0x0040u : e0 << 7, f1 = e1 == 0u ? 0x0040u : e1 << 7;
#pragma unroll
            for (int c = 0; c < 8; ++c) expand8<QMODE, false>(words[c], c < 4 ? f0 | f0 << 16 : f1 | f1 << 16, o + 4 * c);
          }
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&ss.w_empty[group], (slot_use(KB, acc, kb) & 1) ^ 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
        tc_fence_after();
        tmem_st_32x32(tmem_base + lane_addr + kSlotCol + group * 32, o);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ss.w_full[group]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: thread = weight row, columns = tokens
    for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
      const int buf = acc & 1;
      const bool late = !mbar_wait(&ss.tmem_full[buf], (acc >> 1) & 1, abort_flag, kTimeoutEpilogue);
      // with barriers between the warps below, a warp that gives up alone would leave the others waiting for it
      if (EPI == EPI_SILU_MUL ? vote_any_128(late) : __any_sync(0xffffffffu, late)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * BT;
      const int n_tok = t.m_end - t.m0;
#pragma unroll 1
      for (int c = 0; c < n_tok; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(taddr + c, v);
        tmem_ld_wait();
        if (EPI == EPI_SILU_MUL) {
          // rows [64 b, 64 b + 32) are the gates of output columns n0 / 2 + 32 b .., the next 32 rows their up values
          const int b2 = quad >> 1;
          if (quad & 1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) ss.xch[b2][j][lane] = __uint_as_float(v[j]);
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
          const int col = t.n0 / 2 + b2 * 32 + lane;
          if (!(quad & 1) && col < p.N / 2) {
            __nv_bfloat16* dst = p.D + (size_t)(t.m0 + c) * p.ldd + col;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c + j < n_tok) dst[(size_t)j * p.ldd] = __float2bfloat16(silu(__uint_as_float(v[j])) * ss.xch[b2][j][lane]);
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
        } else {
          const int col = t.n0 + quad * 32 + lane;
          if (col < p.N) {
            __nv_bfloat16* dst = p.D + (size_t)(t.m0 + c) * p.ldd + col;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c + j < n_tok) dst[(size_t)j * p.ldd] = __float2bfloat16(__uint_as_float(v[j]));
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ss.tmem_empty[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
  if (threadIdx.x == 0 && ss.abort_flag != 0 && p.status != nullptr) atomicMax(p.status, ss.abort_flag);
}

// Load-time / debugging expansion of a packed tensor to bf16: one thread per 32-weight block.
__global__ void mxfp4_dequant_kernel(const uint8_t* __restrict__ wq, const uint8_t* __restrict__ ws,
                                     __nv_bfloat16* __restrict__ out, long long n_blocks) {
  const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_blocks) return;
  const float f = e8m0_to_float(ws[b]);
  const uint4 v = *reinterpret_cast<const uint4*>(wq + b * 16);
  const uint32_t words[4] = {v.x, v.y, v.z, v.w};
  __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(out + b * 32);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __half2_raw hr = __nv_cvt_fp4x2_to_halfraw2(
          static_cast<__nv_fp4x2_storage_t>((words[c] >> (8 * k)) & 0xFFu), __NV_E2M1);
      const float2 ff = __half22float2(*reinterpret_cast<const __half2*>(&hr));
      o[c * 4 + k] = __floats2bfloat162_rn(ff.x * f, ff.y * f);
    }
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

template <int EPI, int QMODE>
static int launch(const void* A, const void* Wq, const Params& p, int b_rows, int num_sms, cudaStream_t stream) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -10;
  CUtensorMap tmX, tmQ;
  {
    cuuint64_t dims[2] = {(cuuint64_t)p.K, (cuuint64_t)p.M};
    cuuint64_t strides[1] = {(cuuint64_t)p.K * 2};
    cuuint32_t box[2] = {BK, kBox};
    cuuint32_t es[2] = {1, 1};
    if (enc(&tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(A), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -11;
  }
  {
    cuuint64_t dims[2] = {(cuuint64_t)p.K / 2, (cuuint64_t)b_rows};
    cuuint64_t strides[1] = {(cuuint64_t)p.K / 2};
    cuuint32_t box[2] = {128, BW};
    cuuint32_t es[2] = {1, 1};
    if (enc(&tmQ, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(Wq), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -12;
  }
  static DeviceOnce attr_set;
  auto kern = w4_gemm_kernel<EPI, QMODE>;
  const size_t smem = kXStages * kXBytes + kQStages * kQBytes + sizeof(Shared) + 1024;
  if (!ensure_dynamic_smem(kern, smem, attr_set)) return -13;
  const int n_tiles = (p.N + BW - 1) / BW;
  long long grid = ((long long)p.M / BT + (p.offsets != nullptr ? p.groups : 1)) * n_tiles;      // an upper bound of the tiles
  if (grid > num_sms) grid = num_sms;
  if (grid < 1) grid = 1;
  kern<<<(int)grid, kThreads, smem, stream>>>(tmX, tmQ, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -14;
}

}  // namespace mx
}  // namespace bg

extern "C" {

// A: [M, K] bf16 row-major; Wq: [groups * N, K / 2] packed e2m1 (low nibble = even k); Ws: [groups * N, K / 32]
// e8m0; D: [M, ldd] bf16.  offsets == nullptr -> dense; counts: rows present in every segment, or null (rows past them stay
// undefined).  K % 64 == 0.  epi 1: rows of W interleaved (32 gate, 32 up), D gets N / 2 columns.  Returns 0 on a successful launch.
int bg_mxfp4_gemm(int epi, const void* A, const void* Wq, const void* Ws, void* D, int ldd, const int* offsets, const int* counts,
                  int groups, int M, int N, int K, int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::mx;
  if (M <= 0 || N <= 0) return 0;
  if (K % BK != 0 || groups > kMaxGroups || (epi == EPI_SILU_MUL && (N % 128) != 0) || (ldd % 8) != 0) return -1;
  if (offsets == nullptr) groups = 1;
  Params p;
  p.ws = reinterpret_cast<const uint8_t*>(Ws); p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd;
  p.offsets = offsets; p.counts = offsets != nullptr ? counts : nullptr; p.groups = groups; p.M = M; p.N = N; p.K = K; p.status = status;
  if (epi == EPI_SILU_MUL) return launch<EPI_SILU_MUL, QMODE_MXFP4>(A, Wq, p, groups * N, num_sms, stream);
  return launch<EPI_STORE, QMODE_MXFP4>(A, Wq, p, groups * N, num_sms, stream);
}

// INT4 W4A16 (group size 32): Wq packs two offset-binary nibbles per byte (low nibble = even k, value = q - 8),
// Ws: [groups * N, K / 32] bf16 scales.  Everything else as bg_mxfp4_gemm.
// Replaces (by behaviour): the Marlin / INT4 WGMMA grouped kernels of the Kimi-K2.5 family (W4A16, gs = 32).
int bg_int4_gemm(int epi, const void* A, const void* Wq, const void* Ws, void* D, int ldd, const int* offsets, const int* counts,
                 int groups, int M, int N, int K, int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::mx;
  if (M <= 0 || N <= 0) return 0;
  if (K % BK != 0 || groups > kMaxGroups || (epi == EPI_SILU_MUL && (N % 128) != 0) || (ldd % 8) != 0) return -1;
  if (offsets == nullptr) groups = 1;
  Params p;
  p.ws = reinterpret_cast<const uint8_t*>(Ws); p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd;
  p.offsets = offsets; p.counts = offsets != nullptr ? counts : nullptr; p.groups = groups; p.M = M; p.N = N; p.K = K; p.status = status;
  if (epi == EPI_SILU_MUL) return launch<EPI_SILU_MUL, QMODE_INT4>(A, Wq, p, groups * N, num_sms, stream);
  return launch<EPI_STORE, QMODE_INT4>(A, Wq, p, groups * N, num_sms, stream);
}

// out[i] = e2m1(wq[i]) * 2^(ws[i / 32] - 127), n elements (multiple of 32).
int bg_mxfp4_dequant(const void* wq, const void* ws, void* out, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 32 != 0) return -1;
  const long long nb = n / 32;
  bg::mx::mxfp4_dequant_kernel<<<(unsigned)((nb + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const uint8_t*>(wq), reinterpret_cast<const uint8_t*>(ws),
      reinterpret_cast<__nv_bfloat16*>(out), nb);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
