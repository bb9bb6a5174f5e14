// MXFP4 weights (e2m1, one e8m0 scale per 32) times bf16 tokens on the block-scaled tensor-core product, dense and ragged grouped.
//
//   D[m, n] = sum_k X[m, k] * e2m1(Wq[n, k]) * 2^(Ws[n, k / 32] - 127)
//
// Weights stay 4-bit up to the tensor cores (kind::mxf8f6f4 with e2m1 as the M side: sixteen nibbles in the first half of a 16-byte container of
// shared memory), and their scales are the product's own.  Tokens are the N side as two e4m3 parts (mx_parts.cuh), twice as many columns, whose two
// accumulators the epilogue adds.  The parts hold all eight bits of an element down to 2^-14 of the largest of its 32; a smaller one is off by up to
// 2^-22 of that largest, where bf16 operands lose nothing.  On activations the sums are closer to 64 bits than those of bf16 operands (relative error over
// 2,944 elements 5.7e-8 against 3.1e-7; tokens spread over 30 binades 1.7e-6 against 3.1e-6; normal numbers and gated activations: fewer outputs that are not
// the rounded 64-bit ones, 0 against 9e-5 and 5e-4 against 2e-3).  Further off are outputs whose weight is zero at an element that dwarfs the rest of its 32:
// rms of the bf16 outputs with one such element a row 2^12 above the others 1.667e-3 as without, 2^14 1.68e-3, 2^16 1.95e-3, 2^18 4.1e-3, 2^20 1.5e-2; with one in
// every 32 1.69e-3, 2.7e-3, 9.5e-3, 3.6e-2, 0.14; no difference where the weight is not zero.
//
// 128 experts of 6,144 x 2,880 and of 2,880 x 3,072, four a token, cold weights, against weights that are expanded to bf16 (gemm_mxfp4.cu): one token 41
// and 27 us -> 30 and 22, 16 tokens 239 and 130 -> 131 and 84, 160 tokens 553 and 291 -> 287 and 176 (186 and 93 at copy bandwidth), 1,500 tokens 573
// and 303 -> 461 and 278; 3,000 tokens (94 rows an expert) 605 and 328 -> 643 and 382, where the two columns a token cost more than the expansion and
// the caller keeps that kernel.  Bound by the threads that issue: a step's two scale copies, four products and commit take the MMA thread some 450
// clocks (a load's wait 70), where the weights' bytes take 360.  Token loads in the weights' warp cost 322 us instead of 287, weights as eight-byte
// copies of threads 414, tiles prefetched into L2 nothing.
//
// Roles (288 threads, one CTA per SM, persistent over tiles of 128 weight rows and up to BT - 8 tokens):
//   warp 0       TMA producer: weights, a tile's weight scales (rows are neighbours: one copy)
//   warp 1       TMEM allocator; copies scales to TMEM and issues the products
//   warps 2, 3   scales of every second K step (128 elements), as the 128 x 4 images that the copy takes
//   warps 4..7   epilogue
//   warp 8       TMA producer: token parts
#include "mx_parts.cuh"
#include "pair.cuh"
#include "token_tiles.cuh"

namespace bg {
namespace mxb {

constexpr int BW = 128;                   // weight rows of a tile (MMA M)
constexpr int BK = 128;                   // elements of K per stage: a byte each, one 128-byte swizzle atom
constexpr int kThreads = 288;
constexpr int kTmemCols = 512;
constexpr int kMaxGroups = 1024;
constexpr int kMaxStages = 8;
constexpr int kWBytes = BW * BK;          // 16 KB, half of it padding
constexpr int kWCopied = BW * BK / 2;     // what a copy counts
constexpr int kMaxShared = 227 * 1024;

// tokens of a tile as the product sees them: from an eight on, in eights (BT at most: the walker cuts tiles of BT - 8)
__device__ __forceinline__ int tile_tokens(const TokenTile& t) { return ((t.m_end + 7) & ~7) - (t.m0 & ~7); }

struct Params {
  const uint8_t* wq;     // [groups * N, K / 2]
  const uint8_t* ws;     // [groups * N, K / 32]
  const uint8_t* xp;     // [M / 8 rounded up][2][8][K] parts
  const uint8_t* xs;     // [K / 128 rounded up][M][4]
  __nv_bfloat16* D;      // [M, ldd]
  int ldd, wide;
  const int* offsets;    // [groups + 1] segment starts; null = dense
  const int* counts;     // [groups] rows present in a segment, or null: all of it
  int groups, M, N, K;
  int stages;
  int* status;
};

template <int BT>
struct Shared {
  static constexpr int kSfB = (2 * BT + 127) / 128 * 512;
  __align__(128) uint8_t sfa[kMaxStages][512];
  __align__(128) uint8_t sfb[kMaxStages][kSfB];
  uint64_t full[kMaxStages], empty[kMaxStages];    // full: both loads, a scale warp
  uint64_t raw_full[2], raw_empty[2];              // a tile's weight scales
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  Segments<kMaxGroups> seg;
};

struct Ring {                                      // stage and how often the ring came round
  int s = 0;
  uint32_t round = 0;
  __device__ __forceinline__ void next(int n, int stages) {
    s += n;
    if (s >= stages) { s -= stages; ++round; }
  }
};

__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 32 rows of 16 bytes, plain layout: 8-row groups 128 bytes apart
__device__ __forceinline__ uint64_t scale_desc(uint32_t a) {
  return static_cast<uint64_t>((a & 0x3FFFFu) >> 4) | static_cast<uint64_t>(128 >> 4) << 16 | static_cast<uint64_t>(128 >> 4) << 32 |
         static_cast<uint64_t>(1) << 46;
}
// 512 bytes of scales to four columns of every lane quadrant
__device__ __forceinline__ void copy_scales(uint32_t tmem, uint32_t smem) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(scale_desc(smem)) : "memory");
}
__device__ __forceinline__ void mma_block(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], %1, %2, %3, [%4], [%5], p;\n"
      "}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
      : "memory");
}
// e2m1 x e4m3 -> fp32, e8m0 scales, M = 128; bits 4 and 29: which of a column's four scales (0 here)
__device__ __forceinline__ uint32_t block_idesc(int n) {
  return 5u << 7 | static_cast<uint32_t>(n >> 3) << 17 | 1u << 23 | static_cast<uint32_t>(BW >> 4) << 24;
}
// bytes and both addresses are multiples of 16
__device__ __forceinline__ void copy_bulk(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ float e4m3_to_float(uint32_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(b), __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}
// A dot product that came out as NaN, term by term: parts do not carry an infinity.
__device__ __noinline__ float not_finite(const Params& p, int token, int wrow) {
  const uint8_t* a = p.xp + (size_t)mxp::part_row(token, 0) * p.K;
  const uint8_t* b = a + (size_t)8 * p.K;
  float sum = 0.f;
  for (int k = 0; k < p.K; ++k) {
    const int e = p.ws[(size_t)wrow * (p.K / 32) + k / 32];
    const uint32_t w = p.wq[(size_t)wrow * (p.K / 2) + k / 2] >> (4 * (k & 1)) & 15u, m = w & 7u;
    const float mag = e == 255 ? __int_as_float(0x7FC00000) : ldexpf(m < 2u ? 0.5f * m : 0.5f * (2u + (m & 1u)) * (1u << (m >> 1) >> 1), e - 127);
    float x;
    if ((a[k] & 0x7Fu) == mxp::kNan) x = __int_as_float(b[k] == 0 ? 0x7FC00000 : b[k] >> 7 ? 0xFF800000 : 0x7F800000);
    else x = ldexpf(e4m3_to_float(a[k]) + e4m3_to_float(b[k]) / (1 << mxp::kPartShift), p.xs[((size_t)(k / BK) * p.M + token) * 4 + k % BK / 32] - 127);
    sum = fmaf(x, w & 8u ? -mag : mag, sum);
  }
  return sum;
}

template <int BT>
__global__ void __launch_bounds__(kThreads, 1)
mxfp4_block_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmTail, const __grid_constant__ CUtensorMap tmX128,
                   const __grid_constant__ CUtensorMap tmX16, const Params p) {
  constexpr int kXBytes = 2 * BT * BK;
  constexpr int kAccCols = 224, kSfCol = 2 * kAccCols, kSfStep = 12;      // scale columns of a step: 4 + up to 8
  static_assert(kSfCol + 2 * kSfStep <= kTmemCols && 2 * BT <= kAccCols, "TMEM");
  using Sh = Shared<BT>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stages = p.stages;
  uint8_t* w_tiles = smem;
  uint8_t* x_tiles = smem + stages * kWBytes;
  uint8_t* raw = x_tiles + stages * kXBytes;           // two tiles' weight scales as they are stored
  const int sk = p.K / 32, raw_bytes = BW * sk;
  Sh& ss = *reinterpret_cast<Sh*>(raw + 2 * raw_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
  const int KB = (p.K + BK - 1) / BK;
  const int n_tiles = (p.N + BW - 1) / BW;
  volatile int* abort_flag = &ss.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&ss.full[s], 3); mbar_init(&ss.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ss.raw_full[b], 1); mbar_init(&ss.raw_empty[b], 2); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ss.tmem_full[b], 1); mbar_init(&ss.tmem_empty[b], 4); }
    ss.abort_flag = 0;
    mbar_fence_init();
  }
  if (p.offsets != nullptr) load_segments<BT - 8>(ss.seg, p.offsets, p.counts, p.groups);
  if (warp == 1) {
    tmem_alloc(&ss.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;
  TokenWalker<BT - 8, BW, kMaxGroups> walk(p.offsets != nullptr ? &ss.seg : nullptr, p.groups, n_tiles, p.M);
  TokenTile t;
  Ring ring;
  uint32_t acc = 0;
  bool ok = true;
  auto wait_empty = [&](const Ring& r) { return mbar_wait(&ss.empty[r.s], (r.round & 1) ^ 1, abort_flag, kTimeoutProducer); };

  if (warp == 0) {
    // ------------------------------------------------------------ weights, and a tile's weight scales
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      uint32_t steps = 0;
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
        const int wrow = t.g * p.N + t.n0, b = acc & 1;
        for (int kb = 0; kb < KB; ++kb, ring.next(1, stages), ++steps) {
          if (!wait_empty(ring)) { ok = false; break; }
          const int s = ring.s, k0 = min(kb * BK, p.K - BK);           // the last step of a K of 64 more is the last 128 elements
          mbar_expect_tx(&ss.full[s], kWCopied);
          if (k0 == kb * BK) tma_load_2d(w_tiles + s * kWBytes, &tmW, &ss.full[s], k0, wrow);
          else tma_load_2d(w_tiles + s * kWBytes, &tmTail, &ss.full[s], 0, wrow);
          if (kb == 0) {
            if (!mbar_wait(&ss.raw_empty[b], ((acc >> 1) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
            const uint32_t bytes = min(BW, p.N - t.n0) * sk;
            mbar_expect_tx(&ss.raw_full[b], bytes);
            copy_bulk(smem_u32(raw + b * raw_bytes), p.ws + (size_t)wrow * sk, bytes, &ss.raw_full[b]);
          }
        }
      }
      if (ok) {                            // every stage's last use is consumed, so every copy has landed
        for (int s = 0; s < stages && static_cast<uint32_t>(s) < steps; ++s) {
          const uint32_t last = s < ring.s ? ring.round : ring.round - 1;
          if (!mbar_wait(&ss.empty[s], last & 1, abort_flag, kTimeoutProducer)) break;
        }
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
      }
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------ token parts as they lie: eights of tokens, part by part
    if (elect_one()) {
      tma_prefetch_desc(&tmX128);
      tma_prefetch_desc(&tmX16);
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x) {
        const int rows = 2 * tile_tokens(t), first = 2 * (t.m0 & ~7);
        for (int kb = 0; kb < KB; ++kb, ring.next(1, stages)) {
          if (!wait_empty(ring)) { ok = false; break; }
          const int s = ring.s, k0 = min(kb * BK, p.K - BK);
          mbar_expect_tx(&ss.full[s], rows * BK);
          uint8_t* x = x_tiles + s * kXBytes;
          int r = 0;
          for (; r + 128 <= rows; r += 128) tma_load_2d(x + r * BK, &tmX128, &ss.full[s], k0, first + r);
          for (; r < rows; r += 16) tma_load_2d(x + r * BK, &tmX16, &ss.full[s], k0, first + r);
        }
      }
      if (!ok)
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);     // bounded grace period for copies in flight
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint64_t wdesc = make_smem_desc_sw128(smem_u32(w_tiles)), xdesc = make_smem_desc_sw128(smem_u32(x_tiles));
      uint32_t it = 0;
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
        const int buf = acc & 1, cols = tile_tokens(t);
        const uint32_t d = tmem_base + buf * kAccCols, idesc = block_idesc(2 * cols);
        if (!mbar_wait(&ss.tmem_empty[buf], ((acc >> 1) & 1) ^ 1, abort_flag, kTimeoutMma)) { ok = false; break; }
        for (int kb = 0; kb < KB; ++kb, ++it, ring.next(1, stages)) {
          const int s = ring.s;
          if (!mbar_wait(&ss.full[s], ring.round & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sfa = tmem_base + kSfCol + (it & 1) * kSfStep, sfb = sfa + 4;
          copy_scales(sfa, smem_u32(ss.sfa[s]));
          for (int c = 0; c < 2 * cols; c += 128) copy_scales(sfb + c / 32, smem_u32(ss.sfb[s]) + c * 4);
          const uint64_t adesc = wdesc + static_cast<uint32_t>(s * (kWBytes >> 4)), bdesc = xdesc + static_cast<uint32_t>(s * (kXBytes >> 4));
          const bool whole = kb * BK + BK <= p.K;                      // else the first half was part of the step before it
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q >= 2 || whole)
              mma_block(d, adesc + 2 * q, bdesc + 2 * q, idesc + static_cast<uint32_t>(q) * (1u << 4 | 1u << 29), sfa, sfb, kb > 0 || q > 0 ? 1u : 0u);
          tc_commit(&ss.empty[s]);
        }
        if (ok) tc_commit(&ss.tmem_full[buf]);
      }
    }
  } else if (warp < 4) {
    // ------------------------------------------------------------ scales: row r of an image at (r % 32) * 16 + r / 32 * 4, a byte a block of 32
    constexpr int kImgB = Sh::kSfB / 128;
    int turn = warp & 1;                   // steps until this warp's next: they alternate, across tiles too
    if (turn) ring.next(1, stages);
    for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
      const int cols = tile_tokens(t), b = acc & 1;
      const uint32_t* xrow[kImgB];
      uint32_t less[kImgB];
#pragma unroll
      for (int i = 0; i < kImgB; ++i) {                                 // column c: the first or second part of token c / 16 * 8 + c % 8
        const int c = 32 * i + lane, part = c >> 3 & 1;
        xrow[i] = reinterpret_cast<const uint32_t*>(p.xs) + min((t.m0 & ~7) + min(c / 16 * 8 + c % 8, cols - 1), p.M - 1);
        less[i] = part ? 0x01010101u * mxp::kPartShift : 0u;
      }
      uint32_t next[2][kImgB];                                          // two own steps ahead
      auto load = [&](int kb, uint32_t (&v)[kImgB]) {
#pragma unroll
        for (int i = 0; i < kImgB; ++i) v[i] = kb < KB && 32 * i < 2 * cols ? __ldg(xrow[i] + (size_t)kb * p.M) - less[i] : 0u;
      };
      load(turn, next[0]);
      load(turn + 2, next[1]);
      if (!__all_sync(0xffffffffu, mbar_wait(&ss.raw_full[b], (acc >> 1) & 1, abort_flag, kTimeoutProducer))) { ok = false; break; }
      const uint8_t* wrow[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) wrow[i] = raw + b * raw_bytes + min(32 * i + lane, p.N - t.n0 - 1) * sk;
      int kb = turn;
      for (; kb < KB; kb += 2, ring.next(2, stages)) {
        uint32_t now[kImgB], a[4];
#pragma unroll
        for (int i = 0; i < kImgB; ++i) { now[i] = next[0][i]; next[0][i] = next[1][i]; }
        load(kb + 4, next[1]);
        const int k0 = min(kb * BK, p.K - BK);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint16_t* src = reinterpret_cast<const uint16_t*>(wrow[i] + k0 / 32);
          a[i] = src[0] | static_cast<uint32_t>(src[1]) << 16;
        }
        if (k0 != kb * BK)
#pragma unroll
          for (int i = 0; i < kImgB; ++i) now[i] <<= 16;               // the last step's blocks are the window's second half
        if (!__all_sync(0xffffffffu, wait_empty(ring))) { ok = false; break; }
        *reinterpret_cast<uint4*>(ss.sfa[ring.s] + lane * 16) = make_uint4(a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int i = 0; i < kImgB; i += 4)
          *reinterpret_cast<uint4*>(ss.sfb[ring.s] + i * 128 + lane * 16) = make_uint4(now[i], now[i + 1], now[i + 2], now[i + 3]);
        fence_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ss.full[ring.s]);
      }
      turn = kb - KB;
      if (ok && lane == 0) mbar_arrive(&ss.raw_empty[b]);
    }
  } else {
    // ------------------------------------------------------------ epilogue: a warp's 32 weight rows
    for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
      const int buf = acc & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&ss.tmem_full[buf], (acc >> 1) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * kAccCols;
      const int base = t.m0 & ~7, cols = tile_tokens(t), row0 = t.n0 + quad * 32, col = row0 + 8 * (lane & 3);
#pragma unroll 1
      for (int c = 0; row0 < p.N && c < cols; c += 16) {                // sixteen tokens, both parts
        uint32_t v[2][16];
        float sum[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h) pair::tmem_ld_16x32(taddr + (static_cast<uint32_t>(16 * h) << 16) + 2 * c, v[h]);
        tmem_ld_wait();
        bool nan = false;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            sum[h][j] = __uint_as_float(v[h][j / 4 * 8 + j % 4]) + __uint_as_float(v[h][j / 4 * 8 + 4 + j % 4]);
            nan |= sum[h][j] != sum[h][j];
          }
        if (nan) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int tok = base + c + 8 * (j / 4) + 2 * (lane & 3) + (j & 1), row = row0 + 16 * h + 8 * ((j >> 1) & 1) + (lane >> 2);
              if (sum[h][j] != sum[h][j] && tok >= t.m0 && tok < t.m_end && row < p.N) sum[h][j] = not_finite(p, tok, t.g * p.N + row);
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t x[4] = {pair::pack_bf16(sum[0][4 * j], sum[0][4 * j + 1]), pair::pack_bf16(sum[0][4 * j + 2], sum[0][4 * j + 3]),
                                 pair::pack_bf16(sum[1][4 * j], sum[1][4 * j + 1]), pair::pack_bf16(sum[1][4 * j + 2], sum[1][4 * j + 3])};
          const int tok = base + c + 8 * j + (lane >> 2);
          pair::store_32x8(x, tok >= t.m0 && tok < t.m_end ? p.D + (size_t)tok * p.ldd + col : nullptr, p.N - col, p.wide != 0);
        }
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

// Rows of x as parts.  pos null: row r to row r; else token t to the rows pos[t * topk ..] that are not negative.  Bound by its bytes.
__global__ void __launch_bounds__(128)
mx_split_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ pos, int topk, mxp::Parts out) {
  const int k = (blockIdx.y * 128 + threadIdx.x) * 16;
  if (k >= out.K) return;                  // K is a multiple of 32: a block's two lanes stay together
  const int row = blockIdx.x;
  __align__(16) __nv_bfloat162 v[8];
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * ldx + k);
  reinterpret_cast<uint4*>(v)[0] = src[0];
  reinterpret_cast<uint4*>(v)[1] = src[1];
  const mxp::Split<16> s(v);
  if (pos == nullptr) {
    s.store(out, row, k);
    return;
  }
  for (int j = 0; j < topk; ++j) {
    const int r = pos[(size_t)row * topk + j];
    if (r >= 0) s.store(out, r, k);
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
// 16-byte containers of sixteen nibbles, or bytes; 128 elements of `rows` rows
static int make_map(CUtensorMap* m, bool nibbles, const void* base, uint64_t rows, uint64_t cols, uint64_t stride, uint32_t box_rows) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {stride};
  cuuint32_t box[2] = {BK, box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, nibbles ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

template <int BT>
static int launch(Params& p, int num_sms, cudaStream_t stream) {
  CUtensorMap tw, tail, t128, t16;
  const uint64_t wrows = (uint64_t)p.groups * p.N, kq = p.K / 2;
  if (make_map(&tw, true, p.wq, wrows, p.K / BK * BK, kq, BW) != 0) return -11;
  tail = tw;                                                          // read only where K ends in half a step
  if (p.K % BK != 0 && make_map(&tail, true, p.wq + (p.K - BK) / 2, wrows, BK, kq, BW) != 0) return -11;
  const uint64_t xrows = (uint64_t)(p.M + 7) / 8 * 16;
  if (make_map(&t16, false, p.xp, xrows, p.K, p.K, 16) != 0) return -12;
  t128 = t16;                                                         // read only by tiles of 128 rows of parts
  if (2 * BT >= 128 && xrows >= 128 && make_map(&t128, false, p.xp, xrows, p.K, p.K, 128) != 0) return -12;
  static DeviceOnce once;
  auto kern = mxfp4_block_kernel<BT>;
  if (!ensure_dynamic_smem(kern, kMaxShared, once)) return -13;
  const int fixed = sizeof(Shared<BT>) + 1024 + 2 * BW * (p.K / 32), stage = kWBytes + 2 * BT * BK;
  p.stages = (kMaxShared - fixed) / stage;
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  if (p.stages < 2) return -15;
  const int n_tiles = (p.N + BW - 1) / BW;
  long long grid = ((long long)p.M / (BT - 8) + p.groups) * n_tiles;      // an upper bound of the tiles
  if (grid > num_sms) grid = num_sms;
  if (grid < 1) grid = 1;
  kern<<<(int)grid, kThreads, fixed + p.stages * stage, stream>>>(tw, tail, t128, t16, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -14;
}

}  // namespace mxb
}  // namespace bg

extern "C" {

// 1 where the block-scaled product takes these weights: whole 128-element steps in a 32-byte aligned row, scales in 16-byte pieces, and a tile's scales
// twice beside two stages.
int bg_mxfp4_block_takes(const void* Wq, const void* Ws, long long N, int K) {
  return K >= 128 && K % 64 == 0 && K <= 12288 && N * (K / 32) % 16 == 0 && reinterpret_cast<uintptr_t>(Wq) % 32 == 0 && reinterpret_cast<uintptr_t>(Ws) % 16 == 0;
}

// xp [M / 8 rounded up][2][8][K] and xs [K / 128 rounded up][M][4]: rows as bg_mx_split makes them; Wq [groups * N, K / 2] packed e2m1 (low nibble = even k); Ws [groups * N,
// K / 32] e8m0; D [M, ldd] bf16.  offsets null: dense; counts: rows present in every segment, or null (rows past them stay undefined).
// rows: expected in a segment, for the width of a token tile.
int bg_mxfp4_block_gemm(const void* xp, const void* xs, const void* Wq, const void* Ws, void* D, int ldd, const int* offsets, const int* counts,
                        int groups, int M, int N, int K, float rows, int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::mxb;
  if (M <= 0 || N <= 0) return 0;
  if (!bg_mxfp4_block_takes(Wq, Ws, N, K) || groups > kMaxGroups || groups <= 0 || ldd % 8 != 0 || reinterpret_cast<uintptr_t>(xs) % 4 != 0) return -1;
  if (offsets == nullptr) groups = 1;
  Params p;
  p.wq = reinterpret_cast<const uint8_t*>(Wq); p.ws = reinterpret_cast<const uint8_t*>(Ws);
  p.xp = reinterpret_cast<const uint8_t*>(xp); p.xs = reinterpret_cast<const uint8_t*>(xs);
  p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd; p.wide = reinterpret_cast<uintptr_t>(D) % 16 == 0;
  p.offsets = offsets; p.counts = offsets != nullptr ? counts : nullptr; p.groups = groups; p.M = M; p.N = N; p.K = K; p.status = status;
  // 32 or 96 tokens a tile.  128 experts of 6,144 x 2,880, us: 24 rows each 334 / 401, 28 369 / 405, 30 412 / 412, 32 449 / 416, 47 602 / 449; of 2,880 x 3,072: 28
  // 218 / 246, 30 234 / 248, 32 248 / 250, 36 275 / 257; 32 experts of 6,144 x 2,880: 28 113 / 119, 30 121 / 121, 36 148 / 123
  return rows <= 30.f ? launch<40>(p, num_sms, stream) : launch<104>(p, num_sms, stream);
}

// x [T, ldx] bf16 -> parts p [rows / 8 rounded up][2][8][K], s [K / 128 rounded up][rows][4].  pos [T, topk]: the rows a token goes to (negative: none), or null: its
// own.  K % 32 == 0, x and ldx in 16-byte pieces.
int bg_mx_split(const void* x, long long ldx, const int* pos, int topk, int T, void* p, void* s, int rows, int K, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0 || K <= 0) return 0;
  if (K % 32 != 0 || ldx % 8 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0) return -1;
  const mxp::Parts out{reinterpret_cast<uint8_t*>(p), reinterpret_cast<uint8_t*>(s), rows, K};
  mxb::mx_split_kernel<<<dim3(T, (K / 16 + 127) / 128), 128, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(x), ldx, pos, topk, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
