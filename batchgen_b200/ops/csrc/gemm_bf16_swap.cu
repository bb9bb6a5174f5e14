// bf16 GEMM with the weights on the tensor-core M side and up to 256 tokens as N (D^T = W . X^T), dense and ragged grouped, for products of few
// tiles, short K or rows that start anywhere.
//
// A weight tile of 128 rows meets all tokens of its segment (up to 256 at a time, cut evenly, rounded up to 16) in one product of that width.
// With enough 256 x 256 tiles and K from 512 on, pairs of CTAs move fewer operand bytes (gemm_bf16_pair.cu).  Below, tiles of half the size fill
// the SMs better, us here and on pairs: 1,024 x 4,096 x 2,880 25 / 27, 2,000 x 1,024 x 4,096 29 / 31, 160 x 32,768 x 512 15 / 17; of short K a pair stores
// a tile longer than it multiplies the next: 6,000 x 4,096 x 256 24.5 / 28.7, x 512 32.8 / 32.8; and two bytes a store do not mind where a row
// starts: 1,100 x 20,004 x 1,024 51 / 139.
//
// Roles (192 threads, one CTA per SM, persistent): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 2..5 epilogue (thread = weight
// row; two accumulators of 256 columns, so one is stored while the other is filled).  All waits are bounded.
#define BG_FILE_TAG 33     // kernel-trace ids of this file are (tag << 16) | line
#include "common.cuh"
#include "token_tiles.cuh"

namespace bg {
namespace bswap {

constexpr int BW = 128;                   // weight rows of a tile (MMA M)
constexpr int BT = 256;                   // most tokens of a tile (MMA N)
constexpr int kBox = 32;                  // token rows of one TMA box
constexpr int BK = 64;                    // elements of K per stage (one 128-byte swizzle atom)
constexpr int kStages = 4;
constexpr int kThreads = 192;
constexpr int kTmemCols = 512;
constexpr int kMaxGroups = 1024;
constexpr int kWBytes = BW * BK * 2;      // 16 KB
constexpr int kXBytes = BT * BK * 2;      // 32 KB

struct Params {
  __nv_bfloat16* D;      // [M, ldd]
  int ldd;
  const int* offsets;    // [groups + 1] segment starts; null = dense
  const int* counts;     // [groups] rows present in a segment, or null: all of it
  int groups, M, N, K;
  int* status;
};

struct Shared {
  uint64_t full[kStages], empty[kStages];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  Segments<kMaxGroups> seg;
};

__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_swap_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params p) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_tiles = smem;
  uint8_t* x_tiles = smem + kStages * kWBytes;
  Shared& ss = *reinterpret_cast<Shared*>(x_tiles + kStages * kXBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
  const int KB = p.K / BK;
  const int n_tiles = (p.N + BW - 1) / BW;
  volatile int* abort_flag = &ss.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&ss.full[s], 1); mbar_init(&ss.empty[s], 1); }
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
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x) {
        const int boxes = (tile_cols(t) + kBox - 1) / kBox, row = t.g * p.N + t.n0;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kStages;
          if (!mbar_wait(&ss.empty[s], ((it / kStages) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
          mbar_expect_tx(&ss.full[s], kWBytes + boxes * kBox * BK * 2);
          tma_load_2d(w_tiles + s * kWBytes, &tmW, &ss.full[s], kb * BK, row);
          for (int b = 0; b < boxes; ++b)
            tma_load_2d(x_tiles + s * kXBytes + b * kBox * BK * 2, &tmX, &ss.full[s], kb * BK, t.m0 + b * kBox);
        }
      }
      if (ok) {
        const uint32_t n = it < (uint32_t)kStages ? it : (uint32_t)kStages;
        for (uint32_t j = it - n; j < it; ++j)
          if (!mbar_wait(&ss.empty[j % kStages], (j / kStages) & 1, abort_flag, kTimeoutProducer)) break;
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
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
          const int s = it % kStages;
          if (!mbar_wait(&ss.full[s], (it / kStages) & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          const uint64_t adesc = make_smem_desc_sw128(smem_u32(w_tiles + s * kWBytes));
          const uint64_t bdesc = make_smem_desc_sw128(smem_u32(x_tiles + s * kXBytes));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            mma_f16(tmem_base + buf * BT, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) ? 1u : 0u);
          tc_commit(&ss.empty[s]);
        }
        if (ok) tc_commit(&ss.tmem_full[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: thread = weight row, columns = tokens
    for (int tile = blockIdx.x; ok && walk.get(tile, t); tile += gridDim.x, ++acc) {
      const int buf = acc & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&ss.tmem_full[buf], (acc >> 1) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * BT;
      const int n_tok = t.m_end - t.m0, col = t.n0 + quad * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < n_tok; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(taddr + c, v);
        tmem_ld_wait();
        if (col < p.N) {
          __nv_bfloat16* dst = p.D + (size_t)(t.m0 + c) * p.ldd + col;
          if (c + 32 <= n_tok) {
#pragma unroll
            for (int j = 0; j < 32; ++j) dst[(size_t)j * p.ldd] = __float2bfloat16(__uint_as_float(v[j]));
          } else {
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

static int make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {BK, box_rows};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

}  // namespace bswap
}  // namespace bg

extern "C" {

// X [M, K] bf16 tokens, W [groups * N, K] bf16 -> D [M, ldd] bf16.  K a multiple of 64.  offsets null: dense; counts: rows present in
// every segment, or null (rows past them stay undefined).
int bg_gemm_bf16_swap_grouped(const void* X, const void* W, void* D, int ldd, const int* offsets, const int* counts, int groups, int M, int N, int K,
                              int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::bswap;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % BK != 0 || groups > kMaxGroups || groups <= 0) return -1;
  if (offsets == nullptr) groups = 1;
  Params p;
  p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd; p.offsets = offsets; p.counts = offsets != nullptr ? counts : nullptr;
  p.groups = groups; p.M = M; p.N = N; p.K = K; p.status = status;
  CUtensorMap tw, tx;
  if (make_map(&tw, W, (uint64_t)groups * N, (uint64_t)K, BW) != 0) return -11;
  if (make_map(&tx, X, (uint64_t)M, (uint64_t)K, kBox) != 0) return -12;
  static bg::DeviceOnce once;
  const size_t smem = kStages * (kWBytes + kXBytes) + sizeof(Shared) + 1024;
  if (!bg::ensure_dynamic_smem(gemm_bf16_swap_kernel, smem, once)) return -13;
  long long grid = ((long long)M / BT + (offsets != nullptr ? groups : 1)) * ((N + BW - 1) / BW);      // an upper bound of the tiles
  if (grid > num_sms) grid = num_sms;
  bg::launch_pdl(gemm_bf16_swap_kernel, dim3((int)grid), dim3(kThreads), smem, stream, tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -14;
}

// the dense form
int bg_gemm_bf16_swap(const void* X, const void* W, void* D, int ldd, int M, int N, int K, int num_sms, int* status, cudaStream_t stream) {
  return bg_gemm_bf16_swap_grouped(X, W, D, ldd, nullptr, nullptr, 1, M, N, K, num_sms, status, stream);
}

}  // extern "C"

BG_TRACE_SETTER(gemm_bf16_swap)
