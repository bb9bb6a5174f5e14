// bf16 GEMM of prompt-sized steps on pairs of CTAs: 256 weight rows as M, up to 256 tokens as N (D^T = W . X^T), dense and ragged grouped.
//
// A mixture gives an expert anything from a token to a few hundred.  A weight tile meets all tokens of its segment (up to 256 at a time, cut
// evenly, rounded up to 32) in one product of that width, so weights cross L2 once and the padding is below 32 tokens.  What bounds a
// 128 x 256 tile on one CTA is its operands: 48 KB a K step of 64, written to and read from shared memory in the 512 clocks of the product
// (440 - 500 ns measured); a pair stages 32 KB in each CTA for the same work and runs at what the library's kernel does.  One CTA -> pair, us:
// dense 4,096 x 16,576 x 2,304 224 -> 207 (library 216), 5,200 x 12,288 x 2,304 214 -> 195, 8,000 x 2,304 x 4,096 121 -> 105; 256 matrices of 2,048 x
// 2,304, Poisson rows, 128 each 457 -> 423 (5.7 TB/s of weights), 512 each 1,064 -> 993; of 2,304 x 1,024 244 -> 226.  Outputs are bit for bit the
// same.  Bound by the tensor cores' power at prompt sizes, by the weights' bytes below some 150 rows a segment.
//
// The epilogue reads 16 lanes x 8 columns an instruction, transposes 8 x 8 blocks between lanes and stores 16 bytes a thread: eight tokens of
// 64 bytes, where a lane per weight row would store two bytes a thread.
//
// Roles (384 threads, one CTA per SM, pairs persistent): warp 0 TMA producer of the CTA's halves, warp 1 of the first CTA MMA issuer for both,
// warp 1 TMEM owner, warps 4..11 epilogue (two accumulators of 256 columns).  All waits are bounded.
#define BG_FILE_TAG 34     // kernel-trace ids of this file are (tag << 16) | line
#include "pair.cuh"
#include "token_tiles.cuh"

namespace bg {
namespace bpair {

constexpr int BW = 256;                   // weight rows of a tile (MMA M), half of them in each CTA
constexpr int BT = 256;                   // most tokens of a tile (MMA N), half of them in each CTA's shared memory
constexpr int BK = 64;                    // elements of K per stage (one 128-byte swizzle atom)
constexpr int kStages = 6;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 128 + 32 * kEpiWarps;
constexpr int kTmemCols = 512;
constexpr int kMaxGroups = 1024;
constexpr int kRowBytes = BK * 2;
constexpr int kWBytes = BW / 2 * kRowBytes;      // 16 KB
constexpr int kXBytes = BT / 2 * kRowBytes;      // 16 KB

struct Params {
  __nv_bfloat16* D;      // [M, ldd]
  int ldd;
  const int* offsets;    // [groups + 1] segment starts; null = dense
  const int* counts;     // [groups] rows present in a segment, or null: all of it
  int groups, M, N, K;
  int wide;              // D's rows are 16-byte aligned
  int* status;
};

struct Shared {
  uint64_t full[kStages], empty[kStages];          // full: the leader's, for both CTAs' bytes
  uint64_t tmem_full[2], tmem_empty[2];            // empty: the leader's, for both CTAs' epilogue warps
  uint32_t tmem_base;
  int abort_flag;
  Segments<kMaxGroups> seg;
};

__device__ __forceinline__ int pair_cols(const TokenTile& t) { return (t.m_end - t.m0 + 31) / 32 * 32; }

__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX64, const __grid_constant__ CUtensorMap tmX16,
                      const Params p) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_tiles = smem;
  uint8_t* x_tiles = smem + kStages * kWBytes;
  Shared& ss = *reinterpret_cast<Shared*>(x_tiles + kStages * kXBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3;
  const int rank = pair::cluster_rank(), first = blockIdx.x >> 1, step = gridDim.x >> 1;
  const int KB = p.K / BK;
  const int n_tiles = (p.N + BW - 1) / BW;
  volatile int* abort_flag = &ss.abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&ss.full[s], 1); mbar_init(&ss.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ss.tmem_full[b], 1); mbar_init(&ss.tmem_empty[b], 2 * kEpiWarps); }
    ss.abort_flag = 0;
    mbar_fence_init();
  }
  if (p.offsets != nullptr) load_segments<BT>(ss.seg, p.offsets, p.counts, p.groups);
  if (warp == 1) {
    pair::alloc(&ss.tmem_base, kTmemCols);
    pair::relinquish();
  }
  tc_fence_before();
  __syncthreads();
  pair::cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;
  TokenWalker<BT, BW, kMaxGroups> walk(p.offsets != nullptr ? &ss.seg : nullptr, p.groups, n_tiles, p.M);
  TokenTile t;
  uint32_t it = 0, acc = 0;
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer: this CTA's halves
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX64);
      for (int tile = first; ok && walk.get(tile, t); tile += step) {
        const int half = pair_cols(t) / 2;                         // tokens of this CTA: a multiple of 16
        const int wrow = t.g * p.N + t.n0 + rank * (BW / 2), xrow = t.m0 + rank * half;
        const uint32_t bytes = 2 * (kWBytes + half * kRowBytes);
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kStages;
          if (!pair::wait_cluster(&ss.empty[s], ((it / kStages) & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&ss.full[s], bytes);
          const uint32_t bar = pair::leader_addr(&ss.full[s]);
          uint8_t* x = x_tiles + s * kXBytes;
          pair::load_2d(w_tiles + s * kWBytes, &tmW, bar, kb * BK, wrow);
          int r = 0;
          for (; r + 64 <= half; r += 64) pair::load_2d(x + r * kRowBytes, &tmX64, bar, kb * BK, xrow + r);
          for (; r < half; r += 16) pair::load_2d(x + r * kRowBytes, &tmX16, bar, kb * BK, xrow + r);
        }
      }
      if (ok) {
        const uint32_t n = it < (uint32_t)kStages ? it : (uint32_t)kStages;
        for (uint32_t j = it - n; j < it; ++j)
          if (!pair::wait_cluster(&ss.empty[j % kStages], (j / kStages) & 1, abort_flag, kTimeoutProducer)) break;
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer, for both CTAs
    if (rank == 0 && elect_one()) {
      for (int tile = first; ok && walk.get(tile, t); tile += step, ++acc) {
        const int buf = acc & 1;
        const uint32_t idesc = make_idesc(BW, pair_cols(t), 1, 1);   // bf16 x bf16 -> fp32
        if (!pair::wait_cluster(&ss.tmem_empty[buf], ((acc >> 1) & 1) ^ 1, abort_flag, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % kStages;
          if (!pair::wait_cluster(&ss.full[s], (it / kStages) & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
          tc_fence_after();
          const uint64_t adesc = make_smem_desc_sw128(smem_u32(w_tiles + s * kWBytes));
          const uint64_t bdesc = make_smem_desc_sw128(smem_u32(x_tiles + s * kXBytes));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            pair::mma_f16(tmem_base + buf * BT, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) ? 1u : 0u);
          pair::commit(&ss.empty[s]);
        }
        if (ok) pair::commit(&ss.tmem_full[buf]);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ epilogue: warp = (32 weight rows, every second 32 tokens)
    const int side = (warp - 4) >> 2;
    for (int tile = first; ok && walk.get(tile, t); tile += step, ++acc) {
      const int buf = acc & 1;
      if (!__all_sync(0xffffffffu, pair::wait_cluster(&ss.tmem_full[buf], (acc >> 1) & 1, abort_flag, kTimeoutEpilogue))) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + buf * BT;
      const int n_tok = t.m_end - t.m0, row0 = t.n0 + rank * (BW / 2) + quad * 32, col = row0 + 8 * (lane & 3);
#pragma unroll 1
      for (int c = 32 * side; row0 < p.N && c < n_tok; c += 64) {
        uint32_t lo[16], hi[16];
        pair::tmem_ld_16x32(taddr + c, lo);
        pair::tmem_ld_16x32(taddr + (16u << 16) + c, hi);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t x[4] = {pair::pack_bf16(__uint_as_float(lo[4 * j]), __uint_as_float(lo[4 * j + 1])),
                                 pair::pack_bf16(__uint_as_float(lo[4 * j + 2]), __uint_as_float(lo[4 * j + 3])),
                                 pair::pack_bf16(__uint_as_float(hi[4 * j]), __uint_as_float(hi[4 * j + 1])),
                                 pair::pack_bf16(__uint_as_float(hi[4 * j + 2]), __uint_as_float(hi[4 * j + 3]))};
          const int tok = c + 8 * j + (lane >> 2);
          pair::store_32x8(x, tok < n_tok ? p.D + (size_t)(t.m0 + tok) * p.ldd + col : nullptr, p.N - col, p.wide != 0);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair::arrive_cluster(pair::leader_addr(&ss.tmem_empty[buf]));
    }
  }

  tc_fence_before();
  __syncthreads();
  pair::cluster_sync();                    // no CTA leaves while the other's products, loads or arrivals may reach it
  tc_fence_after();
  if (warp == 1) pair::dealloc(tmem_base, kTmemCols);
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

}  // namespace bpair
}  // namespace bg

extern "C" {

// X [M, K] bf16 tokens, W [groups * N, K] bf16 -> D [M, ldd] bf16.  K a multiple of 64.  offsets null: dense; counts: rows present in
// every segment, or null (rows past them stay undefined).
int bg_gemm_bf16_pair(const void* X, const void* W, void* D, int ldd, const int* offsets, const int* counts, int groups, int M, int N,
                      int K, int num_sms, int* status, cudaStream_t stream) {
  using namespace bg::bpair;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % BK != 0 || groups > kMaxGroups || groups <= 0 || num_sms < 2) return -1;
  if (offsets == nullptr) groups = 1;
  Params p;
  p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd; p.offsets = offsets; p.counts = offsets != nullptr ? counts : nullptr;
  p.groups = groups; p.M = M; p.N = N; p.K = K; p.status = status;
  p.wide = ldd % 8 == 0 && reinterpret_cast<uintptr_t>(D) % 16 == 0;
  CUtensorMap tw, tx64, tx16;
  if (make_map(&tw, W, (uint64_t)groups * N, (uint64_t)K, BW / 2) != 0) return -11;
  if (make_map(&tx64, X, (uint64_t)M, (uint64_t)K, 64) != 0 || make_map(&tx16, X, (uint64_t)M, (uint64_t)K, 16) != 0) return -12;
  static bg::DeviceOnce once;
  const size_t smem = kStages * (kWBytes + kXBytes) + sizeof(Shared) + 1024;
  if (!bg::ensure_dynamic_smem(gemm_bf16_pair_kernel, smem, once)) return -13;
  const int n_tiles = (N + BW - 1) / BW;
  long long pairs = ((long long)M / BT + (offsets != nullptr ? groups : 1)) * n_tiles;      // an upper bound of the tiles
  if (pairs > num_sms / 2) pairs = num_sms / 2;
  bg::launch_pdl_cluster(gemm_bf16_pair_kernel, dim3(2 * (int)pairs), dim3(kThreads), dim3(2), smem, stream, tw, tx64, tx16, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -14;
}

}  // extern "C"

BG_TRACE_SETTER(gemm_bf16_pair)
