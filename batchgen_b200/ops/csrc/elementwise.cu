// Memory-bound fused elementwise kernels: (residual add +) RMSNorm (+ per-token 1x128 e4m3
// quantisation), activation quantisation with optional SiLU*up, and the MLA latent-KV producer
// (RMSNorm of c_kv + RoPE of k_pe + paged cache write).
//
// Quantisation contract: scale = max(amax, 1e-4) / 448 (optionally rounded up to a power of two),
// q = x * (1 / scale) rounded to nearest e4m3, saturating.  The fused norm+quant kernel rounds
// the normalised value to bf16 first, so its bytes equal those of the unfused pair
// (the reference keeps the same contract: batchgen_kernels/src/attention/csrc/add_rmsnorm_fp8_quant.cu:243).
// Scales are written in [KB, stride] layout (scale of row t, block kb at s[kb * stride + t]),
// the layout the GEMM epilogue reads with coalesced loads.
//
// Replaces (by behaviour): batchgen_kernels/src/attention/csrc/rmsnorm.cu:88-254,
// add_rmsnorm_fp8_quant.cu:243, batchgen_kernels/src/moe/fp8_blockwise/fp8_blockwise_ops.cu:39-445,
// batchgen_kernels/src/attention/fused_kv_norm_rope_cache.cu:14, batchgen_kernels/triton/fp8_quantize.py.
#define BG_FILE_TAG 1      // kernel-trace ids of this file are (tag << 16) | line
#include "quant_blocks.cuh"

namespace bg {

constexpr int kNormThreads = 256;

__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < (blockDim.x >> 5)) ? red[lane] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

// One block per row.  Each thread owns NV vectors of 8 consecutive elements, all of them read before the first is used and kept in registers
// between the two passes; 16 consecutive threads cover one 128-wide quantisation block, so the block amax is a 16-lane shuffle
// reduction.  Bound by its bytes: with the row in shared memory, eight lanes on a bank, 4,739 rows of 7,168 with sum and quantisation took
// 63.6 us, now 59 (floor 42); 1,536 rows 28.7, now 26.7; 256 and fewer as before (12).
template <bool ADD, bool QUANT, int NV>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ residual,
               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out, uint8_t* __restrict__ out_q,
               float* __restrict__ out_s, int s_stride, int H, int ldx, int ldo, float eps, int pow2) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  __shared__ float red[32];
  const int t = blockIdx.x;
  const __nv_bfloat16* xr = x + (size_t)t * ldx;
  __nv_bfloat16* rr = ADD ? residual + (size_t)t * H : nullptr;
  uint4 xv[NV], rv[ADD ? NV : 1];
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int v = threadIdx.x + n * kNormThreads;
    if (v >= H / 8) continue;
    xv[n] = *reinterpret_cast<const uint4*>(xr + v * 8);
    if (ADD) rv[n] = *reinterpret_cast<const uint4*>(rr + v * 8);
  }
  float ss = 0.f;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int v = threadIdx.x + n * kNormThreads;
    if (v >= H / 8) continue;
    __nv_bfloat162* xp = reinterpret_cast<__nv_bfloat162*>(&xv[n]);
    if (ADD) {
      const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&rv[n]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {         // the sum as stored (bf16) is what gets normalised
        const float2 a = __bfloat1622float2(xp[i]), b = __bfloat1622float2(rp[i]);
        xp[i] = __floats2bfloat162_rn(a.x + b.x, a.y + b.y);
      }
      *reinterpret_cast<uint4*>(rr + v * 8) = xv[n];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = __bfloat1622float2(xp[i]);
      ss += a.x * a.x;
      ss += a.y * a.y;
    }
  }
  const float total = block_sum_256(ss, red);
  const float rstd = rsqrtf(total / (float)H + eps);
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int v = threadIdx.x + n * kNormThreads;
    if (v >= H / 8) continue;               // H is a multiple of 128 where blocks are quantised: their lanes stay together
    uint4 wraw = *reinterpret_cast<const uint4*>(w + v * 8);
    const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wraw);
    const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xv[n]);
    __align__(16) __nv_bfloat162 o[4];
    float y[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 ww = __bfloat1622float2(wp[i]), a = __bfloat1622float2(xp[i]);
      o[i] = __floats2bfloat162_rn(a.x * rstd * ww.x, a.y * rstd * ww.y);
      float2 b = __bfloat1622float2(o[i]);
      y[2 * i] = b.x;
      y[2 * i + 1] = b.y;
    }
    if (out != nullptr) *reinterpret_cast<uint4*>(out + (size_t)t * ldo + v * 8) = *reinterpret_cast<const uint4*>(o);
    if (QUANT) {
      const float s = quant_block(y, out_q + (size_t)t * H + v * 8, pow2, 0xffffu << (threadIdx.x & 16));
      if ((threadIdx.x & 15) == 0) out_s[(size_t)(v / 16) * s_stride + t] = s;
    }
  }
}

// Activation quantisation.  MODE 0: x [T, K].  MODE 1: x [T, 2K] = gate | up -> quantise silu(gate)*up.  Warps walk the rows (quant_blocks.cuh).
template <int MODE, int U>
__global__ void __launch_bounds__(256)
act_quant_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ s, int s_stride,
                 int T, int K, int ldx, int pow2, const int* __restrict__ valid_rows,
                 const int* __restrict__ row_src) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int lane = threadIdx.x & 31, rows = valid_rows != nullptr ? min(T, *valid_rows) : T;
  for (BlockWalk<U> walk(rows, K); walk.more(); walk.next()) {
    const int t = walk.row;
    if (row_src != nullptr && row_src[t] < 0) continue;    // padding row of an expert segment: nothing reads it
    const __nv_bfloat16* xr = x + (size_t)t * ldx;
    uint4 raw[U], up[MODE == 1 ? U : 1];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = walk.block(u, lane);
      if (kb * 128 >= K) continue;
      raw[u] = *reinterpret_cast<const uint4*>(xr + kb * 128 + (lane & 15) * 8);
      if (MODE == 1) up[u] = *reinterpret_cast<const uint4*>(xr + K + kb * 128 + (lane & 15) * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = walk.block(u, lane);
      if (kb * 128 >= K) continue;
      float f[8];
      unpack8(raw[u], f);
      if (MODE == 1) {
        float g[8];
        unpack8(up[u], g);
        // round the activation to bf16 first: same bytes as silu_mul (bf16) followed by act_quant
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(__float2bfloat16(silu(f[i]) * g[i]));
      }
      const float sc = quant_block(f, q + (size_t)t * K + kb * 128 + (lane & 15) * 8, pow2, 0xffffu << (lane & 16));
      if ((lane & 15) == 0) s[(size_t)kb * s_stride + t] = sc;
    }
  }
}

// MODE 1 for many blocks, a CTA a row.  Exponential and division bound it as much as its bytes, so resident warps count more than loads in flight:
// 4,739 rows of 7,168 51 us, warps that walk the rows 60 with one block a half-warp and 80 with four, 2,400 rows of 4,096 20.5, 22.5 and 31; for
// few blocks the walk's spread over the SMs wins, 256 rows of 7,168 12.3 against 10.2.
__global__ void __launch_bounds__(256)
silu_quant_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ s, int s_stride, int K, int ldx, int pow2,
                       const int* __restrict__ valid_rows, const int* __restrict__ row_src) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int t = blockIdx.x;
  if (valid_rows != nullptr && t >= *valid_rows) return;
  if (row_src != nullptr && row_src[t] < 0) return;
  const __nv_bfloat16* xr = x + (size_t)t * ldx;
  for (int v = threadIdx.x; v < K / 8; v += blockDim.x) {            // K is a multiple of 128: a block's sixteen lanes stay together
    float f[8], u[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + v * 8), f);
    unpack8(*reinterpret_cast<const uint4*>(xr + K + v * 8), u);
    // round the activation to bf16 first: same bytes as silu_mul (bf16) followed by act_quant
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(__float2bfloat16(silu(f[i]) * u[i]));
    const float sc = quant_block(f, q + (size_t)t * K + v * 8, pow2, 0xffffu << (threadIdx.x & 16));
    if ((threadIdx.x & 15) == 0) s[(size_t)(v / 16) * s_stride + t] = sc;
  }
}

// MLA latent-KV producer.  One block (128 threads) per token:
//   cache[slot, 0:kv_lora]        = rmsnorm(kv_a[t, 0:kv_lora]) * w
//   cache[slot, kv_lora:+rope]    = rope(kv_a[t, kv_lora:], position[t])
// slot < 0 writes nothing.  cos/sin are fp32 tables [max_pos, rope/2].
__global__ void __launch_bounds__(128)
mla_kv_write_kernel(const __nv_bfloat16* __restrict__ kv_a, int ld, const __nv_bfloat16* __restrict__ w,
                    const int* __restrict__ positions, const float* __restrict__ cos_t,
                    const float* __restrict__ sin_t, const long long* __restrict__ slots,
                    __nv_bfloat16* __restrict__ cache, int kv_lora, int rope, float eps, int interleaved) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  __shared__ float red[32];
  const int t = blockIdx.x;
  const long long slot = slots[t];
  const __nv_bfloat16* src = kv_a + (size_t)t * ld;
  float ss = 0.f;
  for (int i = threadIdx.x; i < kv_lora; i += blockDim.x) {
    const float v = __bfloat162float(src[i]);
    ss += v * v;
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) tot += red[i];
  if (slot < 0) return;
  const float rstd = rsqrtf(tot / (float)kv_lora + eps);
  __nv_bfloat16* dst = cache + (size_t)slot * (kv_lora + rope);
  for (int i = threadIdx.x; i < kv_lora; i += blockDim.x)
    dst[i] = __float2bfloat16(__bfloat162float(src[i]) * rstd * __bfloat162float(w[i]));
  const int half = rope / 2;
  const int pos = positions[t];
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float c = cos_t[(size_t)pos * half + i], s = sin_t[(size_t)pos * half + i];
    const int i0 = interleaved ? 2 * i : i, i1 = interleaved ? 2 * i + 1 : i + half;
    const float a = __bfloat162float(src[kv_lora + i0]), b = __bfloat162float(src[kv_lora + i1]);
    dst[kv_lora + i0] = __float2bfloat16(a * c - b * s);
    dst[kv_lora + i1] = __float2bfloat16(b * c + a * s);
  }
}

// A pair turned by an angle, written out so that every kernel rounds alike: left to the compiler, two kernels contracted the second sum differently
// (a query in 30,000 off by a bit of bf16 with its row's alignment).
__device__ __forceinline__ float2 turn(float a, float b, float c, float s) { return make_float2(__fmaf_rn(a, c, -__fmul_rn(b, s)), __fmaf_rn(a, s, __fmul_rn(b, c))); }

// In-place RoPE on the trailing `rope` dims of every head of q [T, H, D].
__global__ void rope_q_kernel(__nv_bfloat16* __restrict__ q, int H, int D, int rope, const int* __restrict__ positions,
                              const float* __restrict__ cos_t, const float* __restrict__ sin_t, int interleaved,
                              long long ld_t) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int t = blockIdx.x;
  const int half = rope / 2;
  const int pos = positions[t];
  for (int idx = threadIdx.x; idx < H * half; idx += blockDim.x) {
    const int h = idx / half, i = idx % half;
    __nv_bfloat16* p = q + (size_t)t * ld_t + (size_t)h * D + (D - rope);
    const float c = cos_t[(size_t)pos * half + i], s = sin_t[(size_t)pos * half + i];
    const int i0 = interleaved ? 2 * i : i, i1 = interleaved ? 2 * i + 1 : i + half;
    const float2 y = turn(__bfloat162float(p[i0]), __bfloat162float(p[i1]), c, s);
    p[i0] = __float2bfloat16(y.x);
    p[i1] = __float2bfloat16(y.y);
  }
}

// The same, eight pairs a thread in 16-byte pieces (rope a multiple of 16, pieces on 16-byte boundaries).  Bound by
// its bytes: two bytes an access took 63.5 us for 4,739 tokens of 128 heads with 64 rotated dims, now 34.8 (floor
// 24 at the 32-byte sectors touched); 4 tokens 15, now 8.  Where a token has a pair a thread at most, and few tokens keep the SMs waiting for one
// round of loads, the other kernel's shorter chain is faster: 64 tokens of 8 heads x 64 dims 1.58 us, here 1.73; 4,000 tokens 12.3, here 10.2.
template <bool INTERLEAVED>
__global__ void __launch_bounds__(256)
rope_q_wide_kernel(__nv_bfloat16* __restrict__ q, int H, int D, int rope, const int* __restrict__ positions,
                   const float* __restrict__ cos_t, const float* __restrict__ sin_t, long long ld_t) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int t = blockIdx.x, half = rope / 2, per = rope / 16;
  const float* ct = cos_t + (size_t)positions[t] * half;
  const float* st = sin_t + (size_t)positions[t] * half;
  for (int idx = threadIdx.x; idx < H * per; idx += blockDim.x) {
    const int h = idx / per, i = (idx - h * per) * 8;                // pairs i .. i + 7
    __nv_bfloat16* p = q + (size_t)t * ld_t + (size_t)h * D + (D - rope);
    uint4* p0 = reinterpret_cast<uint4*>(p + (INTERLEAVED ? 2 * i : i));
    uint4* p1 = reinterpret_cast<uint4*>(p + (INTERLEAVED ? 2 * i + 8 : i + half));
    float x[8], y[8], c[8], s[8], a[8], b[8];
    unpack8(*p0, x);
    unpack8(*p1, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      c[j] = ct[i + j];
      s[j] = st[i + j];
      a[j] = INTERLEAVED ? (j < 4 ? x[2 * (j & 3)] : y[2 * (j & 3)]) : x[j];
      b[j] = INTERLEAVED ? (j < 4 ? x[2 * (j & 3) + 1] : y[2 * (j & 3) + 1]) : y[j];
    }
    __align__(16) __nv_bfloat162 o[8];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 y0 = turn(a[j], b[j], c[j], s[j]), y1 = turn(a[j + 1], b[j + 1], c[j + 1], s[j + 1]);
      if (INTERLEAVED) {
        o[j] = __floats2bfloat162_rn(y0.x, y0.y);
        o[j + 1] = __floats2bfloat162_rn(y1.x, y1.y);
      } else {
        o[j / 2] = __floats2bfloat162_rn(y0.x, y1.x);
        o[4 + j / 2] = __floats2bfloat162_rn(y0.y, y1.y);
      }
    }
    *p0 = reinterpret_cast<const uint4*>(o)[0];
    *p1 = reinterpret_cast<const uint4*>(o)[1];
  }
}

}  // namespace bg

extern "C" {

// y = rmsnorm(x (+ residual)) * w; residual (if given) is updated in place with the sum.
// out (bf16, may be null), out_q/out_s (e4m3 + scales, may be null).  H % 128 == 0 when quantising,
// H % 8 == 0 always.
int bg_rmsnorm(const void* x, void* residual, const void* w, void* out, void* out_q, float* out_s, int s_stride,
               int T, int H, int ldx, int ldo, float eps, int pow2, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  if (H % 8 != 0 || (out_q != nullptr && H % 128 != 0)) return -1;
  if (H > 12256) return -1;                                    // within six vectors of eight a thread
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto R = reinterpret_cast<__nv_bfloat16*>(residual);
  auto W = reinterpret_cast<const __nv_bfloat16*>(w);
  auto O = reinterpret_cast<__nv_bfloat16*>(out);
  auto Q = reinterpret_cast<uint8_t*>(out_q);
  const int nv = (H + 8 * kNormThreads - 1) / (8 * kNormThreads);
#define BG_LAUNCH(ADD, QNT)                                                                                                                        \
  bg::launch_pdl(nv <= 1 ? rmsnorm_kernel<ADD, QNT, 1> : nv <= 2 ? rmsnorm_kernel<ADD, QNT, 2> : nv <= 4 ? rmsnorm_kernel<ADD, QNT, 4>            \
                                                                                                        : rmsnorm_kernel<ADD, QNT, 6>,            \
                 dim3(T), dim3(kNormThreads), 0, stream, X, R, W, O, Q, out_s, s_stride, H, ldx, ldo, eps, pow2)
  if (residual != nullptr && out_q != nullptr) BG_LAUNCH(true, true);
  else if (residual != nullptr) BG_LAUNCH(true, false);
  else if (out_q != nullptr) BG_LAUNCH(false, true);
  else BG_LAUNCH(false, false);
#undef BG_LAUNCH
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// mode 0: quantise x [T, K] (row stride ldx); mode 1: quantise silu(x[:, :K]) * x[:, K:2K].
// valid_rows (device int, may be null) limits the rows that are processed.
int bg_act_quant(int mode, const void* x, void* q, float* s, int s_stride, int T, int K, int ldx, int pow2,
                 const int* valid_rows, const int* row_src, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  if (K % 128 != 0) return -1;
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto Q = reinterpret_cast<uint8_t*>(q);
  const bool many = many_blocks(T, K);
  if (mode != 0 && many) {
    const int threads = K / 8 >= 256 ? 256 : (K / 8 + 31) / 32 * 32;
    bg::launch_pdl(silu_quant_rows_kernel, dim3(T), dim3(threads), 0, stream, X, Q, s, s_stride, K, ldx, pow2, valid_rows, row_src);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  auto kern = mode == 0 ? (many ? act_quant_kernel<0, 4> : act_quant_kernel<0, 1>) : act_quant_kernel<1, 1>;
  bg::launch_pdl(kern, dim3(walk_grid(T, K, many ? 4 : 1)), dim3(256), 0, stream, X, Q, s, s_stride, T, K, ldx, pow2, valid_rows, row_src);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bg_mla_kv_write(const void* kv_a, int ld, const void* w, const int* positions, const float* cos_t,
                    const float* sin_t, const long long* slots, void* cache, int T, int kv_lora, int rope, float eps,
                    int interleaved, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  bg::launch_pdl(mla_kv_write_kernel, dim3(T), dim3(128), 0, stream, reinterpret_cast<const __nv_bfloat16*>(kv_a), ld,
                                             reinterpret_cast<const __nv_bfloat16*>(w), positions, cos_t, sin_t, slots,
                                             reinterpret_cast<__nv_bfloat16*>(cache), kv_lora, rope, eps, interleaved);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bg_rope_q(void* q, int T, int H, int D, int rope, const int* positions, const float* cos_t, const float* sin_t,
              int interleaved, long long ld_t, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  auto Q = reinterpret_cast<__nv_bfloat16*>(q);
  const bool few = (long long)H * (rope / 2) <= 256 && T <= 1024;
  if (!few && rope % 16 == 0 && D % 8 == 0 && ld_t % 8 == 0 && reinterpret_cast<uintptr_t>(q) % 16 == 0)
    bg::launch_pdl(interleaved ? rope_q_wide_kernel<true> : rope_q_wide_kernel<false>, dim3(T), dim3(256), 0, stream, Q, H, D, rope, positions, cos_t, sin_t, ld_t);
  else
    bg::launch_pdl(rope_q_kernel, dim3(T), dim3(256), 0, stream, Q, H, D, rope, positions, cos_t, sin_t, interleaved, ld_t);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"

BG_TRACE_SETTER(elementwise)
