// MoE routing kernels for the single-GPU path and the NCCL baseline path:
//   router_topk      sigmoid (+bias) group-limited top-k / softmax top-k, one warp per token
//   moe_count        per-local-expert counts -> 128-aligned segment offsets
//   moe_scatter      (token, k) pairs -> grouped row positions
//   moe_gather_quant gather token rows into the expert-grouped buffer fused with e4m3 quantisation
//   moe_combine      out[t] = sum_k w[t,k] * y[pos[t,k]] (+ shared-expert output), fixed k order
//
// Replaces (by behaviour): batchgen_kernels/src/moe/routing/gate_sigmoid_topk.cu:72,304,
// gate_topk_softmax.cu:44, mgn/moe_fused_gate.cu:84, routing/dispatch_count_gather.cu:32-239,
// dispatch_scatter_3d.cu:152-345, routing/reduce_weighted_scatter.cu:27 and
// dispatch_scatter_3d.cu:366-661 (ordered reduce: the k order here is fixed, so results are
// bit-reproducible run to run).
#define BG_FILE_TAG 2      // kernel-trace ids of this file are (tag << 16) | line
#include "common.cuh"
#include "mx_parts.cuh"
#include "quant_blocks.cuh"

namespace bg {

constexpr int kMaxExperts = 1024;
constexpr int kMaxTopK = 16;

// One warp per token.  E <= 1024, K <= 16, n_group <= 32.
__global__ void __launch_bounds__(128)
router_topk_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ bias, int* __restrict__ idx_out,
                   float* __restrict__ w_out, int T, int E, int K, int n_group, int topk_group, int norm, float scale,
                   int softmax_mode, int group_max, const int* __restrict__ num_valid) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  __shared__ float choice_s[4][kMaxExperts];
  __shared__ float score_s[4][kMaxExperts];
  __shared__ float group_s[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  float* choice = choice_s[warp];
  float* score = score_s[warp];
  if (num_valid != nullptr && t >= *num_valid) {  // padding row: deterministic filler
    for (int k = lane; k < K; k += 32) {
      idx_out[(size_t)t * K + k] = -1;
      w_out[(size_t)t * K + k] = 0.f;
    }
    return;
  }
  const float* lrow = logits + (size_t)t * ldl;
  // scoring modes: 0 sigmoid, 1 softmax over the selected logits, 2 softmax over every expert, 3 sqrt(softplus)
  float rmax = -INFINITY, rinv = 0.f;
  if (softmax_mode == 2) {
    for (int e = lane; e < E; e += 32) rmax = fmaxf(rmax, lrow[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    float rsum = 0.f;
    for (int e = lane; e < E; e += 32) rsum += expf(lrow[e] - rmax);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
    rinv = 1.0f / rsum;
  }
  for (int e = lane; e < E; e += 32) {
    const float l = lrow[e];
    if (softmax_mode == 1) {
      score[e] = l;
      choice[e] = l;
    } else {
      float s;
      if (softmax_mode == 0) s = 1.0f / (1.0f + expf(-l));
      else if (softmax_mode == 2) s = expf(l - rmax) * rinv;
      else s = sqrtf(l > 20.f ? l : log1pf(expf(l)));
      score[e] = s;
      choice[e] = bias != nullptr ? s + bias[e] : s;
    }
  }
  __syncwarp();
  if (n_group > 1) {
    const int gs = E / n_group;
    if (lane < n_group) {
      float m1 = -INFINITY, m2 = -INFINITY;
      for (int i = 0; i < gs; ++i) {
        const float v = choice[lane * gs + i];
        if (v > m1) { m2 = m1; m1 = v; } else if (v > m2) { m2 = v; }
      }
      group_s[warp][lane] = group_max ? m1 : m1 + m2;
    }
    __syncwarp();
    // keep the topk_group best groups (ties -> lower index); lane g decides for group g
    if (lane < n_group) {
      const float mine = group_s[warp][lane];
      int better = 0;
      for (int g = 0; g < n_group; ++g) {
        const float o = group_s[warp][g];
        better += (o > mine) || (o == mine && g < lane);
      }
      if (better >= topk_group) {
        for (int i = 0; i < gs; ++i) choice[lane * gs + i] = -INFINITY;
      }
    }
    __syncwarp();
  }
  float wsum = 0.f;
  float my_w = 0.f;
  int my_i = -1;
  float sel_max = -INFINITY;
  for (int k = 0; k < K; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = choice[e];
      if (v > best) { best = v; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (bi == 0x7fffffff) bi = 0;
    if (k == 0) sel_max = best;
    float wv = score[bi];
    if (softmax_mode == 1) wv = expf(wv - sel_max);
    wsum += wv;
    if (lane == k) { my_w = wv; my_i = bi; }
    __syncwarp();
    if (lane == 0) choice[bi] = -INFINITY;
    __syncwarp();
  }
  if (lane < K) {
    float wv = my_w;
    if (softmax_mode == 1) wv = wv / wsum;
    else if (norm == 2 || (norm && K > 1)) wv = wv / (wsum + 1e-20f);
    idx_out[(size_t)t * K + lane] = my_i;
    w_out[(size_t)t * K + lane] = wv * scale;
  }
}

// Single block: counts of pairs routed to local experts [lo, hi) -> offsets with every segment
// start aligned to `align` rows; cursor[] zeroed for the scatter pass; total rows in offsets[El].
// Bound by latency: eight indices of a thread are in flight together, and the running sum over the experts is a warp's scan
// (one pair after the other and expert after expert: 4,096 tokens of 8 experts 25 -> 8 us, 160 of 4 6 -> 3).
__global__ void __launch_bounds__(1024)
moe_count_kernel(const int* __restrict__ topk_idx, int n_pairs, int lo, int hi, int align, int* __restrict__ offsets,
                 int* __restrict__ cursor, const int* __restrict__ num_valid, int K) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  __shared__ int cnt[kMaxExperts];
  const int El = hi - lo;
  for (int e = threadIdx.x; e < El; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  const int limit = (num_valid != nullptr) ? min(n_pairs, *num_valid * K) : n_pairs;
  for (int i0 = threadIdx.x; i0 < limit; i0 += 8 * blockDim.x) {
    int e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j * blockDim.x;
      e[j] = i < limit ? topk_idx[i] : lo - 1;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (e[j] >= lo && e[j] < hi) atomicAdd(&cnt[e[j] - lo], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, per = (El + 31) / 32, first = min(lane * per, El), last = min(first + per, El);
    int sum = 0;
    for (int e = first; e < last; ++e) sum += ((cnt[e] + align - 1) / align) * align;
    int run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += v;
    }
    if (lane == 31) offsets[El] = run;
    run -= sum;
    for (int e = first; e < last; ++e) {
      offsets[e] = run;
      run += ((cnt[e] + align - 1) / align) * align;
    }
  }
  for (int e = threadIdx.x; e < El; e += blockDim.x) cursor[e] = 0;
}

__global__ void moe_scatter_kernel(const int* __restrict__ topk_idx, int n_pairs, int K, int lo, int hi,
                                   const int* __restrict__ offsets, int* __restrict__ cursor, int* __restrict__ pos,
                                   int* __restrict__ src_row, const int* __restrict__ num_valid) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pairs) return;
  const int limit = (num_valid != nullptr) ? *num_valid * K : n_pairs;
  const int e = (i < limit) ? topk_idx[i] : -1;
  if (e >= lo && e < hi) {
    const int r = offsets[e - lo] + atomicAdd(&cursor[e - lo], 1);
    pos[i] = r;
    src_row[r] = i / K;
  } else {
    pos[i] = -1;
  }
}

// Gather hidden[src_row[r]] (bf16) and quantise to e4m3 with 1x128 scales; warps walk the grouped rows (quant_blocks.cuh).  Padding rows
// (src < 0) become zeros with scale 0 so they produce exact zeros, or are left untouched when `zero_padding` is 0 (the grouped GEMM is
// then given the real row counts).
template <int U>
__global__ void __launch_bounds__(256)
moe_gather_quant_kernel(const __nv_bfloat16* __restrict__ hidden, int ldh, const int* __restrict__ src_row,
                        const int* __restrict__ total_rows, uint8_t* __restrict__ q, float* __restrict__ s,
                        int s_stride, int cap, int K, int pow2, int zero_padding) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int lane = threadIdx.x & 31, rows = min(cap, *total_rows);
  for (BlockWalk<U> walk(rows, K); walk.more(); walk.next()) {
    const int r = walk.row, src = src_row[r];
    if (src < 0 && !zero_padding) continue;
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = walk.block(u, lane);
      raw[u] = src >= 0 && kb * 128 < K ? *reinterpret_cast<const uint4*>(hidden + (size_t)src * ldh + kb * 128 + (lane & 15) * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = walk.block(u, lane);
      if (kb * 128 >= K) continue;
      float f[8];
      unpack8(raw[u], f);
      const float sc = quant_block(f, q + (size_t)r * K + kb * 128 + (lane & 15) * 8, pow2, 0xffffu << (lane & 16));
      if ((lane & 15) == 0) s[(size_t)kb * s_stride + r] = src >= 0 ? sc : 0.f;
    }
  }
}

// The same by token: each is quantised once, its bytes and scales go to the row of every expert it has (pos [T, topk], < 0: none); padding rows
// stay untouched.  Bound by its bytes: 4,739 tokens of 7,168 to eight rows each 84 us, quantised
// again for every row 145 (floor 49); 256 tokens 11 against 18.
template <int U>
__global__ void __launch_bounds__(256)
moe_spread_quant_kernel(const __nv_bfloat16* __restrict__ hidden, int ldh, const int* __restrict__ pos, int topk, uint8_t* __restrict__ q, float* __restrict__ s,
                        int s_stride, int T, int K, int pow2) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int lane = threadIdx.x & 31;
  for (BlockWalk<U> walk(T, K); walk.more(); walk.next()) {
    const int t = walk.row, mine = lane < topk ? pos[(size_t)t * topk + lane] : -1;
    if (!__any_sync(0xffffffffu, mine >= 0)) continue;
    uint4 raw[U];
    uint2 bytes[U];
    float sc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kb = walk.block(u, lane);
      raw[u] = kb * 128 < K ? *reinterpret_cast<const uint4*>(hidden + (size_t)t * ldh + kb * 128 + (lane & 15) * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float f[8];
      unpack8(raw[u], f);
      sc[u] = quant_block(f, reinterpret_cast<uint8_t*>(&bytes[u]), pow2, 0xffffu << (lane & 16));
    }
    for (int j = 0; j < topk; ++j) {
      const int r = __shfl_sync(0xffffffffu, mine, j);
      if (r < 0) continue;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kb = walk.block(u, lane);
        if (kb * 128 >= K) continue;
        *reinterpret_cast<uint2*>(q + (size_t)r * K + kb * 128 + (lane & 15) * 8) = bytes[u];
        if ((lane & 15) == 0) s[(size_t)kb * s_stride + r] = sc[u];
      }
    }
  }
}

// out[t] = (extra[t] if given) + sum_k w[t,k] * y[pos[t,k]], k ascending.  A CTA per 1,024 columns of a
// token: a thread owns 8 columns and has the top-k rows' loads in flight together, so a 48-token decode step still fills
// the SMs instead of walking each row serially in 48 blocks.  256 threads with the chunks of a token
// far apart in the grid took 148 us for 4,739 tokens of 7,168 with eight rows each, now 135 (floor 105 for its bytes); 256 tokens 16.5 either way.
constexpr int kCombineThreads = 128;
__global__ void __launch_bounds__(kCombineThreads)
moe_combine_kernel(const __nv_bfloat16* __restrict__ y, int ldy, const int* __restrict__ pos,
                   const float* __restrict__ w, const __nv_bfloat16* __restrict__ extra, int lde,
                   __nv_bfloat16* __restrict__ out, int ldo, int K, int H, int out_fp32) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int chunks = (H / 8 + kCombineThreads - 1) / kCombineThreads, t = blockIdx.x / chunks;
  __shared__ int p_s[kMaxTopK];
  __shared__ float w_s[kMaxTopK];
  if (threadIdx.x < K) {
    p_s[threadIdx.x] = pos[(size_t)t * K + threadIdx.x];
    w_s[threadIdx.x] = w[(size_t)t * K + threadIdx.x];
  }
  __syncthreads();
  const int v = (blockIdx.x - t * chunks) * kCombineThreads + threadIdx.x;
  if (v < H / 8) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 8) {
      uint4 raw[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + j;
        const int p = k < K ? p_s[k] : -1;
        raw[j] = p >= 0 ? *reinterpret_cast<const uint4*>(y + (size_t)p * ldy + v * 8) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + j;
        if (k >= K || p_s[k] < 0) continue;
        const float wk = w_s[k];
        const __nv_bfloat162* yp = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 a = __bfloat1622float2(yp[i]);
          acc[2 * i] = fmaf(wk, a.x, acc[2 * i]);
          acc[2 * i + 1] = fmaf(wk, a.y, acc[2 * i + 1]);
        }
      }
    }
    if (extra != nullptr) {
      uint4 raw = *reinterpret_cast<const uint4*>(extra + (size_t)t * lde + v * 8);
      const __nv_bfloat162* ep = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 a = __bfloat1622float2(ep[i]);
        acc[2 * i] += a.x;
        acc[2 * i + 1] += a.y;
      }
    }
    if (out_fp32) {
      float* o = reinterpret_cast<float*>(out) + (size_t)t * ldo + v * 8;
      *reinterpret_cast<float4*>(o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      *reinterpret_cast<float4*>(o + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
      __align__(16) __nv_bfloat162 o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
      *reinterpret_cast<uint4*>(out + (size_t)t * ldo + v * 8) = *reinterpret_cast<const uint4*>(o);
    }
  }
}

// Gated activation of bf16 rows [gate | up] of 2 F columns -> [F], in fp32, rounded once.  KIND 0: SiLU(g) u; 1: GPT-OSS, g clamped above
// and u on both sides at `limit`, (u + 1) g sigmoid(1.702 g); 2: the same clamps, SiLU(g) u.  Rows past *total_rows, and padding rows of
// an expert's segment (row_src < 0), are skipped: blocks walk the rows, so a capacity far above the rows that are present costs
// nothing.  Bound by reading 4 F and writing 2 F bytes a row.  As tensor operations it was some ten passes in fp32 over the whole capacity:
// 4 us instead of some 1,000 us for one token and 4 of 128 experts of 3,072 columns (16,512 rows of capacity); 18,600 rows of the same
// width take 97 us (3.5 TB/s), bound by the exponential and the division, which stay those of fp32: __expf and __fdividef took 64 us, but
// their error grows with |g| (1.5e-6 of the value at 20) and their quotient is zero past 2^126.
// A clamp lets a NaN through, like the tensor operation does.
// PARTS: the rows leave as the 4-bit product's operand (mx_parts.cuh) instead of bf16, from the same rounded values.
template <int KIND, bool PARTS>
__global__ void __launch_bounds__(256)
gated_rows_kernel(const __nv_bfloat16* __restrict__ z, long long ldz, __nv_bfloat16* __restrict__ out, int ldo, int rows, int F, float limit,
                  const int* __restrict__ total_rows, const int* __restrict__ row_src, mxp::Parts parts) {
  bg::pdl_prologue((BG_FILE_TAG << 16) | __LINE__);
  const int n = total_rows != nullptr ? min(rows, *total_rows) : rows;
  for (int r = blockIdx.x; r < n; r += gridDim.x) {
    if (row_src != nullptr && row_src[r] < 0) continue;
    const __nv_bfloat16* zr = z + (size_t)r * ldz;
    for (int v = threadIdx.x; v < F / 8; v += blockDim.x) {
      const uint4 graw = *reinterpret_cast<const uint4*>(zr + v * 8), uraw = *reinterpret_cast<const uint4*>(zr + F + v * 8);
      const __nv_bfloat162* gp = reinterpret_cast<const __nv_bfloat162*>(&graw);
      const __nv_bfloat162* up = reinterpret_cast<const __nv_bfloat162*>(&uraw);
      auto one = [&](float g, float u) {
        if (KIND != 0) {
          g = g > limit ? limit : g;
          u = u > limit ? limit : u < -limit ? -limit : u;
        }
        return KIND == 1 ? (u + 1.f) * g / (1.f + expf(-1.702f * g)) : g / (1.f + expf(-g)) * u;
      };
      __align__(16) __nv_bfloat162 o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 g = __bfloat1622float2(gp[i]), u = __bfloat1622float2(up[i]);
        o[i] = __floats2bfloat162_rn(one(g.x, u.x), one(g.y, u.y));
      }
      if (PARTS) {                               // F is a multiple of 32: a block's four lanes stay together
        const mxp::Split<8> s(o);
        s.store(parts, r, v * 8);
      } else {
        *reinterpret_cast<uint4*>(out + (size_t)r * ldo + v * 8) = *reinterpret_cast<const uint4*>(o);
      }
    }
  }
}

template <bool PARTS>
static int gated_rows(int kind, const void* z, long long ldz, void* out, int ldo, int rows, int F, float limit, const int* total_rows,
                      const int* row_src, int num_sms, const mxp::Parts& parts, cudaStream_t stream) {
  const dim3 grid(min(rows, num_sms * 16)), block(min(256, (F / 8 + 31) / 32 * 32));
  auto kern = kind == 0 ? gated_rows_kernel<0, PARTS> : kind == 1 ? gated_rows_kernel<1, PARTS> : gated_rows_kernel<2, PARTS>;
  bg::launch_pdl(kern, grid, block, 0, stream, reinterpret_cast<const __nv_bfloat16*>(z), ldz, reinterpret_cast<__nv_bfloat16*>(out), ldo, rows, F, limit,
                 total_rows, row_src, parts);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace bg

extern "C" {

// z [rows, ldz] bf16 -> out [rows, ldo]; F, ldz and ldo multiples of 8.  total_rows, row_src: device, or null.
int bg_gated_rows(int kind, const void* z, long long ldz, void* out, int ldo, int rows, int F, float limit, const int* total_rows,
                  const int* row_src, int num_sms, cudaStream_t stream) {
  using namespace bg;
  if (rows <= 0 || F <= 0) return 0;
  if (F % 8 || ldz % 8 || ldo % 8 || ldz < 2ll * F || ldo < F || kind < 0 || kind > 2) return -1;
  return gated_rows<false>(kind, z, ldz, out, ldo, rows, F, limit, total_rows, row_src, num_sms, mxp::Parts{}, stream);
}

// The same rows as parts p [rows / 8 rounded up][2][8][F] and scales s [F / 128 rounded up][rows][4] of the 4-bit product; F a multiple of 32.
int bg_gated_parts(int kind, const void* z, long long ldz, void* p, void* s, int rows, int F, float limit, const int* total_rows,
                   const int* row_src, int num_sms, cudaStream_t stream) {
  using namespace bg;
  if (rows <= 0 || F <= 0) return 0;
  if (F % 32 || ldz % 8 || ldz < 2ll * F || kind < 0 || kind > 2) return -1;
  const mxp::Parts parts{reinterpret_cast<uint8_t*>(p), reinterpret_cast<uint8_t*>(s), rows, F};
  return gated_rows<true>(kind, z, ldz, nullptr, 0, rows, F, limit, total_rows, row_src, num_sms, parts, stream);
}

// logits: rows of E values, ldl apart; norm: weights divided by their sum, 1 unless K is 1, 2 always; group_max: a group counts with
// its best expert instead of its best two
int bg_router_topk(const float* logits, int ldl, const float* bias, int* idx, float* w, int T, int E, int K, int n_group,
                   int topk_group, int norm, float scale, int softmax_mode, int group_max, const int* num_valid,
                   cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  if (E > kMaxExperts || K > kMaxTopK || K > E || ldl < E || n_group > 32 || (n_group > 1 && E % n_group != 0)) return -1;
  bg::launch_pdl(router_topk_kernel, dim3((T + 3) / 4), dim3(128), 0, stream, logits, ldl, bias, idx, w, T, E, K, n_group, topk_group, norm, scale,
                                                      softmax_mode, group_max, num_valid);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// hidden [T, ldh] quantised to the rows pos [T, topk] (negative: none) of q [.., K] and s; topk at most 32
int bg_moe_spread_quant(const void* hidden, int ldh, const int* pos, int topk, void* q, float* s, int s_stride, int T, int K, int pow2,
                        cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  if (K % 128 != 0 || topk <= 0 || topk > 32) return -1;
  const bool many = many_blocks(T, K);
  bg::launch_pdl(many ? moe_spread_quant_kernel<4> : moe_spread_quant_kernel<1>, dim3(walk_grid(T, K, many ? 4 : 1)), dim3(256), 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(hidden), ldh, pos, topk, reinterpret_cast<uint8_t*>(q), s, s_stride, T, K, pow2);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Builds offsets [El+1], pos [T*K], src_row [cap] (pre-filled with -1 here) for experts [lo, hi).
int bg_moe_permute(const int* topk_idx, int T, int K, int lo, int hi, int align, int* offsets, int* cursor, int* pos,
                   int* src_row, int cap, const int* num_valid, cudaStream_t stream) {
  using namespace bg;
  if (hi - lo > kMaxExperts) return -1;
  if (cudaMemsetAsync(src_row, 0xFF, (size_t)cap * sizeof(int), stream) != cudaSuccess) return -3;
  const int n_pairs = T * K;
  bg::launch_pdl(moe_count_kernel, dim3(1), dim3(1024), 0, stream, topk_idx, n_pairs, lo, hi, align, offsets, cursor, num_valid, K);
  if (n_pairs > 0)
    bg::launch_pdl(moe_scatter_kernel, dim3((n_pairs + 255) / 256), dim3(256), 0, stream, topk_idx, n_pairs, K, lo, hi, offsets, cursor, pos,
                                                                 src_row, num_valid);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bg_moe_gather_quant(const void* hidden, int ldh, const int* src_row, const int* total_rows, void* q, float* s,
                        int s_stride, int cap, int K, int pow2, int zero_padding, cudaStream_t stream) {
  using namespace bg;
  if (cap <= 0) return 0;
  if (K % 128 != 0) return -1;
  const bool many = many_blocks(cap, K);
  bg::launch_pdl(many ? moe_gather_quant_kernel<4> : moe_gather_quant_kernel<1>, dim3(walk_grid(cap, K, many ? 4 : 1)), dim3(256), 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(hidden), ldh, src_row, total_rows, reinterpret_cast<uint8_t*>(q), s, s_stride, cap, K, pow2, zero_padding);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bg_moe_combine(const void* y, int ldy, const int* pos, const float* w, const void* extra, int lde, void* out,
                   int ldo, int T, int K, int H, int out_fp32, cudaStream_t stream) {
  using namespace bg;
  if (T <= 0) return 0;
  if (K > kMaxTopK || H % 8 != 0) return -1;
  bg::launch_pdl(moe_combine_kernel, dim3(T * ((H / 8 + kCombineThreads - 1) / kCombineThreads)), dim3(kCombineThreads), 0, stream, reinterpret_cast<const __nv_bfloat16*>(y), ldy, pos, w,
                                            reinterpret_cast<const __nv_bfloat16*>(extra), lde,
                                            reinterpret_cast<__nv_bfloat16*>(out), ldo, K, H, out_fp32);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"

BG_TRACE_SETTER(moe_route)
