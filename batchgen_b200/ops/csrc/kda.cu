// Kimi Delta Attention (gated delta-rule linear attention): decode and short pieces token by token, longer pieces in chunks.
//
// Per head the layer keeps a state S [D keys x D values] (fp32) and the last three raw inputs of every
// q/k/v channel (the window of the width-4 causal depthwise convolution).  For each token, in order:
//
//   q, k, v  = silu(conv4(raw q, k, v))                   q, k then L2-normalised, q times `scale`
//   a        = exp(-exp(A_log[h]) * softplus(f + dt_bias))  per key channel (decay in (0, 1])
//   S        = diag(a) S
//   u        = sigmoid(beta) * (v - S^T k)
//   S        = S + k u^T
//   o        = S^T q
//   out      = o * rsqrt(mean(o^2) + eps) * w_norm * sigmoid(z)
//
// One CTA handles one (sequence, head); two threads share value column j of S in registers (D / 2 rows each),
// so S^T k, S^T q and the rank-one update need one exchange of two partial sums per token besides the two
// block-wide sums (the q/k norms and the output norm).  It serves decode and short pieces; longer pieces go through the chunk form
// below.  S^T q is taken from the decayed state in the same pass as
// S^T k (o = S'^T q + u * (k . q)), so the state is swept twice per token, not three times.  Decode is the
// one-token case and is bound by reading and writing the state (2 * D * D * 4 bytes per head and row).
//
// Replaces (by behaviour): the fused KDA decode kernel, the causal conv1d forward/update kernels and the
// chunked / recurrent delta-rule library calls of the reference (attention/kda_fused_decode.cu:147,429,707;
// conv1d/causal_conv1d.cu:446,679; batchgen/models/moonshotai/kimi_linear/serving_modules.py:579-722,1074,1202).
#include "common.cuh"

namespace bg {
namespace kda {

struct Params {
  const __nv_bfloat16* qkv;  // [T, >= 3*H*D]: raw q | k | v blocks of H*D each, row stride qkv_stride
  const __nv_bfloat16* f;    // [T, H*D] decay-gate pre-activation
  const __nv_bfloat16* beta; // [T, H]
  const __nv_bfloat16* z;    // [T, H*D] output gate
  int qkv_stride, f_stride, beta_stride, z_stride;
  const float* conv_w;       // [3*H*D, 4], tap 3 multiplies the current token
  const float* conv_b;       // [3*H*D] or null
  const float* A_log;        // [H]
  const float* dt_bias;      // [H*D]
  const float* norm_w;       // [D]
  float* conv_state;         // [slots, 3*H*D, 3] oldest first
  float* rec_state;          // [slots, H, D, D]
  const int* cu_seqlens;     // [nseq + 1] or null (one token per sequence: decode)
  const int* slots;          // [nseq]; < 0 skips the sequence
  const int* has_initial;    // [nseq] or null (null: always continue from the slot)
  __nv_bfloat16* out;        // [T, H*D] contiguous
  int H;
  float scale, eps;
  int most;                  // sequences of more tokens are left to the chunk form
  int whole;                 // rows of qkv and f in 16-byte pieces
};

__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

template <int D>
__global__ void __launch_bounds__(2 * D, 2) kda_seq_kernel(const Params p) {
  constexpr int R = D / 2;                 // state rows per thread: two threads share a value column
  constexpr int kWarpsHalf = D / 32;
  const int h = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x;
  const int half = tid / D, j = tid % D, warp = tid >> 5, lane = tid & 31;
  const int slot = p.slots[seq];
  if (slot < 0) return;
  const int t0 = p.cu_seqlens ? p.cu_seqlens[seq] : seq;
  const int t1 = p.cu_seqlens ? p.cu_seqlens[seq + 1] : seq + 1;
  if (t1 <= t0 || t1 - t0 > p.most) return;
  const int H = p.H, HD = H * D, c = h * D + j;
  const bool init = p.has_initial == nullptr || p.has_initial[seq] != 0;

  __shared__ __align__(16) float sq[2][D], sk[2][D], sa[2][D], sv[2][D];
  __shared__ float red[2][kWarpsHalf][3], red_o[kWarpsHalf];
  __shared__ float2 part[2][D];

  float S[R];
  float* Sg = p.rec_state + (((size_t)slot * H + h) * D + half * R) * D + j;
  if (init) {
#pragma unroll
    for (int i = 0; i < R; ++i) S[i] = Sg[(size_t)i * D];
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) S[i] = 0.f;
  }
  // half 0 runs the q and k channels of column j, half 1 the v channel and the decay gate
  const int n_ch = half == 0 ? 2 : 1;
  const int ch0 = half == 0 ? 0 : 2;
  float win[2][3], tap[2][4], bias[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (s < n_ch) {
      const size_t ch = (size_t)(ch0 + s) * HD + c;
      const float* cs = p.conv_state + ((size_t)slot * 3 * HD + ch) * 3;
#pragma unroll
      for (int i = 0; i < 3; ++i) win[s][i] = init ? cs[i] : 0.f;
      const float4 w4 = *reinterpret_cast<const float4*>(p.conv_w + ch * 4);
      tap[s][0] = w4.x; tap[s][1] = w4.y; tap[s][2] = w4.z; tap[s][3] = w4.w;
      bias[s] = p.conv_b ? p.conv_b[ch] : 0.f;
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) win[s][i] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) tap[s][i] = 0.f;
      bias[s] = 0.f;
    }
  }
  const float neg_a = -__expf(p.A_log[h]);
  const float dtb = p.dt_bias[c];
  const float nw = p.norm_w[j];

  // x[0..1]: raw conv inputs of this thread's channels; g: z (half 0) or f (half 1); bv: beta of the head
  auto load = [&](int t, float (&x)[2], float& g, float& bv) {
    const __nv_bfloat16* r = p.qkv + (size_t)t * p.qkv_stride + (size_t)ch0 * HD + c;
    x[0] = __bfloat162float(r[0]);
    x[1] = half == 0 ? __bfloat162float(r[HD]) : 0.f;
    g = half == 0 ? __bfloat162float(p.z[(size_t)t * p.z_stride + c]) : __bfloat162float(p.f[(size_t)t * p.f_stride + c]);
    bv = __bfloat162float(p.beta[(size_t)t * p.beta_stride + h]);
  };
  float nx[2], ng, nb;
  load(t0, nx, ng, nb);

  for (int t = t0; t < t1; ++t) {
    const int par = (t - t0) & 1;
    const float x[2] = {nx[0], nx[1]};
    const float g = ng, bv = nb;
    if (t + 1 < t1) load(t + 1, nx, ng, nb);              // next token's inputs fly during this token's math
    float y[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      y[s] = silu(bias[s] + tap[s][0] * win[s][0] + tap[s][1] * win[s][1] + tap[s][2] * win[s][2] + tap[s][3] * x[s]);
      win[s][0] = win[s][1]; win[s][1] = win[s][2]; win[s][2] = x[s];
    }
    if (half == 0) {
      sq[par][j] = y[0]; sk[par][j] = y[1];
      const float r0 = warp_sum(y[0] * y[0]), r1 = warp_sum(y[1] * y[1]), r2 = warp_sum(y[0] * y[1]);
      if (lane == 0) { red[par][warp][0] = r0; red[par][warp][1] = r1; red[par][warp][2] = r2; }
    } else {
      sv[par][j] = y[0];
      sa[par][j] = __expf(neg_a * softplus(g + dtb));
    }
    __syncthreads();
    float qq = 0.f, kk = 0.f, qk = 0.f;
#pragma unroll
    for (int w = 0; w < kWarpsHalf; ++w) { qq += red[par][w][0]; kk += red[par][w][1]; qk += red[par][w][2]; }
    const float rq = rsqrtf(qq + 1e-6f) * p.scale, rk = rsqrtf(kk + 1e-6f);
    // pass 1: decay, S'^T k and S'^T q over this thread's rows (raw k, q; the scalar norms scale the sums)
    float ak = 0.f, aq = 0.f;
    const float* pa = &sa[par][half * R];
    const float* pk = &sk[par][half * R];
    const float* pq = &sq[par][half * R];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 a4 = *reinterpret_cast<const float4*>(pa + i);
      const float4 k4 = *reinterpret_cast<const float4*>(pk + i);
      const float4 q4 = *reinterpret_cast<const float4*>(pq + i);
      S[i] *= a4.x;     ak = fmaf(S[i], k4.x, ak);     aq = fmaf(S[i], q4.x, aq);
      S[i + 1] *= a4.y; ak = fmaf(S[i + 1], k4.y, ak); aq = fmaf(S[i + 1], q4.y, aq);
      S[i + 2] *= a4.z; ak = fmaf(S[i + 2], k4.z, ak); aq = fmaf(S[i + 2], q4.z, aq);
      S[i + 3] *= a4.w; ak = fmaf(S[i + 3], k4.w, ak); aq = fmaf(S[i + 3], q4.w, aq);
    }
    part[half][j] = make_float2(ak, aq);
    __syncthreads();
    const float2 p0 = part[0][j], p1 = part[1][j];
    const float u = sigmoid(bv) * (sv[par][j] - (p0.x + p1.x) * rk);
    const float o = (p0.y + p1.y) * rq + u * (qk * rq * rk);
    const float uk = u * rk;
    // pass 2: rank-one update
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 k4 = *reinterpret_cast<const float4*>(pk + i);
      S[i] = fmaf(k4.x, uk, S[i]);
      S[i + 1] = fmaf(k4.y, uk, S[i + 1]);
      S[i + 2] = fmaf(k4.z, uk, S[i + 2]);
      S[i + 3] = fmaf(k4.w, uk, S[i + 3]);
    }
    if (half == 0) {
      const float ro = warp_sum(o * o);
      if (lane == 0) red_o[warp] = ro;
    }
    __syncthreads();
    if (half == 0) {
      float oo = 0.f;
#pragma unroll
      for (int w = 0; w < kWarpsHalf; ++w) oo += red_o[w];
      p.out[(size_t)t * HD + c] = __float2bfloat16(o * rsqrtf(oo / D + p.eps) * nw * sigmoid(g));
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) Sg[(size_t)i * D] = S[i];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (s < n_ch) {
      float* cs = p.conv_state + ((size_t)slot * 3 * HD + (size_t)(ch0 + s) * HD + c) * 3;
#pragma unroll
      for (int i = 0; i < 3; ++i) cs[i] = win[s][i];
    }
  }
}

// ---------------------------------------------------------------- prompts in chunk form
// The recurrence of 64 tokens at a time, all as precise as in fp32.  With G the running sum of the log decay inside the chunk, M[i, j] =
// sum_c k_i k_j exp(G_i - G_j) for j < i and P the same of q_i and k_j for j <= i, the writes are U = T (V - (K exp(G)) S) with
// T = (I + diag(b) M)^-1 diag(b), so that with W = T (K exp(G)), UV = T V, Q' = Q exp(G) - P W and O0 = P UV
//
//   U = UV - W S,   O = O0 + Q' S,   S <- exp(G_last) S + (K exp(G_last - G))^T U
//
// `chunk_prepare` makes W, Q', Kd = K exp(G_last - G), UV and O0 of every (chunk, head) at once, from the raw projections; `chunk_chain`
// walks the chunks of a (sequence, head, 64 value columns) on the tensor cores with S in registers; `chunk_finish` norms and gates whole heads.  Every
// exponent is a sum of the log decays of its own range of tokens, at most zero, and never a difference of running sums: behind a strong
// decay a difference would carry that decay's rounding into the weak ones after it (tokens of 2^-400 and of 2^-0.001 in turn: states off
// by 1.3e-5 with differences, 1.2e-7 so, 1.4e-7 token by token).  Products of different 16-token blocks meet at the border before the
// later one.
//
// The token-by-token kernel runs a barrier chain of some 2 us a token with a CTA per head.  One prompt of 4,096 tokens, 32 heads: 8,024 us a layer
// so, 913 in chunks (prepare 558, chain 328, finish 42); eight prompts of 300 to 1,024 tokens 1,014 (757, 224, 48).  With the chain in fp32
// FMAs, which shared memory fed at 86 % of its rate, 478 and 573 us of it; with a thread walking the whole chunk for one channel of one input,
// straight from global memory, prepare took 615 and 817, a third of that waiting for loads behind stores and branches.  Prepare has
// one CTA an SM and short steps, each waiting for the one before: inputs 6,100 clocks, convolutions and decays 12,400, the diagonal
// blocks of M and P 11,300, the others 18,200, the inverse 9,500, the products with P and T 12,700.
constexpr int kChunk = 64, kSub = 16, kPad = 132;      // kPad: rows of 128 floats that start 4 banks apart
constexpr int kPart = kChunk * 128;                                // elements of one [64, 128] result
constexpr int kPartRows = 9 * kChunk;                              // of a (chunk, head): three bf16 parts of [W; Q'] (128 rows), then three of Kd
constexpr int kAStride = 68;
constexpr float kLog2e = 1.4426950408889634f;

struct ChunkItem { int seq, t0, n, before; };                      // before: tokens of the sequence ahead of the chunk (up to 3 matter)
struct ChunkSeq { int seq, item0, items, first; };                 // first: the piece starts its sequence; t0 from the first item

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// x / d for d from 1 to 2^60 and |x| up to 2^60: an approximate reciprocal and one correction by the residual (Markstein 1990), which rounds
// like the division or to the number beside it at a third of its instructions (quotients whose residual is below the smallest float, as the
// reciprocal gives them)
__device__ __forceinline__ float quotient(float x, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = x * r;
  return fmaf(fmaf(-q, d, x), r, q);
}
__device__ __forceinline__ float silu_fast(float x) {
  const float d = 1.f + __expf(-x);
  float y = quotient(x, d);
  if (!(fabsf(x) < 40.f)) y = x / d;          // d may be infinite, x may not be finite
  return y;
}
// log(1 + e^x) = max(x, 0) + log(1 + e^-|x|), the logarithm as 2 artanh(s) with s = e / (2 + e) <= 1 / 3, whose series ends below 2^-26 of it with s^16;
// e^-|x| is at most one and keeps its relative precision, which e^x loses towards 20
__device__ __forceinline__ float softplus_series(float x) {
  const float e = __expf(-fabsf(x)), s = quotient(e, 2.f + e), s2 = s * s;
  float a = 2.f / 17.f;
  a = fmaf(a, s2, 2.f / 15.f);
  a = fmaf(a, s2, 2.f / 13.f);
  a = fmaf(a, s2, 2.f / 11.f);
  a = fmaf(a, s2, 2.f / 9.f);
  a = fmaf(a, s2, 2.f / 7.f);
  a = fmaf(a, s2, 2.f / 5.f);
  a = fmaf(a, s2, 2.f / 3.f);
  return fmaxf(x, 0.f) + fmaf(a * s2, s, 2.f * s);
}
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }
// four neighbours as parts, rows of 128, `step` elements from part to part
__device__ __forceinline__ void store_parts(__nv_bfloat16* dst, size_t step, float4 x) {
  float2 a = make_float2(x.x, x.y), b = make_float2(x.z, x.w);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    *reinterpret_cast<uint2*>(dst + i * step) = i < 2 ? make_uint2(cut_bf16x2(a), cut_bf16x2(b)) : make_uint2(last_bf16x2(a), last_bf16x2(b));
}

constexpr int kPrepThreads = 512;
constexpr int kBlocks = kChunk / kSub;
constexpr int kRawRows = kChunk + 3;
constexpr int kPrepareFloats = 4 * kChunk * kPad + (2 * kSub + 3 * kSub) * kPad + 2 * kChunk * kAStride + kChunk + kBlocks * 128;
static_assert(4 * kRawRows * 128 * 2 <= ((2 * kSub + 3 * kSub) * kPad + 2 * kChunk * kAStride) * 4, "raw inputs stand where block operands, M and P come");

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Block row A of M (first 256 threads) and P (the others) against the A blocks before it: a thread has a row and one column of each.  A is known to
// the compiler, or each block's loads would wait behind a branch (4,400 to 5,400 clocks a block row).
template <int A>
__device__ __forceinline__ void against(const float* ke, const float* qe, const float* kd, float* am, float* pm) {
  const int tid = threadIdx.x, i = tid & 15, jj = (tid >> 4) & 15;
  const float* left = (tid < 256 ? ke : qe) + i * kPad;
  float2 sum[A][2] = {};
#pragma unroll 8
  for (int c = 0; c < 128; c += 4) {
    const float4 x = *reinterpret_cast<const float4*>(left + c);
#pragma unroll
    for (int b = 0; b < A; ++b) {
      const float4 d = *reinterpret_cast<const float4*>(kd + (b * kSub + jj) * kPad + c);
      sum[b][0] = __ffma2_rn(make_float2(x.x, x.y), make_float2(d.x, d.y), sum[b][0]);
      sum[b][1] = __ffma2_rn(make_float2(x.z, x.w), make_float2(d.z, d.w), sum[b][1]);
    }
  }
#pragma unroll
  for (int b = 0; b < A; ++b)
    (tid < 256 ? am : pm)[(A * kSub + i) * kAStride + b * kSub + jj] = (sum[b][0].x + sum[b][1].x) + (sum[b][0].y + sum[b][1].y);
}

// Sixteen warps, one CTA an SM: the steps are short and each waits for the one before, so more warps hide more of a step's latency.
__global__ void __launch_bounds__(kPrepThreads, 1)
chunk_prepare(const Params p, const ChunkItem* __restrict__ items, __nv_bfloat16* __restrict__ parts, float* __restrict__ res, float* __restrict__ g_last) {
  constexpr int D = 128;
  extern __shared__ __align__(16) float sm[];
  float* kn = sm;                              // [64][kPad] each
  float* qn = kn + kChunk * kPad;
  float* lg = qn + kChunk * kPad;              // log2 decay of each token
  float* vv = lg + kChunk * kPad;
  float* ke = vv + kChunk * kPad;              // [16], then [16], then [48]: one block row's decayed operands; later K exp(G), W
  float* qe = ke + kSub * kPad;
  float* kd = qe + kSub * kPad;
  float* am = kd + 3 * kSub * kPad;            // [64][kAStride] M, then L = I + diag(b) M and its inverse, then T
  float* pm = am + kChunk * kAStride;          // [64][kAStride] P
  float* bs = pm + kChunk * kAStride;          // [64]
  float* tot = bs + kChunk;                    // [kBlocks][128] log2 decay over a block
  __nv_bfloat16* raw = reinterpret_cast<__nv_bfloat16*>(ke);      // [4][3 + 64][128] raw q, k, v and f, from three tokens ahead of the chunk; until they are used
  const ChunkItem it = items[blockIdx.x];
  const int h = blockIdx.y, H = p.H, HD = H * D;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // ---- inputs: all of the chunk's on their way at once
  if (p.whole) {
    for (int i = tid; i < 4 * kRawRows * 16; i += kPrepThreads) {
      const int part = i / (kRawRows * 16), t = i / 16 % kRawRows - 3, c = i % 16 * 8;
      if (t >= it.n || t < (part < 3 ? -min(it.before, 3) : 0)) continue;
      const __nv_bfloat16* src = part < 3 ? p.qkv + (ptrdiff_t)(it.t0 + t) * p.qkv_stride + part * HD : p.f + (size_t)(it.t0 + t) * p.f_stride;
      cp16(raw + (part * kRawRows + t + 3) * D + c, src + h * D + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  } else {
    for (int i = tid; i < 4 * kRawRows * D; i += kPrepThreads) {
      const int part = i / (kRawRows * D), t = i / D % kRawRows - 3, c = i % D;
      if (t >= it.n || t < (part < 3 ? -min(it.before, 3) : 0)) continue;
      const __nv_bfloat16* src = part < 3 ? p.qkv + (ptrdiff_t)(it.t0 + t) * p.qkv_stride + part * HD : p.f + (size_t)(it.t0 + t) * p.f_stride;
      raw[(part * kRawRows + t + 3) * D + c] = src[h * D + c];
    }
  }
  const int slot = p.slots[it.seq];
  if (slot < 0) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return;
  }
  float* out = res + ((size_t)blockIdx.x * H + h) * 2 * kPart;                     // UV | O
  __nv_bfloat16* wq_out = parts + ((size_t)blockIdx.x * H + h) * kPartRows * D;     // [3][128][128]
  __nv_bfloat16* kd_out = wq_out + 3 * 2 * kPart;                                   // [3][64][128]

  // ---- convolutions, SiLU, log decays: a thread has one channel of a block's sixteen tokens, of q, k, v and f in turn; all of them are read before the
  // first is stored: a store or a branch would hold up the loads behind it
  {
    const int j = tid & 127, c = h * D + j, b = (tid >> 7) * kSub;
    const bool init = p.has_initial == nullptr || p.has_initial[it.seq] != 0;
    const float beta = tid < min(it.n, kChunk) ? __bfloat162float(p.beta[(size_t)(it.t0 + tid) * p.beta_stride + h]) : 0.f;
    const float neg_a = -__expf(p.A_log[h]), dtb = p.dt_bias[c];
    float tap[3][4], bias[3], ahead[3][3] = {};                      // ahead: the three inputs before the block where the step does not have them
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      const int ch = part * HD + c;
      const float4 w = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch * 4);
      tap[part][0] = w.x; tap[part][1] = w.y; tap[part][2] = w.z; tap[part][3] = w.w;
      bias[part] = p.conv_b ? p.conv_b[ch] : 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (b == 0 && it.before < 3 - i && init) ahead[part][i] = p.conv_state[((size_t)slot * 3 * HD + ch) * 3 + i + it.before];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      const __nv_bfloat16* src = raw + (part * kRawRows + b) * D + j;
      float* dst = (part == 0 ? qn : part == 1 ? kn : vv) + b * kPad + j;
      float x[19], y[16];
#pragma unroll
      for (int i = 0; i < 19; ++i) x[i] = i < 3 && b == 0 && it.before < 3 - i ? ahead[part][i] : __bfloat162float(src[i * D]);
#pragma unroll
      for (int i = 0; i < 16; ++i) y[i] = silu_fast(bias[part] + tap[part][0] * x[i] + tap[part][1] * x[i + 1] + tap[part][2] * x[i + 2] + tap[part][3] * x[i + 3]);
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[i * kPad] = b + i < it.n ? y[i] : 0.f;
    }
    const __nv_bfloat16* src = raw + (3 * kRawRows + 3 + b) * D + j;
    float x[16], run = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __bfloat162float(src[i * D]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      x[i] = b + i < it.n ? neg_a * softplus_series(x[i] + dtb) * kLog2e : 0.f;
      run += x[i];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) lg[(b + i) * kPad + j] = x[i];
    tot[b / kSub * 128 + j] = run;
    if (tid < kChunk) bs[tid] = tid < it.n ? sigmoid(beta) : 0.f;
  }
  __syncthreads();
  // ---- unit q (times scale) and k, four tokens a warp
#pragma unroll
  for (int t = warp * 4; t < warp * 4 + 4; ++t) {
    float4 q = *reinterpret_cast<const float4*>(qn + t * kPad + lane * 4), k = *reinterpret_cast<const float4*>(kn + t * kPad + lane * 4);
    const float rq = rsqrtf(warp_sum(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w) + 1e-6f) * p.scale;
    const float rk = rsqrtf(warp_sum(k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w) + 1e-6f);
    *reinterpret_cast<float4*>(qn + t * kPad + lane * 4) = make_float4(q.x * rq, q.y * rq, q.z * rq, q.w * rq);
    *reinterpret_cast<float4*>(kn + t * kPad + lane * 4) = make_float4(k.x * rk, k.y * rk, k.z * rk, k.w * rk);
  }
  __syncthreads();
  // ---- M and P inside the blocks of 16: a warp per row i, lanes over the channels; the sums of a row's 16 columns of both meet in one
  // exchange that halves what a lane holds at every step: lane l ends with column l % 16 of M (l < 16) or P
#pragma unroll 1
  for (int i = warp; i < kChunk; i += 16) {
    const int b0 = i & ~(kSub - 1), r = i - b0;
    const float4 ki = *reinterpret_cast<const float4*>(kn + i * kPad + lane * 4), qi = *reinterpret_cast<const float4*>(qn + i * kPad + lane * 4);
    float4 run = make_float4(0.f, 0.f, 0.f, 0.f);                   // of tokens j + 1 .. r
    float v[32];
#pragma unroll
    for (int j = kSub - 1; j >= 0; --j) {
      v[j] = v[16 + j] = 0.f;
      if (j <= r) {
        const float4 kj = *reinterpret_cast<const float4*>(kn + (b0 + j) * kPad + lane * 4);
        const float4 lj = *reinterpret_cast<const float4*>(lg + (b0 + j) * kPad + lane * 4);
        const float4 e = make_float4(kj.x * ex2(run.x), kj.y * ex2(run.y), kj.z * ex2(run.z), kj.w * ex2(run.w));
        v[j] = j < r ? ki.x * e.x + ki.y * e.y + ki.z * e.z + ki.w * e.w : 0.f;
        v[16 + j] = qi.x * e.x + qi.y * e.y + qi.z * e.z + qi.w * e.w;
        run.x += lj.x; run.y += lj.y; run.z += lj.z; run.w += lj.w;
      }
    }
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
      const bool up = lane & half;
#pragma unroll
      for (int m = 0; m < half; ++m) {
        const float mine = up ? v[m + half] : v[m], give = up ? v[m] : v[m + half];
        v[m] = mine + __shfl_xor_sync(0xffffffffu, give, half);
      }
    }
    (lane < 16 ? am : pm)[i * kAStride + b0 + (lane & 15)] = v[0];
  }
  // ---- block row a against the blocks before it, decays split at the border before block a; half of the threads for M, half for P
  const int blk = tid >> 7, ch = tid & 127, walk = blk * kSub * kPad + ch;
#pragma unroll 1
  for (int a = 1; a < kChunk / kSub; ++a) {
    __syncthreads();
    // a thread walks one channel of a block, up from the border in block a, down to it in the others
    if (blk == a) {
      float run = 0.f;
#pragma unroll
      for (int i = 0; i < kSub; ++i) {
        run += lg[walk + i * kPad];
        const float e = ex2(run);
        ke[i * kPad + ch] = kn[walk + i * kPad] * e;
        qe[i * kPad + ch] = qn[walk + i * kPad] * e;
      }
    } else if (blk < a) {
      float run = 0.f;
      for (int m = blk + 1; m < a; ++m) run += tot[m * 128 + ch];
#pragma unroll
      for (int i = kSub - 1; i >= 0; --i) {
        kd[(blk * kSub + i) * kPad + ch] = kn[walk + i * kPad] * ex2(run);
        run += lg[walk + i * kPad];
      }
    }
    __syncthreads();
    if (a == 1) against<1>(ke, qe, kd, am, pm);
    else if (a == 2) against<2>(ke, qe, kd, am, pm);
    else against<3>(ke, qe, kd, am, pm);
  }
  __syncthreads();
  // ---- diagonal blocks of (I + diag(b) M)^-1: a thread of the first two warps solves for one column
  if (warp < 2) {
    const int b0 = tid & ~(kSub - 1), col = tid & (kSub - 1);
    float x[kSub];
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      const float bi = bs[b0 + i];
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) {
        const float y = am[(b0 + i) * kAStride + b0 + m] * x[m];
        if (m & 1) s1 += y;
        else s0 += y;
      }
      x[i] = (i == col ? 1.f : 0.f) - bi * (s0 + s1);
    }
    __syncwarp();                              // a block's 16 columns are lanes of one warp: M of the block is read
#pragma unroll
    for (int i = 0; i < kSub; ++i) am[(b0 + i) * kAStride + b0 + col] = x[i];
  }
  // ---- K exp(G) over the block operands, Q exp(G) in place, Kd and exp(G_last): a thread walks one channel of a block
  {
    float up = 0.f, down = 0.f;
    for (int m = 0; m < blk; ++m) up += tot[m * 128 + ch];
    for (int m = blk + 1; m < kBlocks; ++m) down += tot[m * 128 + ch];
#pragma unroll
    for (int i = kSub - 2; i >= 0; i -= 2) {                        // two tokens: neighbours swap one, so that a thread stores both channels of the other
      const float y1 = kn[walk + (i + 1) * kPad] * ex2(down);
      down += lg[walk + (i + 1) * kPad];
      const float y0 = kn[walk + i * kPad] * ex2(down);
      down += lg[walk + i * kPad];
      const bool odd = ch & 1;
      const float other = __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 1);
      float2 y = odd ? make_float2(other, y1) : make_float2(y0, other);
      uint32_t* dst = reinterpret_cast<uint32_t*>(kd_out + (blk * kSub + i + odd) * D + (ch & ~1));
      dst[0] = cut_bf16x2(y);
      dst[kPart / 2] = cut_bf16x2(y);
      dst[kPart] = last_bf16x2(y);
    }
    float e = 1.f;
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      up += lg[walk + i * kPad];
      e = ex2(up);
      ke[walk + i * kPad] = kn[walk + i * kPad] * e;
      qn[walk + i * kPad] *= e;
    }
    if (blk == kBlocks - 1) g_last[((size_t)blockIdx.x * H + h) * D + ch] = e;
  }
  // ---- the blocks below: X_ab = -X_aa (sum over b <= m < a of diag(b) M_am X_mb), a block row at a time; the sums stand in the places of
  // X_ab's transposed mirror above the diagonal.  Here and below what lies above a diagonal is left out, not multiplied by zero: a token
  // that is not finite stays out of the rows before it
#pragma unroll 1
  for (int a = 1; a < kChunk / kSub; ++a) {
    __syncthreads();
    for (int o = tid; o < a * 256; o += kPrepThreads) {
      const int b = o >> 8, i = (o >> 4) & 15, j = o & 15;
      const float* row = am + (a * kSub + i) * kAStride;
      float s = 0.f;
      for (int m = b * kSub; m < a * kSub; ++m) s = fmaf(row[m], am[m * kAStride + b * kSub + j], s);
      am[(b * kSub + i) * kAStride + a * kSub + j] = s * bs[a * kSub + i];
    }
    __syncthreads();
    for (int o = tid; o < a * 256; o += kPrepThreads) {
      const int b = o >> 8, i = (o >> 4) & 15, j = o & 15;
      float s = 0.f;
#pragma unroll
      for (int m = 0; m < kSub; ++m)
        if (m <= i) s = fmaf(am[(a * kSub + i) * kAStride + a * kSub + m], am[(b * kSub + m) * kAStride + a * kSub + j], s);
      am[(a * kSub + i) * kAStride + b * kSub + j] = -s;
    }
  }
  __syncthreads();
  for (int o = tid; o < kChunk * kChunk; o += kPrepThreads) {
    const int i = o >> 6, j = o & 63;
    if (j <= i) am[i * kAStride + j] *= bs[j];
  }
  __syncthreads();
  // ---- rows 8 g .. 8 g + 7 of a lower-triangular [64, 64] times a [64, 128], 4 columns a lane; a warp per (g, matrix), g and 7 - g on one
  // scheduler, so that all four have the same work
  const int grp = warp & 4 ? 7 - (warp & 3) : warp & 3;
  const bool second = warp & 8;
  float* mat = (second ? vv : ke) + lane * 4;
  auto product = [&](const float* tri, float2 (&x)[8][2]) {
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r][0] = x[r][1] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int j = 0; j < grp * 8; j += 4) {
      float4 l[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) l[m] = *reinterpret_cast<const float4*>(mat + (j + m) * kPad);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 t = *reinterpret_cast<const float4*>(tri + (grp * 8 + r) * kAStride + j);
        const float tm[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float2 t2 = twice(tm[m]);
          x[r][0] = __ffma2_rn(t2, make_float2(l[m].x, l[m].y), x[r][0]);
          x[r][1] = __ffma2_rn(t2, make_float2(l[m].z, l[m].w), x[r][1]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {                                   // the group's own columns, up to each row's diagonal
      const float4 l = *reinterpret_cast<const float4*>(mat + (grp * 8 + j) * kPad);
#pragma unroll
      for (int r = j; r < 8; ++r) {
        const float2 t2 = twice(tri[(grp * 8 + r) * kAStride + grp * 8 + j]);
        x[r][0] = __ffma2_rn(t2, make_float2(l.x, l.y), x[r][0]);
        x[r][1] = __ffma2_rn(t2, make_float2(l.z, l.w), x[r][1]);
      }
    }
  };
  float2 x[8][2];
  product(am, x);                               // W, UV
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int row = grp * 8 + r;
    const float4 y = make_float4(x[r][0].x, x[r][0].y, x[r][1].x, x[r][1].y);
    *reinterpret_cast<float4*>(mat + row * kPad) = y;
    if (second) *reinterpret_cast<float4*>(out + row * D + lane * 4) = y;
    else store_parts(wq_out + row * D + lane * 4, 2 * kPart, y);
  }
  __syncthreads();
  product(pm, x);                               // P W, P UV
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int row = grp * 8 + r;
    float4 y = make_float4(x[r][0].x, x[r][0].y, x[r][1].x, x[r][1].y);
    if (!second) {
      const float4 q = *reinterpret_cast<const float4*>(qn + row * kPad + lane * 4);
      store_parts(wq_out + kPart + row * D + lane * 4, 2 * kPart, make_float4(q.x - y.x, q.y - y.y, q.z - y.z, q.w - y.w));
    } else {
      *reinterpret_cast<float4*>(out + kPart + row * D + lane * 4) = y;
    }
  }
}

// ---- the chain on the tensor cores, every fp32 operand as three bf16 parts that sum up to it (common.cuh), all nine products.  Those of the leading
// parts have two accumulators, one for each half of the reduction, the small ones accumulators of their own, added in fp32: states are as near to 64
// bits as with fp32 FMAs or nearer (model-like decays 1.6e-7 against 1.7e-7; with the six largest products and one accumulator for the
// leading one 1.9e-7).
constexpr int kCols = 64;                                          // value columns of a CTA
constexpr int kChainThreads = 320;
constexpr int kTile = 64 * 128;                                    // bytes of 64 rows of 64 elements
constexpr int kWqBytes = 3 * 4 * kTile, kKdBytes = 3 * 2 * kTile, kSBytes = 3 * 2 * kTile, kUBytes = 3 * kTile;

struct ChainShared {
  uint64_t wq_full, wq_empty, kd_full, kd_empty, s_ready, u_ready, d1_done, d2_done;
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int kChainBytes = kWqBytes + kKdBytes + kSBytes + kUBytes + sizeof(ChainShared) + 1024;

// tiles whose rows of 64 columns lie behind each other, the reduction running over the rows (16 a step); the next 64 columns are `next` bytes on
__device__ __forceinline__ uint64_t desc_over_rows(uint32_t addr, uint32_t next) {
  return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | static_cast<uint64_t>(next >> 4) << 16 | static_cast<uint64_t>(1024 >> 4) << 32 |
         static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(2) << 61;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// 32 columns of one row as parts into [part][rows][64] tiles (swizzled as a TMA load would).  An infinity is infinite three times: what is cut from it
// leaves NaN, where its products with a finite number in fp32 are infinite.
__device__ __forceinline__ void put_parts(uint8_t* tiles, int part_bytes, int row, int half, const float (&x)[32]) {
  uint8_t* r = tiles + row * 128;
  auto piece = [&](int c) { return ((4 * half + c) ^ (row & 7)) << 4; };
  float2 odd = make_float2(0.f, 0.f);           // NaN once a rest is
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 e = make_float2(x[8 * c + 2 * i], x[8 * c + 2 * i + 1]);
      w[0][i] = cut_bf16x2(e);
      w[1][i] = cut_bf16x2(e);
      w[2][i] = last_bf16x2(e);
      odd = __ffma2_rn(e, make_float2(0.f, 0.f), odd);
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) *reinterpret_cast<uint4*>(r + m * part_bytes + piece(c)) = make_uint4(w[m][0], w[m][1], w[m][2], w[m][3]);
  }
  if (!(odd.x + odd.y == 0.f)) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (fabsf(x[j]) == INFINITY)
        for (int m = 0; m < 3; ++m) *reinterpret_cast<uint16_t*>(r + m * part_bytes + piece(j / 8) + j % 8 * 2) = x[j] > 0.f ? 0x7F80 : 0xFF80;
  }
}

// grid (value columns / 64, H, sequence pieces): walks a piece's chunks.  Warps 0..7: a thread holds 32 value columns of one key of S, takes
// U or O of one token's columns from the first product and the update from the second; warp 8 loads, warp 9 issues.
// Bound by the products (3,456 clocks a chunk) and four hand-overs between threads and tensor cores, one after the other.
__global__ void __launch_bounds__(kChainThreads, 1)
chunk_chain(const __grid_constant__ CUtensorMap map, const Params p, const ChunkSeq* __restrict__ seqs, float* __restrict__ res,
            const float* __restrict__ g_last, int* status) {
  constexpr int D = 128;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* wq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));      // [3][2 key halves][128 rows]
  uint8_t* kd = wq + kWqBytes;                  // [3][2 key halves][64 tokens]
  uint8_t* st = kd + kKdBytes;                  // [3][128 keys]
  uint8_t* ut = st + kSBytes;                   // [3][64 tokens]
  ChainShared& ss = *reinterpret_cast<ChainShared*>(ut + kUBytes);
  const ChunkSeq sq = seqs[blockIdx.z];
  const int h = blockIdx.y, H = p.H, c0 = blockIdx.x * kCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = p.slots[sq.seq];
  if (slot < 0) return;
  volatile int* abort_flag = &ss.abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(&ss.wq_full, 1); mbar_init(&ss.wq_empty, 1);
    mbar_init(&ss.kd_full, 1); mbar_init(&ss.kd_empty, 1);
    mbar_init(&ss.s_ready, 8); mbar_init(&ss.u_ready, 8);
    mbar_init(&ss.d1_done, 1); mbar_init(&ss.d2_done, 1);
    ss.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(&ss.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = ss.tmem_base;             // both products: leading parts (two halves of the reduction), small ones (three)
  bool ok = true;

  if (warp == 8) {
    if (elect_one()) {
      tma_prefetch_desc(&map);
      for (int c = 0; c < sq.items; ++c) {
        const int row = ((sq.item0 + c) * H + h) * kPartRows;
        if (!mbar_wait(&ss.wq_empty, (c & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
        mbar_expect_tx(&ss.wq_full, kWqBytes);
        for (int m = 0; m < 3; ++m)
          for (int half = 0; half < 2; ++half)
            for (int r = 0; r < 2; ++r)
              tma_load_2d(wq + ((m * 2 + half) * 2 + r) * kTile, &map, &ss.wq_full, half * 64, row + m * 2 * kChunk + r * kChunk);
        if (!mbar_wait(&ss.kd_empty, (c & 1) ^ 1, abort_flag, kTimeoutProducer)) { ok = false; break; }
        mbar_expect_tx(&ss.kd_full, kKdBytes);
        for (int m = 0; m < 3; ++m)
          for (int half = 0; half < 2; ++half)
            tma_load_2d(kd + (m * 2 + half) * kTile, &map, &ss.kd_full, half * 64, row + (6 + m) * kChunk);
      }
      if (ok) {                                 // the last copies are consumed
        if (mbar_wait(&ss.wq_empty, (sq.items - 1) & 1, abort_flag, kTimeoutProducer))
          mbar_wait(&ss.kd_empty, (sq.items - 1) & 1, abort_flag, kTimeoutProducer);
      } else {
        for (uint32_t i = 0; i < (1u << 16); ++i) __nanosleep(20);   // bounded grace period for copies in flight
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      // M = 128, bf16; the reduction of the first product lies along A's rows and down B's, of the second down both.  A's second and third part meet
      // B's three side by side in columns 2 .. 4 (of 64), its first part the second and third of B there too and the first one in
      // column 0 for the first half of the reduction, in 1 for the second
      constexpr uint32_t down_b = 1u << 16, down_a = 1u << 15;
      auto product = [&](int steps, auto a, uint32_t b, uint32_t next, uint32_t down) {
#pragma unroll
        for (int i = 1; i < 3; ++i)
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < steps)
              mma_f16(tm + 2 * kCols, a(i, k), desc_over_rows(b + k * 2048, next), make_idesc(128, 3 * kCols, 1, 1) | down, i > 1 || k > 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k < steps) {
            mma_f16(tm + 2 * kCols, a(0, k), desc_over_rows(b + next + k * 2048, next), make_idesc(128, 2 * kCols, 1, 1) | down, 1u);
            mma_f16(tm + (2 * k < steps ? 0 : kCols), a(0, k), desc_over_rows(b + k * 2048, next), make_idesc(128, kCols, 1, 1) | down,
                    k == 0 || 2 * k == steps ? 0u : 1u);
          }
      };
      for (int c = 0; c < sq.items; ++c) {
        if (!mbar_wait(&ss.wq_full, c & 1, abort_flag, kTimeoutMma) || !mbar_wait(&ss.s_ready, c & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        product(D / 16, [&](int i, int k) { return make_smem_desc_sw128(smem_u32(wq) + (i * 2 + k / 4) * 2 * kTile) + 2 * (k % 4); }, smem_u32(st), 2 * kTile,
                down_b);
        tc_commit(&ss.wq_empty);
        tc_commit(&ss.d1_done);
        if (!mbar_wait(&ss.kd_full, c & 1, abort_flag, kTimeoutMma) || !mbar_wait(&ss.u_ready, c & 1, abort_flag, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        product(kChunk / 16, [&](int i, int k) { return desc_over_rows(smem_u32(kd) + i * 2 * kTile + k * 2048, kTile); }, smem_u32(ut), kTile, down_b | down_a);
        tc_commit(&ss.kd_empty);
        tc_commit(&ss.d2_done);
      }
    }
  } else {
    const int half = warp >> 2, row = (warp & 3) * 32 + lane;        // row: a key of S; a row of [W; Q']
    const uint32_t at = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * 32;
    const bool init = !sq.first || p.has_initial == nullptr || p.has_initial[sq.seq] != 0;
    float* Sg = p.rec_state + (((size_t)slot * H + h) * D + row) * D + c0 + half * 32;
    float S[32];
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 x = init ? *reinterpret_cast<const float4*>(Sg + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
    }
    auto hand_over = [&](uint64_t* bar) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto done = [&](uint64_t* bar, int c) {
      if (!__all_sync(0xffffffffu, mbar_wait(bar, c & 1, abort_flag, kTimeoutEpilogue))) return false;
      tc_fence_after();
      return true;
    };
    auto take = [&](float (&d)[32]) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {                                  // 16 columns at a time
        uint32_t a[5][16];
#pragma unroll
        for (int i = 0; i < 5; ++i) tmem_ld16(tm + at + i * kCols + 16 * j, a[i]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float small = (__uint_as_float(a[2][i]) + __uint_as_float(a[3][i])) + __uint_as_float(a[4][i]);
          d[16 * j + i] = (__uint_as_float(a[0][i]) + small) + __uint_as_float(a[1][i]);
        }
      }
    };
    put_parts(st, 2 * kTile, row, half, S);
    hand_over(&ss.s_ready);
    for (int c = 0; c < sq.items; ++c) {
      const size_t item = (size_t)(sq.item0 + c) * H + h;
      float* add = res + item * 2 * kPart + (size_t)row * D + c0 + half * 32;      // rows of UV, then of O
      float x[32];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(add + i);
        x[i] = a.x; x[i + 1] = a.y; x[i + 2] = a.z; x[i + 3] = a.w;
      }
      const float g = g_last[item * D + row];
      if (!done(&ss.d1_done, c)) { ok = false; break; }
      float d[32];
      take(d);
      if (row < kChunk) {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] -= d[i];
        put_parts(ut, kTile, row, half, x);
      } else {
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(add + i) = make_float4(x[i] + d[i], x[i + 1] + d[i + 1], x[i + 2] + d[i + 2], x[i + 3] + d[i + 3]);
      }
      hand_over(&ss.u_ready);
      if (!done(&ss.d2_done, c)) { ok = false; break; }
      take(d);
#pragma unroll
      for (int i = 0; i < 32; ++i) S[i] = fmaf(g, S[i], d[i]);
      if (c + 1 < sq.items) {
        put_parts(st, 2 * kTile, row, half, S);
        hand_over(&ss.s_ready);
      }
    }
    if (ok)
#pragma unroll
      for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(Sg + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 9) tmem_dealloc(ss.tmem_base, 512);
  if (threadIdx.x == 0 && ss.abort_flag != 0 && status != nullptr) atomicMax(status, ss.abort_flag);
}

// out = o / sqrt(mean(o^2) + eps) * w * sigmoid(z), a warp per token of (chunk, head); the last chunk of a sequence's last piece leaves the
// convolution windows (the chunks of the step have read the old ones)
__global__ void __launch_bounds__(256)
chunk_finish(const Params p, const ChunkItem* __restrict__ items, const float* __restrict__ res) {
  constexpr int D = 128;
  const ChunkItem it = items[blockIdx.x];
  const int h = blockIdx.y, H = p.H, HD = H * D, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = p.slots[it.seq];
  if (slot < 0) return;
  const float4 w = *reinterpret_cast<const float4*>(p.norm_w + lane * 4);
  for (int t = warp; t < it.n; t += 8) {
    const float4 o = *reinterpret_cast<const float4*>(res + ((size_t)blockIdx.x * H + h) * 2 * kPart + kPart + t * D + lane * 4);
    const float rs = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / D + p.eps);
    const uint2 raw = *reinterpret_cast<const uint2*>(p.z + (size_t)(it.t0 + t) * p.z_stride + h * D + lane * 4);
    const float2 za = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 zb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    __align__(8) __nv_bfloat162 y[2] = {__floats2bfloat162_rn(o.x * rs * w.x * sigmoid(za.x), o.y * rs * w.y * sigmoid(za.y)),
                                        __floats2bfloat162_rn(o.z * rs * w.z * sigmoid(zb.x), o.w * rs * w.w * sigmoid(zb.y))};
    *reinterpret_cast<uint2*>(p.out + (size_t)(it.t0 + t) * HD + h * D + lane * 4) = *reinterpret_cast<const uint2*>(y);
  }
  const int end = p.cu_seqlens[it.seq + 1];
  if (it.t0 + it.n != end) return;
  const int have = it.before + it.n;                                 // tokens of the step (more than 3, else exactly that many)
  const bool init = p.has_initial == nullptr || p.has_initial[it.seq] != 0;
  for (int i = threadIdx.x; i < 3 * D; i += 256) {
    const int ch = i / D * HD + h * D + i % D;
    float* cs = p.conv_state + ((size_t)slot * 3 * HD + ch) * 3;
    float x[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {                                    // the input 3 - b tokens before the end
      if (have >= 3 - b) x[b] = __bfloat162float(p.qkv[(size_t)(end - 3 + b) * p.qkv_stride + ch]);
      else x[b] = init ? cs[b + have] : 0.f;
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) cs[b] = x[b];
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
// boxes of 64 rows of 64 elements out of rows of 128
static int make_parts_map(CUtensorMap* m, void* base, uint64_t rows) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return -1;
  cuuint64_t dims[2] = {128, rows};
  cuuint64_t strides[1] = {256};
  cuuint32_t box[2] = {64, 64};
  cuuint32_t es[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -2;
}

}  // namespace kda
}  // namespace bg

extern "C" {

// See bg::kda::Params for the layouts.  D = 64 or 128; nseq sequences, H heads (this rank's).  Sequences of at most `longest_short` tokens go
// token by token (0: none do); items [n_items, 4] and seqs [n_seqs, 4] (ChunkItem, ChunkSeq) list chunks of up to 64 tokens and the
// pieces they make, with scratch of n_items * H * (417 * 128) floats, on a 16-byte boundary.
int bg_kda_forward(const void* qkv, int qkv_stride, const void* f, int f_stride, const void* beta, int beta_stride,
                   const void* z, int z_stride, const float* conv_w, const float* conv_b, const float* A_log,
                   const float* dt_bias, const float* norm_w, float* conv_state, float* rec_state,
                   const int* cu_seqlens, const int* slots, const int* has_initial, void* out, int nseq, int H, int D,
                   float scale, float eps, const int* items, int n_items, const int* seqs, int n_seqs, int longest_short,
                   float* scratch, int* status, cudaStream_t stream) {
  using namespace bg::kda;
  if (nseq <= 0) return 0;
  if ((D != 64 && D != 128) || H <= 0) return -1;
  if (n_items > 0 && (D != 128 || H > 65535 || n_seqs <= 0 || n_seqs > 65535 || scratch == nullptr || cu_seqlens == nullptr || z_stride % 4 ||
                      reinterpret_cast<uintptr_t>(z) % 8))
    return -1;
  Params p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv);
  p.f = reinterpret_cast<const __nv_bfloat16*>(f);
  p.beta = reinterpret_cast<const __nv_bfloat16*>(beta);
  p.z = reinterpret_cast<const __nv_bfloat16*>(z);
  p.qkv_stride = qkv_stride; p.f_stride = f_stride; p.beta_stride = beta_stride; p.z_stride = z_stride;
  p.conv_w = conv_w; p.conv_b = conv_b; p.A_log = A_log; p.dt_bias = dt_bias; p.norm_w = norm_w;
  p.conv_state = conv_state; p.rec_state = rec_state;
  p.cu_seqlens = cu_seqlens; p.slots = slots; p.has_initial = has_initial;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.H = H; p.scale = scale; p.eps = eps;
  p.most = longest_short;
  p.whole = qkv_stride % 8 == 0 && f_stride % 8 == 0 && reinterpret_cast<uintptr_t>(qkv) % 16 == 0 && reinterpret_cast<uintptr_t>(f) % 16 == 0;
  if (n_items > 0) {
    static bg::DeviceOnce once_p, once_c;
    if (!bg::ensure_dynamic_smem(chunk_prepare, kPrepareFloats * 4, once_p) || !bg::ensure_dynamic_smem(chunk_chain, kChainBytes, once_c)) return -3;
    auto it = reinterpret_cast<const ChunkItem*>(items);
    const size_t pairs = (size_t)n_items * H;
    auto parts = reinterpret_cast<__nv_bfloat16*>(scratch);
    float* res = scratch + pairs * kPartRows * 64;
    float* g_last = res + pairs * 2 * kPart;
    CUtensorMap tm;
    if (make_parts_map(&tm, parts, pairs * kPartRows) != 0) return -4;
    chunk_prepare<<<dim3(n_items, H), kPrepThreads, kPrepareFloats * 4, stream>>>(p, it, parts, res, g_last);
    chunk_chain<<<dim3(128 / kCols, H, n_seqs), kChainThreads, kChainBytes, stream>>>(tm, p, reinterpret_cast<const ChunkSeq*>(seqs), res, g_last, status);
    chunk_finish<<<dim3(n_items, H), 256, 0, stream>>>(p, it, res);
  }
  if (longest_short <= 0) return cudaGetLastError() == cudaSuccess ? 0 : -2;
  dim3 grid(H, nseq);
  if (D == 128) kda_seq_kernel<128><<<grid, 256, 0, stream>>>(p);
  else kda_seq_kernel<64><<<grid, 128, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
