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
// The recurrence of 64 tokens at a time, all in fp32.  With G the running sum of the log decay inside the chunk, M[i, j] =
// sum_c k_i k_j exp(G_i - G_j) for j < i and P the same of q_i and k_j for j <= i, the writes are U = T (V - (K exp(G)) S) with
// T = (I + diag(b) M)^-1 diag(b), so that with W = T (K exp(G)), UV = T V, Q' = Q exp(G) - P W and O0 = P UV
//
//   U = UV - W S,   O = O0 + Q' S,   S <- exp(G_last) S + (K exp(G_last - G))^T U
//
// `chunk_prepare` makes W, Q', Kd = K exp(G_last - G), UV and O0 of every (chunk, head) at once, from the raw projections; `chunk_chain`
// walks the chunks of a (sequence, head, 32 value columns) with S in shared memory; `chunk_finish` norms and gates whole heads.  Every
// exponent is a sum of the log decays of its own range of tokens, at most zero, and never a difference of running sums: behind a strong
// decay a difference would carry that decay's rounding into the weak ones after it (tokens of 2^-400 and of 2^-0.001 in turn: states off
// by 1.3e-5 with differences, 1.2e-7 so, 1.4e-7 token by token).  Products of different 16-token blocks meet at the border before the
// later one.
//
// The token-by-token kernel runs a barrier chain of some 2 us a token with a CTA per head.  Here the chain's limit is what shared memory
// delivers to the fp32 FMAs (86 % of its rate), of which a token and head has about 75,000, two thirds of them in the chain; prepare waits at its
// short steps' barriers (shared memory 53 %, issue slots 42 %).  One prompt of 4,096 tokens, 32 heads: 8,086 -> 1,226
// us a layer (prepare 605, chain 466, finish 42); with two thirds of the warps and a column-by-column inverse prepare took 833.
constexpr int kChunk = 64, kSub = 16, kPad = 132, kCols = 32;      // kPad: rows of 128 floats that start 4 banks apart
constexpr int kPart = kChunk * 128;                                // floats of one [64, 128] result
constexpr int kItemFloats = 5 * kPart;                             // W | Q' | Kd | UV | O of a (chunk, head)
constexpr int kAStride = 68;
constexpr float kLog2e = 1.4426950408889634f;

struct ChunkItem { int seq, t0, n, before; };                      // before: tokens of the sequence ahead of the chunk (up to 3 matter)
struct ChunkSeq { int seq, item0, items, first; };                 // first: the piece starts its sequence; t0 from the first item

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }

constexpr int kPrepThreads = 512;
constexpr int kBlocks = kChunk / kSub;
constexpr int kPrepareFloats = 4 * kChunk * kPad + (2 * kSub + 3 * kSub) * kPad + 2 * kChunk * kAStride + kChunk + kBlocks * 128;

// Sixteen warps, one CTA an SM: the steps are short and each waits for the one before, so more warps hide more of a step's latency.
__global__ void __launch_bounds__(kPrepThreads, 1)
chunk_prepare(const Params p, const ChunkItem* __restrict__ items, float* __restrict__ res, float* __restrict__ g_last) {
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
  const ChunkItem it = items[blockIdx.x];
  const int h = blockIdx.y, H = p.H, HD = H * D;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slot = p.slots[it.seq];
  if (slot < 0) return;
  float* out = res + ((size_t)blockIdx.x * H + h) * kItemFloats;

  // ---- convolutions, SiLU, log decays: a thread walks the chunk for one channel of q, k, v or f
  {
    const int part = tid >> 7, j = tid & 127, c = h * D + j, ch = part * HD + c;
    const bool init = p.has_initial == nullptr || p.has_initial[it.seq] != 0;
    const __nv_bfloat16* src = part < 3 ? p.qkv + (size_t)it.t0 * p.qkv_stride + ch : p.f + (size_t)it.t0 * p.f_stride + c;
    const int stride = part < 3 ? p.qkv_stride : p.f_stride;
    float win[3] = {0.f, 0.f, 0.f}, tap[4] = {0.f, 0.f, 0.f, 0.f}, bias = 0.f;
    if (part < 3) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {            // the inputs 3, 2, 1 tokens ahead of the chunk: earlier tokens of the step, else the state
        const int back = 3 - i;
        if (it.before >= back) win[i] = __bfloat162float(src[-(ptrdiff_t)back * stride]);
        else if (init) win[i] = p.conv_state[((size_t)slot * 3 * HD + ch) * 3 + i + it.before];
      }
      const float4 w = *reinterpret_cast<const float4*>(p.conv_w + (size_t)ch * 4);
      tap[0] = w.x; tap[1] = w.y; tap[2] = w.z; tap[3] = w.w;
      bias = p.conv_b ? p.conv_b[ch] : 0.f;
    }
    const float neg_a = -__expf(p.A_log[h]), dtb = p.dt_bias[c];
    float* dst = (part == 0 ? qn : part == 1 ? kn : part == 2 ? vv : lg) + j;
    __nv_bfloat16 x[2][16];
    auto load = [&](int b, __nv_bfloat16 (&v)[16]) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = src[(size_t)min(b + i, it.n - 1) * stride];
    };
    load(0, x[0]);
#pragma unroll
    for (int b = 0; b < kChunk; b += 16) {
      if (b + 16 < kChunk) load(b + 16, x[(b / 16 + 1) & 1]);
      const __nv_bfloat16 (&v)[16] = x[(b / 16) & 1];
      float run = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const bool in = b + i < it.n;
        const float xi = __bfloat162float(v[i]);
        if (part < 3) {
          const float y = silu(bias + tap[0] * win[0] + tap[1] * win[1] + tap[2] * win[2] + tap[3] * xi);
          win[0] = win[1]; win[1] = win[2]; win[2] = xi;
          dst[(b + i) * kPad] = in ? y : 0.f;
        } else {
          const float g = in ? neg_a * softplus(xi + dtb) * kLog2e : 0.f;
          run += g;
          dst[(b + i) * kPad] = g;
        }
      }
      if (part == 3) tot[b / 16 * 128 + j] = run;
    }
    if (tid < kChunk) bs[tid] = tid < it.n ? sigmoid(__bfloat162float(p.beta[(size_t)(it.t0 + tid) * p.beta_stride + h])) : 0.f;
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
    const int i = tid & 15, jj = (tid >> 4) & 15;
    const float* left = (tid < 256 ? ke : qe) + i * kPad;
    float2 sum[3][2] = {};
#pragma unroll 4
    for (int c = 0; c < D; c += 4) {
      const float4 x = *reinterpret_cast<const float4*>(left + c);
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if (b < a) {
          const float4 d = *reinterpret_cast<const float4*>(kd + (b * kSub + jj) * kPad + c);
          sum[b][0] = __ffma2_rn(make_float2(x.x, x.y), make_float2(d.x, d.y), sum[b][0]);
          sum[b][1] = __ffma2_rn(make_float2(x.z, x.w), make_float2(d.z, d.w), sum[b][1]);
        }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (b < a)
        (tid < 256 ? am : pm)[(a * kSub + i) * kAStride + b * kSub + jj] = (sum[b][0].x + sum[b][1].x) + (sum[b][0].y + sum[b][1].y);
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
    for (int i = kSub - 1; i >= 0; --i) {
      out[2 * kPart + (blk * kSub + i) * D + ch] = kn[walk + i * kPad] * ex2(down);
      down += lg[walk + i * kPad];
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
  // ---- rows 8 g .. 8 g + 7 of a lower-triangular [64, 64] times a [64, 128], 4 columns a lane; a warp per (g, matrix)
  const int grp = warp >> 1;
  float* mat = (warp & 1 ? vv : ke) + lane * 4;
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
    *reinterpret_cast<float4*>(out + (warp & 1 ? 3 : 0) * kPart + row * D + lane * 4) = y;
  }
  __syncthreads();
  product(pm, x);                               // P W, P UV
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int row = grp * 8 + r;
    float4 y = make_float4(x[r][0].x, x[r][0].y, x[r][1].x, x[r][1].y);
    if (!(warp & 1)) {
      const float4 q = *reinterpret_cast<const float4*>(qn + row * kPad + lane * 4);
      y = make_float4(q.x - y.x, q.y - y.y, q.z - y.z, q.w - y.w);
    }
    *reinterpret_cast<float4*>(out + (warp & 1 ? 4 : 1) * kPart + row * D + lane * 4) = y;
  }
}

constexpr int kChainFloats = 2 * 128 * kPad + kChunk * 128 + kCols * kPad + kChunk * kCols * 2;

__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// grid (value columns / 32, H, sequence pieces): walks a piece's chunks, S of 32 value columns in shared memory as [column][key].
// W and Q' of the next chunk and Kd of this one arrive under the products.
__global__ void __launch_bounds__(256, 1)
chunk_chain(const Params p, const ChunkItem* __restrict__ items, const ChunkSeq* __restrict__ seqs, float* __restrict__ res,
            const float* __restrict__ g_last) {
  constexpr int D = 128;
  extern __shared__ __align__(16) float sm[];
  float* wq2 = sm;                              // two of [128][kPad]: rows of W, then of Q'
  float* kd = wq2 + 2 * 128 * kPad;                  // [64][128]
  float* st = kd + kChunk * 128;                // [32][kPad]
  float2* u2 = reinterpret_cast<float2*>(st + kCols * kPad);       // [64][32] (u, u)
  const ChunkSeq sq = seqs[blockIdx.z];
  const int h = blockIdx.y, H = p.H, c0 = blockIdx.x * kCols;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slot = p.slots[sq.seq];
  if (slot < 0) return;
  const bool init = !sq.first || p.has_initial == nullptr || p.has_initial[sq.seq] != 0;
  float* Sg = p.rec_state + ((size_t)slot * H + h) * D * D + c0;
  auto item = [&](int c) { return res + ((size_t)(sq.item0 + c) * H + h) * kItemFloats; };
  auto fetch_wq = [&](int c) {
    float* wq = wq2 + (c & 1) * 128 * kPad;
    if (c < sq.items)
      for (int i = tid; i < 128 * 32; i += 256) cp16(wq + (i >> 5) * kPad + (i & 31) * 4, item(c) + i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto fetch_kd = [&](int c) {
    if (c < sq.items)
      for (int i = tid; i < kChunk * 32; i += 256) cp16(kd + i * 4, item(c) + 2 * kPart + i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch_wq(0);
  fetch_kd(0);
  for (int i = tid; i < D * kCols; i += 256) st[(i % kCols) * kPad + i / kCols] = init ? Sg[(size_t)(i / kCols) * D + i % kCols] : 0.f;
  // first phase: rows 16 w + rg + 4 q (q < 4) of [W; Q'], columns cg + 8 q
  const int rg = lane >> 3, cg = lane & 7;
  // second phase: keys k0 .. k0 + 7, columns e0, e0 + 1
  const int k0 = (warp & 3) * 32 + (lane >> 3) * 8, e0 = (warp >> 2) * 16 + (lane & 7) * 2;
  for (int c = 0; c < sq.items; ++c) {
    float* it = item(c);
    float* add = it + (warp < 4 ? 3 : 4) * kPart + c0;               // UV or O0
    const int r0 = (warp & 3) * 16 + rg;
    float base[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) base[q][e] = add[(size_t)(r0 + 4 * q) * D + cg + 8 * e];
    const float* gl = g_last + ((size_t)(sq.item0 + c) * H + h) * D + k0;
    const float4 ga = *reinterpret_cast<const float4*>(gl), gb = *reinterpret_cast<const float4*>(gl + 4);
    asm volatile("cp.async.wait_group 1;" ::: "memory");             // W and Q' of this chunk; Kd may be under way
    __syncthreads();
    fetch_wq(c + 1);                                                 // into the buffer of the chunk before
    {
      float2 acc[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[q][e] = make_float2(0.f, 0.f);
      const float* wr = wq2 + (c & 1) * 128 * kPad + (warp * 16 + rg) * kPad;
      const float* sr = st + cg * kPad;
#pragma unroll 4
      for (int k = 0; k < D; k += 4) {
        float4 s[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = *reinterpret_cast<const float4*>(sr + 8 * e * kPad + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 w = *reinterpret_cast<const float4*>(wr + 4 * q * kPad + k);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc[q][e] = __ffma2_rn(make_float2(w.x, w.y), make_float2(s[e].x, s[e].y), acc[q][e]);
            acc[q][e] = __ffma2_rn(make_float2(w.z, w.w), make_float2(s[e].z, s[e].w), acc[q][e]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d = acc[q][e].x + acc[q][e].y;
          if (warp < 4) u2[(r0 + 4 * q) * kCols + cg + 8 * e] = twice(base[q][e] - d);
          else add[(size_t)(r0 + 4 * q) * D + cg + 8 * e] = base[q][e] + d;
        }
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                                 // U and Kd are there, the old S is read
    {
      float2 acc[4][2];
#pragma unroll
      for (int m = 0; m < 4; ++m) acc[m][0] = acc[m][1] = make_float2(0.f, 0.f);
#pragma unroll 8
      for (int i = 0; i < kChunk; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(kd + i * 128 + k0), b = *reinterpret_cast<const float4*>(kd + i * 128 + k0 + 4);
        const float4 u = *reinterpret_cast<const float4*>(u2 + i * kCols + e0);
        const float2 ua = make_float2(u.x, u.y), ub = make_float2(u.z, u.w);
        acc[0][0] = __ffma2_rn(make_float2(a.x, a.y), ua, acc[0][0]); acc[0][1] = __ffma2_rn(make_float2(a.x, a.y), ub, acc[0][1]);
        acc[1][0] = __ffma2_rn(make_float2(a.z, a.w), ua, acc[1][0]); acc[1][1] = __ffma2_rn(make_float2(a.z, a.w), ub, acc[1][1]);
        acc[2][0] = __ffma2_rn(make_float2(b.x, b.y), ua, acc[2][0]); acc[2][1] = __ffma2_rn(make_float2(b.x, b.y), ub, acc[2][1]);
        acc[3][0] = __ffma2_rn(make_float2(b.z, b.w), ua, acc[3][0]); acc[3][1] = __ffma2_rn(make_float2(b.z, b.w), ub, acc[3][1]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float* s = st + (e0 + e) * kPad + k0;
        float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
        *reinterpret_cast<float4*>(s) = make_float4(fmaf(ga.x, a.x, acc[0][e].x), fmaf(ga.y, a.y, acc[0][e].y), fmaf(ga.z, a.z, acc[1][e].x),
                                                    fmaf(ga.w, a.w, acc[1][e].y));
        *reinterpret_cast<float4*>(s + 4) = make_float4(fmaf(gb.x, b.x, acc[2][e].x), fmaf(gb.y, b.y, acc[2][e].y),
                                                        fmaf(gb.z, b.z, acc[3][e].x), fmaf(gb.w, b.w, acc[3][e].y));
      }
    }
    __syncthreads();                                                 // the new S is there, Kd is read
    fetch_kd(c + 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int i = tid; i < D * kCols; i += 256) Sg[(size_t)(i / kCols) * D + i % kCols] = st[(i % kCols) * kPad + i / kCols];
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
    const float4 o = *reinterpret_cast<const float4*>(res + ((size_t)blockIdx.x * H + h) * kItemFloats + 4 * kPart + t * D + lane * 4);
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

}  // namespace kda
}  // namespace bg

extern "C" {

// See bg::kda::Params for the layouts.  D = 64 or 128; nseq sequences, H heads (this rank's).  Sequences of at most `longest_short` tokens go
// token by token (0: none do); items [n_items, 4] and seqs [n_seqs, 4] (ChunkItem, ChunkSeq) list chunks of up to 64 tokens and the
// pieces they make, with scratch of n_items * H * (5 * 64 + 1) * 128 floats.
int bg_kda_forward(const void* qkv, int qkv_stride, const void* f, int f_stride, const void* beta, int beta_stride,
                   const void* z, int z_stride, const float* conv_w, const float* conv_b, const float* A_log,
                   const float* dt_bias, const float* norm_w, float* conv_state, float* rec_state,
                   const int* cu_seqlens, const int* slots, const int* has_initial, void* out, int nseq, int H, int D,
                   float scale, float eps, const int* items, int n_items, const int* seqs, int n_seqs, int longest_short,
                   float* scratch, cudaStream_t stream) {
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
  if (n_items > 0) {
    static bg::DeviceOnce once_p, once_c;
    if (!bg::ensure_dynamic_smem(chunk_prepare, kPrepareFloats * 4, once_p) || !bg::ensure_dynamic_smem(chunk_chain, kChainFloats * 4, once_c))
      return -3;
    auto it = reinterpret_cast<const ChunkItem*>(items);
    float* g_last = scratch + (size_t)n_items * H * kItemFloats;
    chunk_prepare<<<dim3(n_items, H), kPrepThreads, kPrepareFloats * 4, stream>>>(p, it, scratch, g_last);
    chunk_chain<<<dim3(128 / kCols, H, n_seqs), 256, kChainFloats * 4, stream>>>(p, it, reinterpret_cast<const ChunkSeq*>(seqs), scratch, g_last);
    chunk_finish<<<dim3(n_items, H), 256, 0, stream>>>(p, it, scratch);
  }
  if (longest_short <= 0) return cudaGetLastError() == cudaSuccess ? 0 : -2;
  dim3 grid(H, nseq);
  if (D == 128) kda_seq_kernel<128><<<grid, 256, 0, stream>>>(p);
  else kda_seq_kernel<64><<<grid, 128, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
