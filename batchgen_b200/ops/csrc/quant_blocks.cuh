// 1 x 128 e4m3 quantisation: the block itself, and the walk of kernels whose rows are many or partly absent.
#pragma once
#include "common.cuh"

namespace bg {

__device__ __forceinline__ float quant_scale(float amax, int pow2) {
  float s = fmaxf(amax, 1e-4f) * (1.0f / 448.0f);
  if (pow2) s = exp2f(ceilf(log2f(s)));
  return s;
}
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(p[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}
// eight of a block's 128 elements, sixteen neighbouring lanes (`lanes`) a block: writes their bytes and returns the block's scale
__device__ __forceinline__ float quant_block(const float (&f)[8], uint8_t* q, int pow2, uint32_t lanes) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(lanes, amax, o));
  const float s = quant_scale(amax, pow2), inv = 1.0f / s;
  __align__(8) uint16_t o4[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) o4[i] = to_e4m3x2(f[2 * i] * inv, f[2 * i + 1] * inv);
  *reinterpret_cast<uint2*>(q) = *reinterpret_cast<const uint2*>(o4);
  return s;
}

// Rows of K elements in groups of 2 U blocks, a group a warp (a half-warp a block): all U loads of a lane are on their way together, and a
// capacity above the rows that are present costs nothing.  A CTA a row kept one load in flight and cost its start for every padding row:
// expert rows of 2,048 for 4,739 tokens (8 of 256 experts, segments of 128) 94 us, now 65; 4 tokens 14, now 8.  Few blocks (a decode step) take U = 1, so
// that they spread over the SMs.
// The line between the two is where a lane of every resident warp of 148 SMs has a block, us with U = 1 and 4: tokens of 7,168 to eight expert rows, 4,736 blocks
// 8.2 / 10.3, 14,208 10.6 / 11.9, 18,944 12.4 / 12.2, 37,888 18.4 / 16.4, 150,000 51.4 / 47.1; rows alone 14,208 8.3 / 8.4, 18,944 9.0 / 8.4, 150,000 22.6 / 18.5.
constexpr int kSms = 148;
constexpr int kWalkBlocks = kSms * 8;
inline bool many_blocks(long long rows, int K) { return rows * (K / 128) >= kSms * 64ll * 2; }
inline int walk_grid(long long rows, int K, int U) {
  const long long warps = rows * ((K / 128 + 2 * U - 1) / (2 * U)), blocks = (warps + 7) / 8;
  return static_cast<int>(blocks < kWalkBlocks ? blocks : kWalkBlocks);
}
template <int U>
struct BlockWalk {
  int groups, rows, row, group, d_row, d_group;
  __device__ BlockWalk(int n, int K) : groups((K / 128 + 2 * U - 1) / (2 * U)), rows(n) {
    const int warp = blockIdx.x * 8 + (threadIdx.x >> 5), all = gridDim.x * 8;      // blocks of 256 threads
    row = warp / groups; group = warp - row * groups;
    d_row = all / groups; d_group = all - d_row * groups;
  }
  __device__ bool more() const { return row < rows; }
  __device__ void next() {
    row += d_row;
    group += d_group;
    if (group >= groups) { group -= groups; ++row; }
  }
  __device__ int block(int u, int lane) const { return (group * U + u) * 2 + (lane >> 4); }
};

}  // namespace bg
