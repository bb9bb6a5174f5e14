// bf16 rows as two e4m3 parts with one power-of-two scale per 32 elements: the tokens' operand of the block-scaled 4-bit product.
//
// x = 2^s (p1 + 2^-5 p2) with 2^s such that the largest element of the 32 lies in [2^7, 2^8).  p1 takes the first four significant bits, p2 the
// rest: a bf16 number has eight, so the sum is exact down to 2^-14 of the largest element and off by at most 2^-22 of it below (from 2^-18 of it on
// down bits are missing for good, and 2^-22 of it may become zero).  An element that is not
// finite has the NaN of e4m3 as p1 and says what it was in p2 (0: NaN, else the sign of an infinity), for the product's epilogue.
#pragma once
#include "common.cuh"

namespace bg {
namespace mxp {

constexpr int kPartShift = 5;
constexpr uint32_t kNan = 0x7F, kOne = 0x38;      // e4m3

__host__ __device__ __forceinline__ int part_row(int row, int part) { return (row / 8 * 2 + part) * 8 + row % 8; }

struct Parts {
  uint8_t* p;        // [rows / 8 rounded up][2][8][K]: eight rows' first parts, then their second parts
  uint8_t* s;        // [K / 128 rounded up][rows][4] e8m0 of p1, one per 32 elements; p2's is five less
  int rows, K;
};

// N elements of a row, k .. k + N - 1 (k a multiple of N); 32 / N neighbouring lanes hold a block and come here together
template <int N>
struct Split {
  uint32_t p1[N / 4], p2[N / 4];
  uint32_t scale;
  __device__ __forceinline__ explicit Split(const __nv_bfloat162 (&x)[N / 2]) {
    constexpr int kLanes = 32 / N;
    float2 v[N / 2];
    float top = 0.f;
    uint32_t odd = 0;                              // elements that are not finite
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      v[i] = __bfloat1622float2(x[i]);
      const float a = fabsf(v[i].x), b = fabsf(v[i].y);
      if (!(a < __int_as_float(0x7F800000))) odd |= 1u << (2 * i);
      else top = fmaxf(top, a);
      if (!(b < __int_as_float(0x7F800000))) odd |= 2u << (2 * i);
      else top = fmaxf(top, b);
    }
    const uint32_t group = ((1u << kLanes) - 1) << (threadIdx.x & 31 & ~(kLanes - 1));
#pragma unroll
    for (int o = kLanes / 2; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(group, top, o));
    scale = static_cast<uint32_t>(max(static_cast<int>(__float_as_uint(top) >> 23) - 7, kPartShift));
    const float inv = __uint_as_float((254u - scale) << 23);
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      const float2 a = make_float2(v[2 * i].x * inv, v[2 * i].y * inv), b = make_float2(v[2 * i + 1].x * inv, v[2 * i + 1].y * inv);
      const uint32_t lo = to_e4m3x2(a.x, a.y), hi = to_e4m3x2(b.x, b.y);
      const __half2_raw hl = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(lo), __NV_E4M3);
      const __half2_raw hh = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(hi), __NV_E4M3);
      const float2 fl = __half22float2(*reinterpret_cast<const __half2*>(&hl)), fh = __half22float2(*reinterpret_cast<const __half2*>(&hh));
      constexpr float kUp = 1 << kPartShift;
      p1[i] = lo | hi << 16;
      p2[i] = to_e4m3x2((a.x - fl.x) * kUp, (a.y - fl.y) * kUp) | static_cast<uint32_t>(to_e4m3x2((b.x - fh.x) * kUp, (b.y - fh.y) * kUp)) << 16;
    }
    if (odd != 0) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (!(odd >> i & 1)) continue;
        const float f = i & 1 ? v[i / 2].y : v[i / 2].x;
        const uint32_t what = f != f ? 0u : f > 0.f ? kOne : kOne | 0x80u;
        p1[i / 4] = (p1[i / 4] & ~(0xFFu << 8 * (i % 4))) | kNan << 8 * (i % 4);
        p2[i / 4] = (p2[i / 4] & ~(0xFFu << 8 * (i % 4))) | what << 8 * (i % 4);
      }
    }
  }
  __device__ __forceinline__ void store(const Parts& t, int row, int k) const {
    uint8_t* a = t.p + (size_t)part_row(row, 0) * t.K + k;
    uint8_t* b = a + (size_t)8 * t.K;
    if (N == 16) {
      *reinterpret_cast<uint4*>(a) = make_uint4(p1[0], p1[1], p1[2 % (N / 4)], p1[3 % (N / 4)]);
      *reinterpret_cast<uint4*>(b) = make_uint4(p2[0], p2[1], p2[2 % (N / 4)], p2[3 % (N / 4)]);
    } else {
      *reinterpret_cast<uint2*>(a) = make_uint2(p1[0], p1[1]);
      *reinterpret_cast<uint2*>(b) = make_uint2(p2[0], p2[1]);
    }
    if (k % 32 == 0) t.s[((size_t)(k / 128) * t.rows + row) * 4 + k % 128 / 32] = static_cast<uint8_t>(scale);
  }
};

}  // namespace mxp
}  // namespace bg
