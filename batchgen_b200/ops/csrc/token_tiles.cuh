// Tiles of the kernels that hold weights as the MMA's M side and tokens as N: segments of tokens (one per group, or one for a dense
// product) cut evenly into tiles of at most BT rows, rounded up to 16.
//
// Every role of a CTA walks the segments by itself, so a step over an empty or short segment has to be cheap: no division up to BT
// rows, and 16 segments at a time where none of their tiles is wanted.  One token in 4 of 128 segments, 4-bit products with cold weights: with two
// divisions a segment 74.8 us (6,144 x 2,880) and 62.7 (2,880 x 3,072), 34.7 and 21.3 here; 160 tokens 583 and 320, 547 and 286.
#pragma once
#include <stdint.h>

namespace bg {

struct TokenTile { int g, n0, m0, m_end; };          // weight rows n0 .., tokens m0 .. m_end (at most BT)

// tokens of a tile as the MMA's N
__device__ __forceinline__ int tile_cols(const TokenTile& t) { return (t.m_end - t.m0 + 15) / 16 * 16; }

template <int MAX_GROUPS>
struct Segments {                                    // in shared memory
  int offs[MAX_GROUPS + 1];
  int cnt[MAX_GROUPS];                               // rows present
  int part[(MAX_GROUPS + 15) / 16];                  // token tiles of 16 segments
};

template <int BT>
__device__ __forceinline__ int token_tiles(int rows) { return rows <= BT ? (rows > 0 ? 1 : 0) : (rows + BT - 1) / BT; }

// All threads of the block; the caller synchronises it afterwards.  counts: rows present in every segment, or null: all of it.
template <int BT, int MAX_GROUPS>
__device__ __forceinline__ void load_segments(Segments<MAX_GROUPS>& s, const int* offsets, const int* counts, int groups) {
  for (int i = threadIdx.x; i <= groups; i += blockDim.x) s.offs[i] = offsets[i];
  for (int i = threadIdx.x; i < groups; i += blockDim.x) {
    const int whole = offsets[i + 1] - offsets[i];
    s.cnt[i] = counts != nullptr ? min(max(counts[i], 0), whole) : whole;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (groups + 15) / 16; i += blockDim.x) {
    int sum = 0;
    for (int g = 16 * i; g < min(16 * i + 16, groups); ++g) sum += token_tiles<BT>(s.cnt[g]);
    s.part[i] = sum;
  }
}

// Tiles in the order (group, weight tile, token tile): token tiles of one weight tile are neighbours.
template <int BT, int BW, int MAX_GROUPS>
struct TokenWalker {
  const Segments<MAX_GROUPS>* seg;                   // null: one segment of M rows
  int groups, n_tiles, M, g, before;
  __device__ TokenWalker(const Segments<MAX_GROUPS>* s, int gr, int nt, int m) : seg(s), groups(gr), n_tiles(nt), M(m), g(0), before(0) {}
  // tile numbers of consecutive calls rise
  __device__ bool get(int tile, TokenTile& t) {
    while (g < groups) {
      if (seg != nullptr && (g & 15) == 0) {
        const int here = seg->part[g >> 4] * n_tiles;
        if (tile >= before + here) { before += here; g += 16; continue; }
      }
      const int rows = seg != nullptr ? seg->cnt[g] : M;
      const int tt = token_tiles<BT>(rows), here = tt * n_tiles;
      if (tile < before + here) {
        const int local = tile - before, base = seg != nullptr ? seg->offs[g] : 0;
        int per = rows, nt = local, mt = 0;
        if (tt > 1) {
          per = ((rows + tt - 1) / tt + 15) / 16 * 16;             // at most BT, and no tile is left empty
          nt = local / tt;
          mt = local % tt;
        }
        t.g = g; t.n0 = nt * BW; t.m0 = base + mt * per; t.m_end = min(t.m0 + per, base + rows);
        return true;
      }
      before += here;
      ++g;
    }
    return false;
  }
};

}  // namespace bg
