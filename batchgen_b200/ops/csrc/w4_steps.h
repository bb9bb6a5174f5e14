// Numbering of the 4-bit GEMM's weight operands in TMEM, shared by the roles of the kernel and by a host model of its barriers.
//
// Expansion group g takes the K steps g, g + 4, .. of every tile and owns one slot, which nobody else writes.  A use of the slot is
// numbered by the group's own steps, so the group and the MMA issuer are never more than one use apart and a phase parity tells them
// all they need.  (Slots that follow the running step change owners at a tile border wherever K / 64 is not a multiple of four; a
// group that skips its last step can then be two uses ahead of what was consumed, where the parity is the same again.)
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define BG_W4_HD __host__ __device__ __forceinline__
#else
#define BG_W4_HD inline
#endif

namespace bg {
namespace mx {

constexpr int kGroups = 4;                // expansion groups, one slot each

// K steps of a tile of KB steps that group g expands
BG_W4_HD uint32_t group_steps(int KB, int g) { return static_cast<uint32_t>(KB - g + kGroups - 1) / kGroups; }
// the group, and slot, of step kb
BG_W4_HD int step_group(int kb) { return kb % kGroups; }
// uses of that slot before step kb of a CTA's tile number `tile`: wait for full with parity (use & 1), for empty with the other one
BG_W4_HD uint32_t slot_use(int KB, uint32_t tile, int kb) { return tile * group_steps(KB, step_group(kb)) + kb / kGroups; }

}  // namespace mx
}  // namespace bg
