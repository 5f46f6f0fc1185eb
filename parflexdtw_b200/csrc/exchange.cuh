// Entries through which a warp's lanes pass a pair to the next lane, once per step
// of a block of kBlk steps (stage1_dp.cuh, Rings): in step t lane i stores into
// entry 31 - i + t and, behind a barrier of the warp, loads lane i - 1's. The
// entry it stores into is the one it loaded itself in the step before, so that
// barrier is all that orders the lanes within a block; a block starts behind
// one. (Two entries per lane in turn, with no barrier between a load and the
// store that follows it, would rely on a warp's accesses going in order.) Plain
// C++ but for the qualifiers: compiled on the host too.
#pragma once
#include "host_device.cuh"

namespace pfx {

constexpr int kXchSteps = 16;
constexpr int kXch = 32 + kXchSteps;
PFX_HD int exchange_store(int lane, int t) { return 31 - lane + t; }
// (lane 0 has no lane before it: its own)
PFX_HD int exchange_load(int lane, int t) { return exchange_store(lane == 0 ? 0 : lane - 1, t); }

}  // namespace pfx
