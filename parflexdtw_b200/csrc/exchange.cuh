// Entries through which a warp's lanes pass a pair to the next lane, once per step
// (stage1_dp.cuh, Rings): lane i stores into entry i in even steps and i + 1 in
// odd ones and, behind a barrier of the warp, loads lane i - 1's. In an odd step
// it stores into the entry that lane i + 2 loaded in the even step before, so a
// second barrier follows an even step's loads (a vote does not order memory); in
// an even step into the entry that it loaded itself. Measured, tiles of 2000 x
// 2000: 4.863 -> 4.868 ms of stage 1 with that barrier. (An entry that moves on
// with every step needs no second barrier, but 48 entries: 0.5 to 1 % slower.)
// Plain C++ but for the qualifiers: compiled on the host too.
#pragma once
#include "host_device.cuh"

namespace pfx {

constexpr int kXch = 34;  // (the last one spare: rings start on an even entry)
PFX_HD int exchange_store(int lane, int step) { return lane + (step & 1); }
// (lane 0 has no lane before it: its own, which is not used)
PFX_HD int exchange_load(int lane, int step) {
    return exchange_store(lane == 0 ? 0 : lane - 1, step);
}

}  // namespace pfx
