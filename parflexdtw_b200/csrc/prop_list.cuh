// Entries of the propagation's lists (stage2.cu, k_valid_lists): a slot of a tile
// anti-diagonal and the slot it reads, in 32 bits each. Slots are numbered
// with 64 bits (n1 n2 2 L of them: 2^31 and more fit the memory with short
// tiles), so an entry holds the slot's place among its diagonal's and the
// distance to its source, which lies in the tile above or to the left. Plain C++
// but for the qualifiers: compiled on the host too.
#pragma once
#include <stdint.h>

#include "host_device.cuh"

namespace pfx {

// First tile row of anti-diagonal a.
PFX_HD int32_t diag_row0(int32_t n2, int32_t a) { return a - (n2 - 1) > 0 ? a - (n2 - 1) : 0; }

// Slot k of a tile in row i of anti-diagonal a: its place in the diagonal
// (L2: slots of a tile, 2 L).
PFX_HD int32_t prop_place(int32_t n2, int32_t L2, int32_t a, int32_t i, int64_t k) {
    return (int32_t)((int64_t)(i - diag_row0(n2, a)) * L2 + k % L2);
}

// Tile row and slot of a place.
PFX_HD int64_t prop_slot(int32_t n2, int32_t L2, int32_t a, int32_t place, int32_t* i) {
    *i = diag_row0(n2, a) + place / L2;
    return ((int64_t)*i * n2 + (a - *i)) * L2 + place % L2;
}

// Distance (>= 1) from slot k back to the slot it reads; ~distance where it
// takes over that slot's value.
PFX_HD int32_t prop_back(int64_t k, int64_t src, bool copy) {
    return copy ? ~(int32_t)(k - src) : (int32_t)(k - src);
}
PFX_HD int64_t prop_src(int64_t k, int32_t back) { return k - (back < 0 ? ~back : back); }

// Whether every place and distance of a geometry has 31 bits (a slot's
// buffers take 61 bytes: one that does not needs 260 GB of them).
PFX_HD bool prop_list_fits(int64_t n1, int64_t n2, int64_t L) {
    const int64_t most = (int64_t)1 << 31;
    return (n1 < n2 ? n1 : n2) * 2 * L < most && (n1 == 1 || (n2 + 1) * 2 * L <= most);
}

}  // namespace pfx
