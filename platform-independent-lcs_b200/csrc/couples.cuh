// couples.cuh -- host-side interface of the couple kernels (couples.cu).
#pragma once

#include "comb.cuh"

namespace slcs {

// Pairs with strand ids (m + n of a pair) up to this comb two to a register.
constexpr int PACKED16_MAX_IDS = 32767;
// Rows per lane and (with a configuration naming them) lanes per couple.
bool packed16_supported(int tm, int seg);
constexpr int COUPLE_TM = 16;

// Two pairs combed together (one per register half), on rows / TM lanes.
struct CoupleDev {
    PairDev a, b;     // b.m = b.n = 0: a is alone
    int32_t nb, rows; // blocks of 4 columns, rows
    // Staged couples: at stage[off] (uint4, off >= COUPLE_HEAD) lie `rows` row
    // symbols, as many h strands, 4 * nb column symbols, as many v strands.
    int32_t off;
    int32_t reserved;
};
constexpr int COUPLE_HEAD = 2; // uint4: symbols and strands of a block of masked columns
// Blocks of columns that the couples of a bundle may have together to be
// combed in shared memory; longer ones are staged in global memory.
constexpr int BUNDLE_BLOCKS = 512;

// What a lane of a bundle combs: lane `sl` of couple `couple` (-1: nothing),
// whose columns start at block `base` of the bundle, and the steps of the
// whole bundle.
struct BundleLane {
    int32_t couple;
    int16_t sl, lanes;
    int32_t base, steps;
};

struct CouplesLaunch {
    const uint8_t *a_blob;
    const uint8_t *b_blob;
    int32_t *out;               // strands as int32, or (out16 set)
    int16_t *out16;             // as int16 at the same offsets
    const CoupleDev *couples;   // device: the staged ones first
    int32_t nstaged;
    uint4 *stage;               // device: a masked block (COUPLE_HEAD), then the staged couples
    // Device, 32 lanes each: staged bundles (longest first), then the others,
    // list by list (longest first): list k, the work of one SM sub-partition, is
    // bundles list_off[k] .. list_off[k + 1) of those.
    const BundleLane *bundles;
    int32_t nstaged_bundles, nlists;
    const int32_t *list_off;    // device: nlists + 1
    int32_t *ticket;            // device: counter of the staged bundles, zero at launch
};

// Warps per SM sub-partition, at most.
constexpr int COUPLE_DEPTH = 3;
// Comb the bundles with `tm` rows per lane and `depth` warps per sub-partition
// (0: COUPLE_DEPTH); `alone`: on SMs that no other kernel's blocks share.
slcs_status launch_couples(const CouplesLaunch &L, int tm, int depth, bool alone, int sms, cudaStream_t stream);

} // namespace slcs
