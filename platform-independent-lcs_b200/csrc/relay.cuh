// relay.cuh -- host-side interface of the relay combing kernel (relay.cu).
#pragma once

#include "comb.cuh"

namespace slcs {

// One launch: items are groups of RelayShape::warps row stripes (32 * rows per
// lane rows each) of a pair.  Groups of a pair are consecutive items in ascending
// order, so the producer of a group was claimed first by a running block.
struct RelayLaunch {
    const PairDev *pairs;   // device; null = the one pair of `single`
    const int2 *items;      // device (pair, group); null = group k of `single`
    int32_t nitems;
    const uint8_t *a_blob;
    const uint8_t *b_blob;
    int32_t *out;           // h then v of every pair (offsets in PairDev)
    int32_t *v_single;      // v of `single` (its h goes to out)
    int2 *rows;             // hand-down rows: (strand, group + 1) per column, zero at launch
    const int64_t *row_off; // device, per pair; null = 0
    int32_t *counters;      // [0] ticket, [1] abort flag, zero at launch; null with one item
    uint32_t *status;
    uint64_t wait_ns;
    PairDev single;
    // Two pairs per register (ids of 15 bits): an item's pair is an entry of
    // duos, two pairs (the second -1 for none) that share its groups, rows and
    // columns (the larger of both); row_off per entry.  Otherwise null.
    const int2 *duos; // device
    bool two;         // duos is set (also with PREPARE_ONLY)
};

// Shape of the kernel: rows per lane, columns per step, warps that comb.
struct RelayShape {
    int tm, tw, warps;
};
inline int32_t relay_groups(int32_t m, const RelayShape &s)
{
    const int32_t rows = 32 * s.tm * s.warps;
    return (m + rows - 1) / rows;
}
// Entries of the hand-down row of a pair (0 with one group).
inline int64_t relay_row_elems(int32_t m, int32_t n, const RelayShape &s)
{
    return relay_groups(m, s) > 1 ? int64_t(n) : 0;
}
slcs_status launch_relay(const RelayLaunch &L, const RelayShape &s, int sms, cudaStream_t stream);

} // namespace slcs
