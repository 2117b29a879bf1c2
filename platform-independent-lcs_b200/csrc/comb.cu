// comb.cu -- seaweed combing on sm_100a.
//
// Replaces the reference's tiled SYCL solvers (src/lcs_tiled.hpp:10-251, the
// sub-group wavefront of src/lcs_common.hpp:131-173 and the register tile of
// src/lcs_common.hpp:59-92) and its host residual fixup
// (src/lcs_grid.hpp:451-493, src/lcs_residual_fixup.hpp:74-121).
//
// Layout of the work
//   * The grid of a pair has m rows (symbols of a) and n columns (symbols of b).
//     A v strand enters every column at the top (id m+j) and moves down; an h
//     strand enters every row at the left (id m-1-r for row r) and moves right.
//     Cell rule (src/lcs_residual_fixup.hpp:49-54): swap the two strands when
//     the symbols match or when h > v.
//   * One warp combs one row stripe of 32*TM rows: lane l keeps rows
//     [l*TM, l*TM+TM) of the stripe -- their symbols and h strands -- in
//     registers for the whole stripe.  Columns advance in blocks of TW (4, or
//     8 for short stripe chains); at step t lane l combs block t-l, so the
//     warp is a 32-deep systolic pipeline and the v strands of a block travel
//     lane to lane with __shfl_up_sync.  Between pipeline fill and drain the
//     steps run without bounds checks and load their column symbols one step
//     ahead.
//   * Lane 31's output is the bottom edge of the stripe.  For the last stripe it
//     is the final v; otherwise it is written to a per-pair scratch row in HBM
//     and a progress counter is released every 32 columns.  Lane 0 of the next
//     stripe (another warp, usually on another SM) acquires that counter and
//     streams the row back with 16-byte cp.async.cg copies, 4 blocks ahead.
//     The scratch row is reused in place: stripe s+1 overwrites block c only
//     after it has read block c.
//   * Warps take stripes from a global ticket counter.  Stripes of one pair
//     have consecutive tickets, so a stripe's producer was claimed earlier by
//     a running warp and every wait ends; each wait is additionally bounded by
//     %globaltimer and raises DEV_ERR_TIMEOUT instead of hanging.  When all
//     stripes fit at once, each SM runs one block of ceil(stripes / SMs)
//     warps, so that the stripes spread evenly over the SMs.
//   * Rows past m and columns past n are masked by data, not by branches:
//     a masked row has a symbol nothing matches and h = -1 (never swaps), a
//     masked column likewise and v = INT_MAX (never swaps), so edge tiles need
//     no host fixup.
#include <algorithm>
#include <climits>
#include <mutex>
#include <type_traits>

#include "cell.cuh"
#include "comb.cuh"
#include "occupancy.cuh"

namespace slcs {

namespace {

constexpr int TN = 4;      // columns per step of the stream kernels (one 16-byte v vector)
// Blocks lane 0 of a stripe prefetches ahead: 2 for stripes of at most 14
// rows per lane, 4 for 16 (on B200 the 4096 pair took 0.83 ms instead of
// 0.87 with 2, the 2^20 pair 300 instead of 302 ms; the 131072 pair's 16-row
// stripes took 12.0 instead of 11.3 ms).
__host__ __device__ constexpr int pref_of(int tm) { return tm >= 16 ? 4 : 2; }
constexpr int RING = 8;    // shared-memory ring slots per warp (> the prefetch)
constexpr int PUBLISH_COLS = 32; // columns between progress releases

struct StripeWait {
    const int32_t *prog;
    int32_t *abort_flag;
    uint32_t *status;
    uint64_t limit_ns;
    int32_t avail;
    uint64_t t0;
    bool dead;

    // Lane 0 only: wait until the producer has published block `blk`.
    __device__ __forceinline__ void until(int blk)
    {
        if (avail > blk || dead) return;
        for (;;) {
            avail = ld_acquire_gpu(prog);
            if (avail > blk) return;
            if (ld_relaxed_gpu(abort_flag)) {
                dead = true;
                return;
            }
            uint64_t now = globaltimer_ns();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > limit_ns) {
                dead = true;
                st_relaxed_gpu(abort_flag, 1);
                raise_status(status, DEV_ERR_TIMEOUT);
                return;
            }
            __nanosleep(128);
        }
    }
};

// One row stripe of one pair, combed by one warp.  TW columns form a block,
// the unit of a step, of a scratch-row transfer and of the shuffle hand-off;
// the ring holds RING blocks of TW strands per warp.  TW = 4 everywhere but
// in launches that pick_tw() gives 8 (short stripe chains of tall tiles).
template <int TM, int TW, bool WIDE>
struct Stripe {
    static constexpr int Q = TW / 4;                 // int4 per block
    static constexpr int PREF = pref_of(TM);
    static constexpr int PUBLISH = PUBLISH_COLS / TW; // blocks between releases

    const uint8_t *__restrict__ b;
    int32_t *vout;
    int32_t *scr;
    int4 *ring;
    int32_t *prog_mine;
    StripeWait W;
    int m, n, nb, lane;
    bool first, has_next;
    uint32_t av[TM];
    int hv[TM], vc[TW];

    // Column symbols of a whole block as one word (b aligned to its size).
    using Word = typename std::conditional<TW == 8, uint2, uint32_t>::type;
    Word bnext; // the word of the block this lane combs next (main loop)

    __device__ __forceinline__ Word word(int blk) const { return __ldg(reinterpret_cast<const Word *>(b + blk * TW)); }

    __device__ __forceinline__ static void unpack(uint32_t w, uint32_t *bs)
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) bs[j] = symbol_code(w, j);
    }
    __device__ __forceinline__ static void unpack(uint2 w, uint32_t *bs)
    {
        unpack(w.x, bs);
        unpack(w.y, bs + 4);
    }

    // Column symbols of block blk: masked past n or when the lane is idle.
    __device__ __forceinline__ void symbols(int blk, bool act, uint32_t (&bs)[TW]) const
    {
        const int c = blk * TW;
#pragma unroll
        for (int j = 0; j < TW; ++j) bs[j] = (act && c + j < n) ? symbol_code(__ldg(b + c + j), 0) : MASKED_COLUMN;
    }

    // Lane 0: the v strands entering block t at the top of the stripe.
    template <bool FULL>
    __device__ __forceinline__ void top(int t, int (&vi)[TW])
    {
        const int c = t * TW;
        if (!FULL && t >= nb) {
#pragma unroll
            for (int j = 0; j < TW; ++j) vi[j] = INT_MAX;
            return;
        }
        if (first) {
#pragma unroll
            for (int j = 0; j < TW; ++j) vi[j] = (FULL || c + j < n) ? m + c + j : INT_MAX;
            return;
        }
        const int nxt = t + PREF;
        if (nxt < nb) {
            W.until(nxt);
            if (!W.dead) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    cp_async_cg16(&ring[(nxt & (RING - 1)) * Q + q], scr + nxt * TW + 4 * q);
            }
        }
        cp_async_commit();
        cp_async_wait<PREF>();
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int4 x = ring[(t & (RING - 1)) * Q + q];
            vi[4 * q + 0] = x.x;
            vi[4 * q + 1] = x.y;
            vi[4 * q + 2] = x.z;
            vi[4 * q + 3] = x.w;
        }
        // Past n the producer's strands are INT_MAX already (masked columns
        // never swap), so a partial last block needs no mask here.
    }

    // Step t: lane l combs block t - l.  FULL: every lane's block is whole
    // and lies in [0, nb), and the symbols of b can be loaded as words.
    template <bool FULL>
    __device__ __forceinline__ void step(int t)
    {
        const int blk = t - lane;
        const bool act = FULL || unsigned(blk) < unsigned(nb);
        int vi[TW];
#pragma unroll
        for (int j = 0; j < TW; ++j) vi[j] = __shfl_up_sync(FULL_MASK, vc[j], 1);
        if (lane == 0) top<FULL>(t, vi);
        uint32_t bs[TW];
        if (FULL) {
            // The word was loaded one step ago; fetch the next one now, so
            // that the load's latency hides behind this step's cells.
            unpack(bnext, bs);
            bnext = word(blk + 1);
        } else {
            symbols(blk, act, bs);
        }
#pragma unroll
        for (int j = 0; j < TW; ++j) {
            int v = vi[j];
#pragma unroll
            for (int k = 0; k < TM; ++k) cell<WIDE>(av[k], bs[j], hv[k], v);
            vc[j] = v;
        }
        if (lane == 31 && act) {
            const int c = blk * TW;
            if (has_next) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    *reinterpret_cast<int4 *>(scr + c + 4 * q) =
                        make_int4(vc[4 * q], vc[4 * q + 1], vc[4 * q + 2], vc[4 * q + 3]);
                if ((blk & (PUBLISH - 1)) == PUBLISH - 1 || (!FULL && blk == nb - 1))
                    st_release_gpu(prog_mine, blk + 1);
            } else {
#pragma unroll
                for (int j = 0; j < TW; ++j)
                    if (FULL || c + j < n) vout[c + j] = vc[j];
            }
        }
    }
};

template <int TM, int TW = 4, bool WIDE = false>
__device__ __forceinline__ void comb_stripe(const CombLaunch &L, const PairDev &P, int64_t scr_off,
                                            int stripe, int task, int4 *ring, int lane)
{
    using StripeT = Stripe<TM, TW, WIDE>;
    StripeT S;
    const int m = P.m, n = P.n;
    const uint8_t *__restrict__ a = L.a_blob + P.a_off;
    int32_t *hout = L.out + P.out_off;
    S.b = L.b_blob + P.b_off;
    S.vout = hout + m;
    S.scr = L.scratch + scr_off;
    S.ring = ring;
    S.prog_mine = L.progress + task;
    S.W = StripeWait{L.progress + (task - 1), L.counters + 1, L.status, L.wait_ns, 0, 0, false};
    S.m = m;
    S.n = n;
    S.nb = (n + TW - 1) / TW;
    S.lane = lane;

    const int r0 = stripe * 32 * TM;
#pragma unroll
    for (int k = 0; k < TM; ++k) {
        const int r = r0 + lane * TM + k;
        const bool in = r < m;
        S.av[k] = in ? symbol_code(a[r], 0) : MASKED_ROW;
        S.hv[k] = in ? (m - 1 - r) : -1;
    }
    S.first = stripe == 0;
    S.has_next = r0 + 32 * TM < m;
    const int nb = S.nb;

    if (!S.first && lane == 0) {
#pragma unroll
        for (int d = 0; d < StripeT::PREF; ++d) {
            if (d < nb) {
                S.W.until(d);
                if (!S.W.dead) {
#pragma unroll
                    for (int q = 0; q < StripeT::Q; ++q)
                        cp_async_cg16(&ring[d * StripeT::Q + q], S.scr + d * TW + 4 * q);
                }
            }
            cp_async_commit();
        }
    }

#pragma unroll
    for (int j = 0; j < TW; ++j) S.vc[j] = INT_MAX;

    // Steps 0..30 fill the pipeline and the last 33 drain it (some lanes idle,
    // the last block may be partial); in between every lane combs a whole
    // block, and the block after it is whole too (its symbols are loaded one
    // step ahead), so those steps run without bounds checks.
    const bool b_aligned = (reinterpret_cast<uintptr_t>(S.b) & (TW - 1)) == 0;
    const int fill = nb + 31 < 31 ? nb + 31 : 31;
    const int full_end = (b_aligned && nb - 2 > 31) ? nb - 2 : fill;
    if (full_end > fill) S.bnext = S.word(fill - lane);
    int t = 0;
    for (; t < fill; ++t) S.template step<false>(t);
    for (; t < full_end; ++t) S.template step<true>(t);
    for (; t < nb + 31; ++t) S.template step<false>(t);
    if (!S.first && lane == 0) cp_async_wait<0>();

#pragma unroll
    for (int k = 0; k < TM; ++k) {
        const int r = r0 + lane * TM + k;
        if (r < m) hout[m - 1 - r] = S.hv[k];
    }
}

// Task k of the launch: its pair, stripe and scratch offset.
__device__ __forceinline__ void task_of(const CombLaunch &L, int k, PairDev &P, int &stripe, int64_t &so)
{
    if (L.tasks) {
        const int2 tk = L.tasks[k];
        P = L.pairs[tk.x];
        stripe = tk.y;
        so = L.scratch_off[tk.x];
    } else {
        P = L.single;
        stripe = k;
        so = 0;
    }
}

// WARPS is the largest block the kernel is launched with (the ring is sized
// for it); a launch may use fewer warps per block.  Warps take tasks from the
// ticket counter: a task's producer always holds a smaller ticket, so it was
// claimed by a warp that is already running, whatever the number of blocks
// the GPU holds at once.  (A static map, warp w of block b on task
// w * gridDim.x + b in a cooperative launch, spreads consecutive stripes over
// the SMs; it combed the 2^20 pair in 763 ms instead of 407 ms, because the
// four stripes sharing a sub-partition then start and finish far apart.)
template <int TM, int WARPS, int TW, bool WIDE = false>
__global__ void __launch_bounds__(WARPS * 32) comb_wavefront_kernel(const CombLaunch L)
{
    __shared__ __align__(16) int4 ring[WARPS][RING * TW / 4];
    const int lane = threadIdx.x & 31;
    const int w = __shfl_sync(FULL_MASK, int(threadIdx.x) >> 5, 0); // warp-uniform for the compiler
    PairDev P;
    int stripe;
    int64_t so;
    for (;;) {
        int k = 0;
        if (lane == 0) k = ld_relaxed_gpu(L.counters + 1) ? INT_MAX : atomicAdd(L.counters, 1);
        k = __shfl_sync(FULL_MASK, k, 0);
        if (k >= L.ntasks) break;
        task_of(L, k, P, stripe, so);
        comb_stripe<TM, TW, WIDE>(L, P, so, stripe, k, ring[w], lane);
    }
}

// ---------------------------------------------------------------------------
// Stream mode (pairs of at most SEG*TM rows).
//
// A segment of SEG lanes is a SEG-deep systolic pipeline like the wavefront
// warp, but its column stream is the concatenation of many pairs: lane l is
// always l blocks behind lane 0, and when a lane finishes the last block of
// one pair it writes its h strands and switches to the next pair.  The
// pipeline fills and drains once per segment instead of once per pair.
//
// Each segment owns a list of pairs fixed when the plan was made (longest
// processing time first over all resident segments), so every lane knows the
// pair after its current one and loads that pair's descriptor and row symbols
// one pair ahead: nothing on a switch waits for memory.
// ---------------------------------------------------------------------------
template <int TM>
struct StreamTask {
    int pair; // -1: no more work
    int m, n, nb;
    const uint8_t *b;
    int32_t *h_out;
    int32_t *v_out;
};

// The pair a lane combs next: descriptor words and its TM row symbols.
template <int TM>
struct NextPair {
    int pair;
    int4 d0, d1; // PairDev: a_off, b_off | out_off, m, n
    uint32_t sym[(TM + 3) / 4];
};

template <int TM>
__device__ __forceinline__ void fetch_next(const CombLaunch &L, int pair, int r0, NextPair<TM> &N)
{
    N.pair = pair;
    if (pair < 0) return;
    const int4 *pd = reinterpret_cast<const int4 *>(L.pairs + pair);
    N.d0 = __ldg(pd);
    N.d1 = __ldg(pd + 1);
    const int64_t a_off = int64_t((uint64_t(uint32_t(N.d0.y)) << 32) | uint32_t(N.d0.x));
    const int m = N.d1.z;
    const uint8_t *a = L.a_blob + a_off + r0;
    constexpr int WORDS = (TM + 3) / 4;
    if (r0 + 4 * WORDS <= m && (reinterpret_cast<uintptr_t>(a) & 3) == 0) {
#pragma unroll
        for (int q = 0; q < WORDS; ++q) N.sym[q] = __ldg(reinterpret_cast<const uint32_t *>(a) + q);
    } else {
#pragma unroll
        for (int q = 0; q < WORDS; ++q) {
            uint32_t w = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (r0 + 4 * q + k < m) w |= uint32_t(__ldg(a + 4 * q + k)) << (8 * k);
            N.sym[q] = w;
        }
    }
}

// Make the fetched pair current: rows r0.. get its symbols and start ids.
template <int TM>
__device__ __forceinline__ void take_next(const CombLaunch &L, const NextPair<TM> &N, int r0, StreamTask<TM> &T,
                                          uint32_t (&av)[TM], int (&hv)[TM])
{
    T.pair = N.pair;
    if (N.pair < 0) {
        T.m = T.n = T.nb = 0;
#pragma unroll
        for (int k = 0; k < TM; ++k) {
            av[k] = MASKED_ROW;
            hv[k] = -1;
        }
        return;
    }
    const int64_t b_off = int64_t((uint64_t(uint32_t(N.d0.w)) << 32) | uint32_t(N.d0.z));
    const int64_t o_off = int64_t((uint64_t(uint32_t(N.d1.y)) << 32) | uint32_t(N.d1.x));
    T.m = N.d1.z;
    T.n = N.d1.w;
    T.nb = (T.n + TN - 1) / TN;
    T.b = L.b_blob + b_off;
    T.h_out = L.out + o_off;
    T.v_out = T.h_out + T.m;
#pragma unroll
    for (int k = 0; k < TM; ++k) {
        const bool in = r0 + k < T.m;
        av[k] = in ? symbol_code(N.sym[k / 4], k % 4) : MASKED_ROW;
        hv[k] = in ? (T.m - 1 - r0 - k) : -1;
    }
}

// The pairs of one segment, in order: its list from the plan, then pairs of
// its class's pool, claimed one at a time.  Only lane 0 of a segment picks;
// lane l learns each pair from lane l - 1, which switched to it one step
// earlier (every lane of a segment sees the same column blocks, l steps
// behind lane 0).  Lane 0 claims its pool tickets one pick ahead, so that the
// atomic's round trip overlaps a whole pair instead of stalling the warp.
struct ItemSource {
    const int32_t *list; // the segment's list
    int count;           // pairs in it
    int q;               // lane 0: position of the next pair to pick
    int cls;
    int ahead;           // lane 0: pool ticket claimed for the next pick (-1: none yet)

    __device__ __forceinline__ int claim(const BatchLaunch &B, int size) const
    {
        return size > 0 ? atomicAdd(B.pool_ticket + cls, 1) : 0;
    }

    __device__ __forceinline__ int pick(const BatchLaunch &B) // -1: no more
    {
        const int off = B.pool_off[cls], size = B.pool_off[cls + 1] - off;
        if (q < count) {
            const int p = list[q];
            if (++q == count && ahead < 0) ahead = claim(B, size);
            return p;
        }
        const int k = ahead >= 0 ? ahead : claim(B, size);
        if (k >= size) {
            ahead = size;
            return -1;
        }
        ahead = claim(B, size);
        return B.pool_list[off + k];
    }
};

template <int TM, int SEG, int TNS>
__device__ __forceinline__ void stream_segment(const BatchLaunch &B, int cls, int seg_id, int lane)
{
    const CombLaunch &L = B.wf;
    const int sl = lane & (SEG - 1); // lane within the segment
    const int r0 = sl * TM;
    const int seg_lane0 = lane & ~(SEG - 1);
    const int beg = B.seg_off[seg_id];
    ItemSource src{B.seg_list + beg, B.seg_off[seg_id + 1] - beg, 0, cls, -1};

    // The first two items, picked by lane 0 and shared with the segment.
    int p0 = -1, p1 = -1;
    if (sl == 0) {
        p0 = src.pick(B);
        if (p0 >= 0) p1 = src.pick(B);
    }
    p0 = __shfl_sync(FULL_MASK, p0, seg_lane0);
    p1 = __shfl_sync(FULL_MASK, p1, seg_lane0);
    StreamTask<TM> T;
    NextPair<TM> N;
    uint32_t av[TM];
    int hv[TM];
    fetch_next<TM>(L, p0, r0, N);
    take_next<TM>(L, N, r0, T, av, hv);
    T.nb = (T.n + TNS - 1) / TNS;
    fetch_next<TM>(L, p1, r0, N);
    int nxt = p1; // the item after the current one (already fetched)
    int blk = -sl;

    int vc[TNS];
#pragma unroll
    for (int j = 0; j < TNS; ++j) vc[j] = INT_MAX;

    for (int it = 0;; ++it) {
        const bool live = T.pair >= 0;
        if ((it & 3) == 0 && !__any_sync(FULL_MASK, live)) break;
        const bool act = live && blk >= 0;
        const int c = blk * TNS;
        const int up = __shfl_up_sync(FULL_MASK, nxt, 1, SEG); // lane l - 1's next item

        int vi[TNS];
#pragma unroll
        for (int j = 0; j < TNS; ++j) vi[j] = __shfl_up_sync(FULL_MASK, vc[j], 1, SEG);
        if (sl == 0) {
#pragma unroll
            for (int j = 0; j < TNS; ++j) vi[j] = (act && c + j < T.n) ? T.m + c + j : INT_MAX;
        }

        uint32_t bs[TNS];
        // Whole-word loads only where b is aligned to TNS bytes (c is a multiple of TNS).
        if (act && c + TNS <= T.n && (reinterpret_cast<uintptr_t>(T.b) & (TNS - 1)) == 0) {
            if constexpr (TNS == 8) {
                const uint2 w = __ldg(reinterpret_cast<const uint2 *>(T.b + c));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    bs[j] = symbol_code(w.x, j);
                    bs[4 + j] = symbol_code(w.y, j);
                }
            } else {
                const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(T.b + c));
#pragma unroll
                for (int j = 0; j < TNS; ++j) bs[j] = symbol_code(w, j);
            }
        } else {
#pragma unroll
            for (int j = 0; j < TNS; ++j)
                bs[j] = (act && c + j < T.n) ? symbol_code(__ldg(T.b + c + j), 0) : MASKED_COLUMN;
        }

#pragma unroll
        for (int j = 0; j < TNS; ++j) {
            int v = vi[j];
#pragma unroll
            for (int k = 0; k < TM; ++k) cell<false>(av[k], bs[j], hv[k], v);
            vc[j] = v;
        }

        if (sl == SEG - 1 && act) {
#pragma unroll
            for (int j = 0; j < TNS; ++j)
                if (c + j < T.n) T.v_out[c + j] = vc[j];
        }

        if (live && ++blk == T.nb) {
            // This lane leaves pair q: write its h strands, move to pair q+1
            // (already fetched) and fetch pair q+2.
#pragma unroll
            for (int k = 0; k < TM; ++k)
                if (r0 + k < T.m) T.h_out[T.m - 1 - r0 - k] = hv[k];
            take_next<TM>(L, N, r0, T, av, hv);
            T.nb = (T.n + TNS - 1) / TNS;
            int p = -1;
            if (T.pair >= 0) p = sl == 0 ? src.pick(B) : up;
            nxt = p;
            fetch_next<TM>(L, p, r0, N);
            blk = 0;
        }
    }
}

// Stream classes compiled into the batch kernel: (rows per lane, lanes per segment).
#define SLCS_STREAM_CLASSES(X) X(4, 8) X(4, 16) X(4, 32) X(8, 8) X(8, 16) X(8, 32) \
    X(12, 8) X(12, 16) X(12, 32) X(16, 8) X(16, 16) X(16, 32)
// Four blocks of 4 warps per SM need at most 128 registers per thread.
template <int TNS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) comb_batch_kernel(const BatchLaunch B)
{
    const int lane = threadIdx.x & 31;
    const int w = __shfl_sync(FULL_MASK, int(threadIdx.x) >> 5, 0); // warp-uniform for the compiler
    const int gw = blockIdx.x * WARPS + w;
    if (gw >= B.nwarps) return;
    // This warp's stream segments (class and lists fixed by the plan).
    int cls = 0;
    while (cls < B.nclass - 1 && gw >= B.class_warp_end[cls]) ++cls;
#define SLCS_CASE(TM, SEG)                                                                 \
    case TM * 100 + SEG:                                                                   \
        stream_segment<TM, SEG, TNS>(B, cls, SEG_SLOTS * gw + lane / SEG, lane);           \
        break;
    switch (B.class_code[cls]) { SLCS_STREAM_CLASSES(SLCS_CASE) default: break; }
#undef SLCS_CASE
}

__global__ void strands_to_perm_kernel(const int32_t *__restrict__ h, int32_t m, const int32_t *__restrict__ v,
                                       int32_t n, int32_t *r2c, int32_t *c2r)
{
    const int32_t size = m + n;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
        const int32_t id = i < m ? h[i] : v[i - m];
        const int32_t col = i < m ? n + i : i - m;
        if (id >= 0 && id < size) {
            if (r2c) r2c[id] = col;
            if (c2r) c2r[col] = id;
        }
    }
}

// The same for every pair of a batch (grid dimension y), each at its
// out_off in both arrays: row -> col only.
__global__ void batch_to_perm_kernel(const PairDev *__restrict__ pairs, const int32_t *__restrict__ strands, int32_t *r2c)
{
    const PairDev d = pairs[blockIdx.y];
    const int32_t size = d.m + d.n;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
        const int32_t id = strands[d.out_off + i];
        if (id >= 0 && id < size) r2c[d.out_off + id] = i < d.m ? d.n + i : i - d.m;
    }
}

// Balanced launch: when every stripe can be resident at once, each SM gets
// one block of ceil(stripes / SMs) warps, so no SM hosts more stripes than
// another by more than one.  (With several blocks per SM, tickets went to
// whichever warps started first, and an SM holding 16 stripes instead of the
// average 13.8 set the pace of the whole wavefront.)  Dynamic shared memory of
// more than half an SM keeps a second block off every SM.
constexpr int WF_SM_WARPS = 16;

struct Balanced {
    bool ok = false;
    int smem = 0;
};

template <int TM, int TW, bool WIDE>
slcs_status balanced_setup(Balanced &B)
{
    int dev = 0, per_sm = 0, optin = 0;
    SLCS_CUDA(cudaGetDevice(&dev));
    SLCS_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    SLCS_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa{};
    SLCS_CUDA(cudaFuncGetAttributes(&fa, comb_wavefront_kernel<TM, WF_SM_WARPS, TW, WIDE>));
    const int want = per_sm / 2 + 1024 - int(fa.sharedSizeBytes);
    if (want <= 0 || want + int(fa.sharedSizeBytes) > optin) return SLCS_OK;
    SLCS_CUDA(cudaFuncSetAttribute(comb_wavefront_kernel<TM, WF_SM_WARPS, TW, WIDE>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, want));
    int occ = 0;
    SLCS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, comb_wavefront_kernel<TM, WF_SM_WARPS, TW, WIDE>,
                                                            WF_SM_WARPS * 32, size_t(want)));
    B.smem = want;
    B.ok = occ == 1;
    return SLCS_OK;
}

// Launches the balanced form when it applies; *done tells whether it did.
template <int TM, int TW, bool WIDE>
slcs_status launch_balanced(const CombLaunch &L, long sms, cudaStream_t stream, int *grid_out, bool *done)
{
    // Function attributes belong to a device: one set-up per device.
    static Balanced per_dev[MAX_DEVICES];
    static bool ready[MAX_DEVICES] = {};
    static std::mutex mu;
    *done = false;
    int dev = 0;
    SLCS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return SLCS_OK; // plain persistent launch
    Balanced &B = per_dev[dev];
    {
        std::lock_guard<std::mutex> g(mu);
        if (!ready[dev]) {
            const slcs_status s = balanced_setup<TM, TW, WIDE>(B);
            if (s != SLCS_OK) return s;
            ready[dev] = true;
        }
    }
    if (!B.ok || sms < 1) return SLCS_OK;
    const long per_sm = (long(L.ntasks) + sms - 1) / sms;
    if (per_sm > WF_SM_WARPS) return SLCS_OK;
    *done = true;
    if (stream == PREPARE_ONLY) return SLCS_OK;
    const long grid = std::min<long>(sms, L.ntasks);
    comb_wavefront_kernel<TM, WF_SM_WARPS, TW, WIDE><<<int(grid), int(per_sm) * 32, size_t(B.smem), stream>>>(L);
    if (grid_out) *grid_out = int(grid);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

// `sms` is the SM count of the current device (passed in by the caller, so
// that entry points that must not allocate never touch the lazily created
// per-device state behind sm_count()).
template <int TM, int WARPS, int TW, bool WIDE>
slcs_status launch_persistent(const CombLaunch &L, long sms, cudaStream_t stream, int *grid_out)
{
    if (sms < 1) sms = 1;
    int occ = 1;
    const slcs_status os = occupancy_of<comb_wavefront_kernel<TM, WARPS, TW, WIDE>>(WARPS * 32, &occ);
    if (os != SLCS_OK) return os;
    if (stream == PREPARE_ONLY) return SLCS_OK;
    // More stripes than fit at once: persistent blocks take stripes from the
    // ticket counter.  Beyond one block per SM the grid is rounded up to a
    // multiple of the SM count, so that every SM hosts the same number of
    // warps.
    long want = (long(L.ntasks) + WARPS - 1) / WARPS;
    if (want > sms) want = (want + sms - 1) / sms * sms;
    long grid = sms * occ;
    if (want < grid) grid = want;
    if (grid < 1) grid = 1;
    comb_wavefront_kernel<TM, WARPS, TW, WIDE><<<int(grid), WARPS * 32, 0, stream>>>(L);
    if (grid_out) *grid_out = int(grid);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

template <int TM, int WARPS, int TW, bool WIDE>
slcs_status launch_variant_tw(const CombLaunch &L, long sms, cudaStream_t stream, int *grid_out)
{
    bool done = false;
    const slcs_status bs = launch_balanced<TM, TW, WIDE>(L, sms, stream, grid_out, &done);
    if (bs != SLCS_OK || done) return bs;
    return launch_persistent<TM, WARPS, TW, WIDE>(L, sms, stream, grid_out);
}

template <int TM, int WARPS, bool WIDE>
slcs_status launch_variant(const CombLaunch &L, long sms, cudaStream_t stream, int *grid_out)
{
    if constexpr (TM == 14 || TM == 16) {
        if (L.tw == 8) return launch_variant_tw<TM, WARPS, 8, WIDE>(L, sms, stream, grid_out);
    }
    return launch_variant_tw<TM, WARPS, 4, WIDE>(L, sms, stream, grid_out);
}

template <int TNS, int WARPS>
slcs_status launch_batch_variant(const BatchLaunch &B, cudaStream_t stream, int *grid_out)
{
    int occ = 1;
    const slcs_status os = occupancy_of<comb_batch_kernel<TNS, WARPS>>(WARPS * 32, &occ);
    if (os != SLCS_OK) return os;
    if (stream == PREPARE_ONLY) {
        if (grid_out) *grid_out = sm_count() * occ;
        return SLCS_OK;
    }
    int grid = B.grid;
    if (grid < 1) grid = 1;
    comb_batch_kernel<TNS, WARPS><<<grid, WARPS * 32, 0, stream>>>(B);
    if (grid_out) *grid_out = grid;
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

} // namespace

// Dispatch on rows per lane, warps per block and the cell rule.
template <int TM>
static slcs_status launch_rows(const CombLaunch &L, int warps, long sms, cudaStream_t stream, int *grid_out)
{
    if (L.wide) {
        if (warps == 2) return launch_variant<TM, 2, true>(L, sms, stream, grid_out);
        if (warps == 8) return launch_variant<TM, 8, true>(L, sms, stream, grid_out);
        return launch_variant<TM, 4, true>(L, sms, stream, grid_out);
    }
    if (warps == 2) return launch_variant<TM, 2, false>(L, sms, stream, grid_out);
    if (warps == 8) return launch_variant<TM, 8, false>(L, sms, stream, grid_out);
    return launch_variant<TM, 4, false>(L, sms, stream, grid_out);
}

static slcs_status launch_comb_sms(const CombLaunch &L, int tile_m, int warps, long sms, cudaStream_t stream,
                                   int *grid_out)
{
    if (L.ntasks <= 0) return SLCS_OK;
    switch (tile_m) {
    case 2: return launch_rows<2>(L, warps, sms, stream, grid_out);
    case 4: return launch_rows<4>(L, warps, sms, stream, grid_out);
    case 8: return launch_rows<8>(L, warps, sms, stream, grid_out);
    case 12: return launch_rows<12>(L, warps, sms, stream, grid_out);
    case 14: return launch_rows<14>(L, warps, sms, stream, grid_out);
    case 16: return launch_rows<16>(L, warps, sms, stream, grid_out);
    default: return fail(SLCS_ERR_UNSUPPORTED, "tile_m must be one of 2, 4, 8, 12, 14, 16");
    }
}

slcs_status launch_comb_on(const CombLaunch &L, int tile_m, int warps, int sms, cudaStream_t stream)
{
    return launch_comb_sms(L, tile_m, warps, sms, stream, nullptr);
}

bool stream_variant_supported(int tm, int seg)
{
    return (tm == 4 || tm == 8 || tm == 12 || tm == 16) && (seg == 8 || seg == 16 || seg == 32);
}

slcs_status launch_batch(const BatchLaunch &B, int tns, cudaStream_t stream, int *grid_out)
{
    if (stream != PREPARE_ONLY && B.nwarps <= 0) return SLCS_OK;
    if (tns == 8) return launch_batch_variant<8, BATCH_WARPS>(B, stream, grid_out);
    if (tns == 4) return launch_batch_variant<4, BATCH_WARPS>(B, stream, grid_out);
    return fail(SLCS_ERR_UNSUPPORTED, "stream columns per step must be 4 or 8");
}

bool tile_m_supported(int tm) { return tm == 2 || tm == 4 || tm == 8 || tm == 12 || tm == 14 || tm == 16; }
int rows_per_stripe(int tm) { return 32 * tm; }

slcs_status launch_comb(const CombLaunch &L, int tile_m, int warps, cudaStream_t stream, int *grid_out)
{
    if (L.ntasks <= 0) return SLCS_OK;
    return launch_comb_sms(L, tile_m, warps, sm_count(), stream, grid_out);
}

slcs_status launch_strands_to_perm(const int32_t *h, int32_t m, const int32_t *v, int32_t n, int32_t *r2c,
                                   int32_t *c2r, cudaStream_t stream)
{
    const int64_t size = int64_t(m) + n;
    if (size <= 0) return SLCS_OK;
    if (r2c) SLCS_CUDA(cudaMemsetAsync(r2c, 0xff, size * sizeof(int32_t), stream));
    if (c2r) SLCS_CUDA(cudaMemsetAsync(c2r, 0xff, size * sizeof(int32_t), stream));
    int blocks = int((size + 255) / 256);
    if (blocks > sm_count() * 8) blocks = sm_count() * 8;
    strands_to_perm_kernel<<<blocks, 256, 0, stream>>>(h, m, v, n, r2c, c2r);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

slcs_status launch_batch_to_perm(const PairDev *pairs, int32_t npairs, int64_t total, const int32_t *strands,
                                 int32_t *r2c, cudaStream_t st)
{
    const int64_t each = std::max<int64_t>(1, total / npairs / 1024);
    constexpr int32_t MOST = 65535; // grid dimension y
    for (int32_t p0 = 0; p0 < npairs; p0 += MOST) {
        const int32_t np = std::min(MOST, npairs - p0);
        const dim3 grid(unsigned(std::min<int64_t>(each, std::max(1, 2368 / np))), unsigned(np));
        batch_to_perm_kernel<<<grid, 256, 0, st>>>(pairs + p0, strands, r2c);
    }
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

} // namespace slcs
