// relay.cu -- the relay kernel: a wavefront that keeps its chain short.
//
// Same work as the wavefront kernel of comb.cu (one warp per row stripe of
// 32 * TM rows, TM rows per lane in registers, strands passing lane to lane
// with shuffles), for combs that are one dependent chain rather than enough
// work for the GPU: a pair of n columns and T stripes takes about
// n / TW + 40 T steps one after another, so a step's latency is the time.
//   * A block is W combing warps and one I/O warp.  Warp w combs stripe
//     W * group + w.  All run in lockstep, K steps (an interval) between
//     barriers; warp w starts DI intervals after warp w - 1.  Strands pass
//     from a warp to the next through a ring in shared memory that the
//     barriers alone keep in order: no flags, no fences, no waits.
//   * A step is the same straight line for every lane: lane 0 takes its
//     strands from the ring (a broadcast read and a select), lane 31 stores
//     its own with a predicated store, and the symbols are a ring of ready
//     codes in which masked columns stand where there is no column, so that
//     filling, draining and ragged ends are no special case.  The next step's
//     reads and match tests, which depend on nothing, are issued in between.
//   * The I/O warp keeps global memory away from the others: per interval it
//     expands the symbols of b, brings the strands that enter the group at the
//     top, and writes out the ones that leave it at the bottom.
//   * Blocks hand down through one row of (strand, group) words per pair.  The
//     group number next to each strand says whose it is, so a reader needs no
//     flag and no fence, and the row is reused in place by every group.  That
//     holds only while a word is stored and loaded as one, so both sides use
//     8-byte relaxed accesses and nothing else (a wider or asynchronous copy
//     promises no such thing).  Entries are loaded ahead and polled only where
//     that was too early.  Every wait is bounded as in the wavefront kernel.
//   * Blocks take groups from a ticket counter; the group above a block's own
//     was therefore claimed by a running block.
//   * Batches whose ids fit 15 bits may put two pairs in a register (TWO, the
//     packed cell rule of cell.cuh): half the instructions for batches that
//     fill the SMs, which are bound by issue; a lone chain's step takes 1.2 to
//     1.8 times as long.  96 pairs of up to 2900 x 3300 309 -> 183 us, 400 of
//     2000 x 2000 538 -> 326, 30 of 9000 x 9000 1222 -> 540 (one B200).
// What it measured on one B200, against the wavefront kernel with the same
// cell rule: 4096 x 4096 728 -> 150 us ((TM, TW, W) = (4, 2, 3)), 20011 x 9973
// 3.41 -> 0.51 ms, 65536 x 65536 5.2 -> 2.6 ms ((8, 2, 3), against 2 x 2
// tiles), 131072 x 131072 9.8 -> 5.8 ms ((8, 4, 4) in two bands, against 4 x 4
// tiles).  The wavefront kernel published progress every 32 columns behind a
// fence and polled for it, about 940 cycles per step of 8 rows x 4 columns
// for a lone warp; a relay step of that shape takes 212, one of 4 x 2 76.
// With three combing warps the I/O warp has an SM sub-partition to itself;
// four (so that more rows fit the SMs) put it beside warp 0, which cost
// 4096 x 4096 182 us instead of 150.
#include <algorithm>
#include <climits>

#include "cell.cuh"
#include "occupancy.cuh"
#include "relay.cuh"

namespace slcs {

namespace {

constexpr int next_pow2(int x)
{
    int p = 1;
    while (p < x) p *= 2;
    return p;
}

// TW strands or codes of one block, TW = 2 or 4.
template <int TW>
__device__ __forceinline__ void load_block(const int32_t *p, int (&x)[TW])
{
    static_assert(TW == 2 || TW == 4, "a block is one vector");
    if constexpr (TW == 2) {
        const int2 v = *reinterpret_cast<const int2 *>(p);
        x[0] = v.x, x[1] = v.y;
    } else {
        const int4 v = *reinterpret_cast<const int4 *>(p);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    }
}

// Lane 31's store, as a predicated instruction (an if around the store made
// the warp diverge and reconverge in every step).
template <int TW>
__device__ __forceinline__ void store_block_if(bool on, int32_t *p, const int (&x)[TW])
{
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    if constexpr (TW == 2) {
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.v2.s32 [%1], {%2, %3};\n\t}"
                     ::"r"(int(on)), "r"(s), "r"(x[0]), "r"(x[1]) : "memory");
    } else {
        asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t"
                     "@q st.shared.v4.s32 [%1], {%2, %3, %4, %5};\n\t}"
                     ::"r"(int(on)), "r"(s), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory");
    }
}

__device__ __forceinline__ int2 ld_relaxed_pair(const int2 *p)
{
    unsigned long long x;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
    return make_int2(int(uint32_t(x)), int(uint32_t(x >> 32)));
}
__device__ __forceinline__ void st_relaxed_pair(int2 *p, int x, int y)
{
    const unsigned long long v = (static_cast<unsigned long long>(uint32_t(y)) << 32) | uint32_t(x);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The cell rule in two steps, for one pair or two.
template <bool TWO>
__device__ __forceinline__ int match(uint32_t a, int b)
{
    if constexpr (TWO) return int(match16(a, uint32_t(b)));
    else return match_far(a, uint32_t(b));
}
template <bool TWO>
__device__ __forceinline__ void swap_if(int far, int &h, int &v)
{
    if constexpr (TWO) {
        uint32_t x = uint32_t(h), y = uint32_t(v);
        pass16(uint32_t(far), x, y);
        h = int(x);
        v = int(y);
    } else {
        pass(far, h, v);
    }
}
template <bool TWO, int TM, int TW>
__device__ __forceinline__ void matches(const uint32_t (&a)[TM], const int (&b)[TW], int (&far)[TM][TW])
{
#pragma unroll
    for (int j = 0; j < TW; ++j)
#pragma unroll
        for (int q = 0; q < TM; ++q) far[q][j] = match<TWO>(a[q], b[j]);
}

// Columns c .. c + 3 of b (n columns, `aligned` to 4 bytes).
__device__ __forceinline__ uint32_t four_columns(const uint8_t *b, int c, int n, bool aligned)
{
    if (aligned && c + 4 <= n) return __ldg(reinterpret_cast<const uint32_t *>(b + c));
    uint32_t x = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (c + j < n) x |= uint32_t(__ldg(b + c + j)) << (8 * j);
    return x;
}

template <int TM, int TW, int W>
struct Relay {
    static constexpr int K = 8;                          // steps of an interval
    static constexpr int C = K * TW;                     // columns of an interval (at most 32)
    // Intervals a warp starts after the one above it: block t leaves lane 31
    // in interval (t + 31) / K and must be read in a later one, t / K + DI.
    static constexpr int DI = (30 + K) / K + 1;
    // How the I/O warp brings the row entries: LOADS words per lane for FETCH
    // intervals at once, issued when the entries before them are delivered or,
    // where intervals are shorter than an L2 round trip and a lane's word is
    // only one of them (DEEP), that many intervals earlier.  A load waits for
    // the one before it: with one per interval, two intervals ahead, 4096 x
    // 4096 took 176 us and 1003 x 250007 482, so 150 and 434 (the latter 472
    // without DEEP).
    static constexpr bool DEEP = C == 32 && TM * TW < 32;
    static constexpr int FETCH = DEEP ? 2 : 32 / C;
    static constexpr int LOADS = FETCH * C / 32;
    // Matches computed one step ahead, while their registers are few (a step
    // of (8, 4): 217 -> 196 cycles in a register probe, of (4, 2) 77 -> 72).
    static constexpr bool PIPE = TM * TW <= 32;
    static constexpr int RING = 4 * K;                   // blocks of a ring between two warps
    // Blocks of symbols between the one being delivered and the one lane 31
    // of the last warp still combs.
    static constexpr int BRING = next_pow2(2 * K + (W - 1) * DI * K + 32);
    struct Shared {
        int32_t strands[W + 1][RING][TW];
        int32_t codes[BRING][TW];
        int32_t item;
    };
};

// One barrier of the whole block, reached from both branches of the kernel.
template <int W>
__device__ __forceinline__ void sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"((W + 1) * 32) : "memory");
}

template <int TM, int TW, int W, bool TWO>
__global__ void __launch_bounds__((W + 1) * 32) relay_kernel(const RelayLaunch L)
{
    constexpr int NO_COLUMN = TWO ? int(MASKED_COLUMN16) : int(MASKED_COLUMN); // symbol of a masked column
    constexpr int NO_V = TWO ? int(MASKED_V16) : INT_MAX;                      // and its strand
    using R = Relay<TM, TW, W>;
    constexpr int K = R::K, C = R::C, DI = R::DI, RING = R::RING, BRING = R::BRING, FETCH = R::FETCH, LOADS = R::LOADS;
    __shared__ __align__(16) typename R::Shared S;
    const int lane = threadIdx.x & 31;
    const int w = __shfl_sync(FULL_MASK, int(threadIdx.x) >> 5, 0); // warp-uniform for the compiler

    for (int k = 0;; ++k) {
        if (L.counters) {
            __syncthreads(); // the item before this one is done with S
            if (threadIdx.x == 0) S.item = ld_relaxed_gpu(L.counters + 1) ? INT_MAX : atomicAdd(L.counters, 1);
            __syncthreads();
            k = S.item;
        }
        if (k >= L.nitems) break;
        const int2 it = L.items ? L.items[k] : make_int2(0, k);
        PairDev P, Q{};
        if constexpr (TWO) {
            const int2 d = L.duos[it.x];
            P = L.pairs[d.x];
            if (d.y >= 0) Q = L.pairs[d.y];
        } else {
            P = L.items ? L.pairs[it.x] : L.single;
        }
        const int m = TWO ? max(P.m, Q.m) : P.m, n = TWO ? max(P.n, Q.n) : P.n, group = it.y;
        const uint8_t *__restrict__ a = L.a_blob + P.a_off;
        const uint8_t *__restrict__ b = L.b_blob + P.b_off;
        const uint8_t *__restrict__ a2 = L.a_blob + Q.a_off; // the second pair's
        const uint8_t *__restrict__ b2 = L.b_blob + Q.b_off;
        int32_t *hout = L.out + P.out_off;
        int32_t *vout = L.items ? hout + P.m : L.v_single;
        int32_t *hout2 = L.out + Q.out_off, *vout2 = hout2 + Q.m;
        int2 *row = L.rows + (L.row_off ? L.row_off[it.x] : 0);
        const int r_group = group * (32 * TM * W);
        const int last = min(W, (m - r_group + 32 * TM - 1) / (32 * TM)) - 1; // the last warp with rows
        const bool bottom = r_group + 32 * TM * (last + 1) >= m;
        const int nb = (n + TW - 1) / TW;
        const int nw = (nb + 31 + K - 1) / K; // intervals a warp runs
        const int ni = nw + last * DI;

        uint32_t av[TM];
        int hv[TM], vc[TW];
        if (w < W) {
            const int r0 = r_group + (w * 32 + lane) * TM;
#pragma unroll
            for (int q = 0; q < TM; ++q) {
                const int r = r0 + q;
                if constexpr (TWO) {
                    av[q] = (r < P.m ? uint32_t(__ldg(a + r)) : MASKED_ROW16 & 0xFFFFu) |
                            (r < Q.m ? uint32_t(__ldg(a2 + r)) << 16 : MASKED_ROW16 & 0xFFFF0000u);
                    hv[q] = max(P.m - r, 0) | max(Q.m - r, 0) << 16;
                } else {
                    av[q] = r < m ? symbol_code(__ldg(a + r), 0) : MASKED_ROW;
                    hv[q] = r < m ? m - 1 - r : -1;
                }
            }
#pragma unroll
            for (int j = 0; j < TW; ++j) vc[j] = NO_V;
        }
        for (int x = threadIdx.x; x < BRING * TW; x += (W + 1) * 32) (&S.codes[0][0])[x] = NO_COLUMN;
        __syncthreads();

        if (w == W) {
            // The I/O warp: lane l moves column l of an interval.
            uint64_t t0 = 0;
            bool dead = false;
            // Symbols come a word of 4 per lane, 128 columns at a time.
            constexpr int SPAN = 128 / C;
            const bool aligned = (reinterpret_cast<uintptr_t>(b) & 3) == 0;
            const bool aligned2 = (reinterpret_cast<uintptr_t>(b2) & 3) == 0;
            uint32_t word = four_columns(b, 4 * lane, P.n, aligned);
            uint32_t word_next = four_columns(b, 128 + 4 * lane, P.n, aligned);
            uint32_t word2 = 0, word2_next = 0;
            if constexpr (TWO) {
                word2 = four_columns(b2, 4 * lane, Q.n, aligned2);
                word2_next = four_columns(b2, 128 + 4 * lane, Q.n, aligned2);
            }
            // Start the loads of the row entries of intervals i .. i + FETCH - 1.
            auto fetch = [&](int i, int2 (&e)[LOADS]) {
#pragma unroll
                for (int x = 0; x < LOADS; ++x) {
                    const int c = i * C + 32 * x + lane;
                    e[x] = make_int2(0, group);
                    if (group && c < n) e[x] = ld_relaxed_pair(row + c);
                }
            };
            // This lane's entry of the x-th of those intervals.
            auto entry = [&](const int2 (&e)[LOADS], int x) {
                if constexpr (C == 32) return e[x];
                else return make_int2(__shfl_sync(FULL_MASK, e[0].x, lane + C * x),
                                      __shfl_sync(FULL_MASK, e[0].y, lane + C * x));
            };
            // Another wait gave up, or this one has reached its limit.  Lane 0
            // decides for the warp: a lane that stopped alone would hand down
            // what it has not got, with no word to the host.
            auto give_up = [&]() {
                bool over = false;
                if (lane == 0) {
                    const uint64_t now = globaltimer_ns();
                    if (t0 == 0) t0 = now;
                    over = ld_relaxed_gpu(L.counters + 1) != 0;
                    if (!over && now - t0 > L.wait_ns) {
                        over = true;
                        st_relaxed_gpu(L.counters + 1, 1);
                        raise_status(L.status, DEV_ERR_TIMEOUT);
                    }
                }
                return __shfl_sync(FULL_MASK, int(over), 0) != 0;
            };
            auto deliver = [&](int i, int2 e) { // e: the lane's row entry as fetch found it
                const int c = i * C + lane;
                const bool in = lane < C && c < n;
                int v = in ? m + c : INT_MAX;
                if constexpr (TWO) // ids plus one
                    v = (c < P.n ? P.m + c + 1 : 0x7FFF) | (c < Q.n ? Q.m + c + 1 : 0x7FFF) << 16;
                if (group) {
                    if (!in) e.y = group;
                    for (int polls = 0; !dead && __any_sync(FULL_MASK, e.y != group); ++polls) {
                        if (e.y != group) e = ld_relaxed_pair(row + c);
                        if ((polls & 31) == 31) dead = give_up();
                    }
                    t0 = 0;
                    if (in) v = e.x;
                }
                const uint32_t x = __shfl_sync(FULL_MASK, word, (i % SPAN) * (C / 4) + lane / 4);
                uint32_t x2 = 0;
                if constexpr (TWO) x2 = __shfl_sync(FULL_MASK, word2, (i % SPAN) * (C / 4) + lane / 4);
                if (lane < C) {
                    const int blk = c / TW, j = c % TW;
                    S.strands[0][blk & (RING - 1)][j] = v;
                    const uint32_t sym = (x >> (8 * (lane & 3))) & 0xffu;
                    if constexpr (TWO) {
                        const uint32_t sym2 = (x2 >> (8 * (lane & 3))) & 0xffu;
                        S.codes[blk & (BRING - 1)][j] =
                            int((c < P.n ? sym : MASKED_COLUMN16 & 0xFFFFu) |
                                (c < Q.n ? sym2 << 16 : MASKED_COLUMN16 & 0xFFFF0000u));
                    } else {
                        S.codes[blk & (BRING - 1)][j] = int(in ? symbol_code(sym, 0) : MASKED_COLUMN);
                    }
                }
                if (i % SPAN == SPAN - 1) {
                    const int ahead = (i / SPAN + 2) * 128 + 4 * lane;
                    word = word_next;
                    word_next = four_columns(b, ahead, P.n, aligned);
                    if constexpr (TWO) {
                        word2 = word2_next;
                        word2_next = four_columns(b2, ahead, Q.n, aligned2);
                    }
                }
            };
            auto flush = [&](int i) { // the strands the last warp put out in interval i
                const int blk0 = (i - last * DI) * K - 31;
                const int c = blk0 * TW + lane;
                if (lane < C && c >= 0 && c < n) {
                    const int blk = c / TW, j = c % TW;
                    const int v = S.strands[last + 1][blk & (RING - 1)][j];
                    if (!bottom) {
                        st_relaxed_pair(row + c, v, group + 1);
                    } else if constexpr (TWO) {
                        if (c < P.n) vout[c] = (v & 0xFFFF) - 1;
                        if (c < Q.n) vout2[c] = int(uint32_t(v) >> 16) - 1;
                    } else {
                        vout[c] = v;
                    }
                }
            };
            int2 now[LOADS], ahead[LOADS];
            fetch(0, now);
            deliver(0, entry(now, 0));
            if constexpr (R::DEEP) fetch(FETCH, ahead);
            else if constexpr (FETCH == 1) fetch(1, now);
            sync<W>();
            for (int i0 = 0; i0 < ni; i0 += FETCH) {
#pragma unroll
                for (int x = 0; x < FETCH; ++x) {
                    const int i = i0 + x, next = (x + 1) % FETCH; // the entry to deliver
                    if (i >= ni) break;
                    if (i) flush(i - 1);
                    if (i + 1 < nw) {
                        if (R::DEEP && next == 0) {
#pragma unroll
                            for (int l = 0; l < LOADS; ++l) now[l] = ahead[l];
                        }
                        deliver(i + 1, entry(now, next));
                        if (R::DEEP && next == 0) fetch(i + 1 + FETCH, ahead);
                        if (!R::DEEP && next == FETCH - 1) fetch(i + 2, now);
                    }
                    sync<W>();
                }
            }
            flush(ni - 1);
        } else {
            // Intervals before this warp's first block, with its blocks, and
            // after its last one.
            const int idle = w <= last ? w * DI : ni;
            for (int i = 0; i <= idle; ++i) sync<W>();
            if (w <= last) {
                for (int il = 0; il < nw; ++il) {
                    const int base = il * K;
                    const int32_t *in = &S.strands[w][base & (RING - 1)][0];
                    int vin[TW], bc[TW];
                    load_block<TW>(in, vin);
                    load_block<TW>(&S.codes[(base - lane) & (BRING - 1)][0], bc);
                    if constexpr (R::PIPE) {
                        int far[TM][TW], next[TM][TW];
                        matches<TWO, TM, TW>(av, bc, far);
                        load_block<TW>(&S.codes[(base + 1 - lane) & (BRING - 1)][0], bc);
#pragma unroll
                        for (int s = 0; s < K; ++s) {
                            int vi[TW];
#pragma unroll
                            for (int j = 0; j < TW; ++j) {
                                vi[j] = __shfl_up_sync(FULL_MASK, vc[j], 1);
                                if (lane == 0) vi[j] = vin[j];
                            }
                            // The next step's strands, symbols and matches, which
                            // wait for nothing, fill the gaps of this step's chain.
                            if (s + 1 < K) {
                                load_block<TW>(in + (s + 1) * TW, vin);
                                matches<TWO, TM, TW>(av, bc, next);
                                if (s + 2 < K) load_block<TW>(&S.codes[(base + s + 2 - lane) & (BRING - 1)][0], bc);
                            }
#pragma unroll
                            for (int j = 0; j < TW; ++j) {
                                int v = vi[j];
#pragma unroll
                                for (int q = 0; q < TM; ++q) swap_if<TWO>(far[q][j], hv[q], v);
                                vc[j] = v;
                            }
#pragma unroll
                            for (int j = 0; j < TW; ++j)
#pragma unroll
                                for (int q = 0; q < TM; ++q) far[q][j] = next[q][j];
                            store_block_if<TW>(lane == 31, &S.strands[w + 1][(base + s - 31) & (RING - 1)][0], vc);
                        }
                    } else {
#pragma unroll 4 // all 8 overflow the instruction cache (16 rows: 708 cycles a step, 4: 388, 2: 425)
                        for (int s = 0; s < K; ++s) {
                            int vi[TW], bs[TW];
#pragma unroll
                            for (int j = 0; j < TW; ++j) {
                                vi[j] = __shfl_up_sync(FULL_MASK, vc[j], 1);
                                if (lane == 0) vi[j] = vin[j];
                                bs[j] = bc[j];
                            }
                            if (s + 1 < K) {
                                load_block<TW>(in + (s + 1) * TW, vin);
                                load_block<TW>(&S.codes[(base + s + 1 - lane) & (BRING - 1)][0], bc);
                            }
#pragma unroll
                            for (int j = 0; j < TW; ++j) {
                                int v = vi[j];
#pragma unroll
                                for (int q = 0; q < TM; ++q) swap_if<TWO>(match<TWO>(av[q], bs[j]), hv[q], v);
                                vc[j] = v;
                            }
                            store_block_if<TW>(lane == 31, &S.strands[w + 1][(base + s - 31) & (RING - 1)][0], vc);
                        }
                    }
                    sync<W>();
                }
                for (int il = nw; il < ni - idle; ++il) {
                    // Past its last block: masked columns for the warp below.
                    if (lane < C) S.strands[w + 1][(il * K - 31 + lane / TW) & (RING - 1)][lane % TW] = NO_V;
                    sync<W>();
                }
            }
            const int r0 = r_group + (w * 32 + lane) * TM;
#pragma unroll
            for (int q = 0; q < TM; ++q)
                if constexpr (TWO) {
                    if (r0 + q < P.m) hout[P.m - 1 - r0 - q] = (hv[q] & 0xFFFF) - 1;
                    if (r0 + q < Q.m) hout2[Q.m - 1 - r0 - q] = int(uint32_t(hv[q]) >> 16) - 1;
                } else {
                    if (r0 + q < m) hout[m - 1 - r0 - q] = hv[q];
                }
        }
        if (!L.counters) break;
    }
}

template <int TM, int TW, int W, bool TWO>
slcs_status launch_shape(const RelayLaunch &L, int sms, cudaStream_t stream)
{
    constexpr auto kernel = relay_kernel<TM, TW, W, TWO>;
    int occ = 1;
    const slcs_status os = occupancy_of<kernel>((W + 1) * 32, &occ);
    if (os != SLCS_OK || stream == PREPARE_ONLY) return os;
    const long grid = std::min<long>(L.nitems, long(std::max(1, sms)) * occ);
    kernel<<<int(grid), (W + 1) * 32, 0, stream>>>(L);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

} // namespace

#define SLCS_RELAY_SHAPES(X) \
    X(1, 4, 3) X(2, 4, 3) X(4, 2, 3) X(8, 2, 3) X(8, 4, 4) X(14, 4, 4) X(14, 4, 8) X(14, 4, 16)
#define SLCS_RELAY_DUO_SHAPES(X) X(2, 4, 3) X(4, 4, 3) X(8, 2, 3) X(8, 4, 4)

slcs_status launch_relay(const RelayLaunch &L, const RelayShape &s, int sms, cudaStream_t stream)
{
    if (L.nitems <= 0 && stream != PREPARE_ONLY) return SLCS_OK;
#define SLCS_CASE(TM, TW, W) \
    if (s.tm == TM && s.tw == TW && s.warps == W) return launch_shape<TM, TW, W, false>(L, sms, stream);
#define SLCS_CASE_TWO(TM, TW, W) \
    if (s.tm == TM && s.tw == TW && s.warps == W) return launch_shape<TM, TW, W, true>(L, sms, stream);
    if (L.two) {
        SLCS_RELAY_DUO_SHAPES(SLCS_CASE_TWO)
    } else {
        SLCS_RELAY_SHAPES(SLCS_CASE)
    }
#undef SLCS_CASE
#undef SLCS_CASE_TWO
    return fail(SLCS_ERR_UNSUPPORTED, "no such relay shape");
}

} // namespace slcs
