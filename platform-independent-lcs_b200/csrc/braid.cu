// braid.cu -- steady-ant braid multiplication on sm_100a.
//
// Replaces staggered_multiply<RowGlue> / steady_ant_seq / ant_passage of the
// reference (src/braid_multiplication.hpp:5-407).  The product of two seaweed
// permutations is computed by the same recursion (halve the shared dimension,
// multiply the halves, glue them with one ant walk), restructured for the GPU:
//
//   * The recursion runs breadth first.  Level l holds every node of that
//     depth side by side in one array of k entries (a node of size s starting
//     at o owns [o, o+s); its children are [o, o+s/2) and [o+s/2, o+s)), so
//     the node containing entry i at level l follows from i alone (node_of).
//   * Downward, each level is a stable partition of every node: P's rows by
//     column < s/2 (get_vert_slice, 5-19) and Q's columns by row < s/2
//     (get_horz_slice, 22-36); the maps from child index to parent index are
//     kept per level.  An entry's place at every level follows from its value
//     and counts, so products of up to 256 nodes write all levels in one pass
//     (fan_kernel).  Larger ones go level by level in one launch: single-pass
//     tiles (they publish their counts and look back over their predecessors)
//     take tickets level by level, and a tile first waits for the tiles of the
//     level above that hold its parent nodes; every wait is bounded.
//   * A node at or below the cutoff is finished by one thread block without
//     further recursion: it passes the crossings of P's part into Q's, S / 2
//     at a time, in S rounds of one packed compare-and-exchange (node_kernel).
//   * Upward, a level scatters both children's products into the parent's
//     rows and columns (inverse_mapping, 191-202) and, in the same pass, into
//     the parent's result (the union of the two halves, 254-268) and into the
//     block counts of the level's delta tables; then it walks the ant
//     (123-189) over every node, which writes the fresh points on top.
//   * A node's walk is cut into segments that run concurrently: on every
//     diagonal e = col - row the walk sits one row above r*(e-1), the first
//     point of diagonal e-1 where the dominance difference (hi points above-left
//     minus lo points below-right) is non-negative, so a segment can start
//     anywhere once r* is known there.  One warp takes a segment: short ones
//     row by row, every row independent of the others (walk_rows), long ones
//     run by run from staged words (ant_walk_warp).  Many short segments take
//     one lane each (walk_lanes_kernel).
//   * Products of one overlap run side by side in the same launches.
#include <climits>
#include <cmath>
#include <vector>

#include "braid.cuh"

namespace slcs {
namespace {

// Entries per block of the slices: two a thread, since a block's time is its
// chain of dependent reads (2048: products 1003 61 -> 54 us, 32768 198 -> 188;
// 256: 1000 x 1000000 pairs 866 -> 936 us, each block then adds more counts).
constexpr int SCAN_BS = 512;
constexpr int PART_PER = 8;     // entries per thread of a partition tile
// Threads of a partition tile: 1024 (8192 entries, one tile per SM at a time,
// a short look-back chain) for large products, 256 (2048 entries) below.
constexpr int PART_BIG_K = 1 << 19;
__host__ __device__ constexpr int part_threads(int k) { return k >= PART_BIG_K ? 1024 : 256; }

// One launch of a kernel works on up to N products side by side (product z of
// grid dimension z): the arguments of each.
template <typename Args, int N>
struct Many {
    static_assert(N * sizeof(Args) <= 4000, "kernel arguments are limited to 4 KB");
    Args of[N];
};

__host__ __device__ __forceinline__ void node_of(int i, int level, int k, int &o, int &s)
{
    o = 0;
    s = k;
    for (int d = 0; d < level; ++d) {
        const int h = s >> 1;
        if (i < o + h) {
            s = h;
        } else {
            o += h;
            s -= h;
        }
    }
}

// Node of level lc, left to right, that holds value v (or place v).
__device__ __forceinline__ int leaf_of(int v, int lc, int k)
{
    int o = 0, s = k, nd = 0;
    for (int d = 0; d < lc; ++d) {
        const int h = s >> 1;
        const bool right = v >= o + h;
        nd = nd * 2 + right;
        o += right ? h : 0;
        s = right ? s - h : h;
    }
    return nd;
}

// Products whose level lc has at most FAN_LEAVES nodes partition every level
// in one pass (fan_kernel), in tiles of FAN_TILE entries.
constexpr int FAN_LEAVES = 256;
constexpr int FAN_TILE = 1024;
__host__ __device__ constexpr int fan_tiles(int k) { return (k + FAN_TILE - 1) / FAN_TILE; }
// Up to this many slice blocks add their predecessors' counts themselves.
constexpr int SLICE_DIRECT = 4096;

// ---------------------------------------------------------------------------
// device-wide exclusive scan of two flag sets (partition of P rows and Q cols)
// ---------------------------------------------------------------------------
struct LevelArgs {
    const int32_t *P;  // r2c, node-local
    const int32_t *Q;  // c2r, node-local
    int32_t *Pn, *Qn;  // next level
    int32_t *pmap, *qmap; // next level: child index -> parent-local index
    int32_t *scanP, *scanQ;
    int k, level;
    const int32_t *bad;
};



// Exclusive scan of the block sums (one block; the count is k / SCAN_BS).
struct BsumArgs {
    int32_t *bp, *bq;
};
template <int N>
__global__ void __launch_bounds__(1024) part_bsum_kernel(const __grid_constant__ Many<BsumArgs, N> M, int nb)
{
    int32_t *bp = M.of[blockIdx.z].bp, *bq = M.of[blockIdx.z].bq;
    __shared__ int wp[32], wq[32];
    __shared__ int carry_p, carry_q;
    if (threadIdx.x == 0) carry_p = carry_q = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        int vp = i < nb ? bp[i] : 0, vq = i < nb ? bq[i] : 0;
        int xp = vp, xq = vq;
        for (int off = 1; off < 32; off <<= 1) {
            int yp = __shfl_up_sync(FULL_MASK, xp, off), yq = __shfl_up_sync(FULL_MASK, xq, off);
            if ((threadIdx.x & 31) >= off) {
                xp += yp;
                xq += yq;
            }
        }
        if ((threadIdx.x & 31) == 31) {
            wp[threadIdx.x >> 5] = xp;
            wq[threadIdx.x >> 5] = xq;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            int sp = wp[threadIdx.x], sq = wq[threadIdx.x];
            for (int off = 1; off < 32; off <<= 1) {
                int yp = __shfl_up_sync(FULL_MASK, sp, off), yq = __shfl_up_sync(FULL_MASK, sq, off);
                if (threadIdx.x >= off) {
                    sp += yp;
                    sq += yq;
                }
            }
            wp[threadIdx.x] = sp;
            wq[threadIdx.x] = sq;
        }
        __syncthreads();
        const int w = threadIdx.x >> 5;
        const int ep = carry_p + (w ? wp[w - 1] : 0) + xp - vp;
        const int eq = carry_q + (w ? wq[w - 1] : 0) + xq - vq;
        __syncthreads();
        if (i < nb) {
            bp[i] = ep;
            bq[i] = eq;
        }
        if (threadIdx.x == 1023) {
            carry_p = ep + vp;
            carry_q = eq + vq;
        }
        __syncthreads();
    }
}



// ---------------------------------------------------------------------------
// one level's partition in a single pass (count, scan and scatter fused)
//
// Tiles of THREADS * PART_PER entries take tickets in launch order, so that a tile's
// predecessors have all started.  A tile counts its flags, publishes the two
// counts at once (AGG; tile 0 its inclusive prefix, INCL), then one warp
// looks back over its predecessors 32 at a time -- adding AGG counts until
// it meets a tile that published INCL -- and publishes its own INCL.  It then writes its exclusive
// scan values and raises its `done` flag after them.  The scatter of an
// entry needs the scan value at its node's first entry; when that entry lies
// in an earlier tile, the tile waits for that tile's `done` (INCL alone is
// published before the scan values are written).  A tile waits only on
// words its predecessors publish without waiting themselves, or on `done`,
// which follows a look-back over such words, so every wait ends; each is
// also bounded by %globaltimer, and one that runs out raises the product's
// error flag (every later kernel returns early) and DEV_ERR_TIMEOUT.
// ---------------------------------------------------------------------------
constexpr unsigned long long TILE_AGG = 1ull << 62, TILE_INCL = 2ull << 62;
constexpr unsigned long long TILE_COUNT_MASK = (1ull << 31) - 1;
constexpr uint64_t PART_WAIT_NS = 2000000000ull;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long pack_counts(unsigned long long flag, int cp, int cq)
{
    return flag | (unsigned long long)(unsigned(cp)) | ((unsigned long long)(unsigned(cq)) << 31);
}

struct FusedArgs {
    LevelArgs L;
    unsigned long long *tiles; // status word per tile of this level, zero at launch
    int32_t *done;             // per tile of this level: scan values written (1), zero at launch
    int32_t *err;              // the product's error flag
    uint32_t *status;          // device status word
};

// Every level above the cutoff in one launch: tickets run level by level
// (ticket t is tile t % kb of level t / kb), and a tile of level l first
// waits until all kb tiles of level l - 1 have scattered (level_done), so
// that it reads finished arrays.  Every wait targets smaller tickets, which
// running blocks hold, so each ends; each is also bounded by %globaltimer.
struct PartAllArgs {
    int32_t *PQ;               // four k-arrays: P and Q of even levels, then of odd levels
    int32_t *maps;             // level l + 1's pmap at maps + 2k(l + 1), its qmap k further
    int32_t *scanP, *scanQ;
    int k, levels, kb;         // levels above the cutoff, tiles per level
    bool pow2;                 // k is a power of two: node boundaries are multiples of the node size
    unsigned long long *tiles; // levels * kb tile status words, zero at launch
    int32_t *done;             // levels * kb scan-written flags, zero at launch
    int32_t *ticket;           // zero at launch
    int32_t *level_done;       // per level: tiles scattered, zero at launch
    int32_t *scat;             // levels * kb: the tile has scattered (1), zero at launch
    int32_t *err;
    uint32_t *status;
};

// Thread 0: spin until done[t] is set, bounded; false on expiry.
__device__ __forceinline__ bool wait_done(const FusedArgs &F, int t)
{
    uint64_t t0 = 0;
    for (;;) {
        if (ld_acquire_gpu(F.done + t)) return true;
        if (ld_relaxed_gpu(F.err)) return false;
        const uint64_t now = globaltimer_ns();
        if (t0 == 0) {
            t0 = now;
        } else if (now - t0 > PART_WAIT_NS) {
            atomicExch(F.err, 1);
            raise_status(F.status, DEV_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(64);
    }
}

template <int PART_THREADS>
struct PartSmem {
    static constexpr int GROUPS = PART_PER * PART_THREADS / 32; // runs of 32 entries per tile
    int s_ok;
    int gp[GROUPS], gq[GROUPS]; // group counts, then their exclusive prefixes in the tile
    int s_ep, s_eq;             // exclusive prefix of the tile
};

// One tile of one level: count, look back, scan, scatter.  False when the
// product failed (err raised here or elsewhere); the block then stops.
template <int PART_THREADS>
__device__ __forceinline__ bool part_tile(const FusedArgs &F, int tile, bool local, PartSmem<PART_THREADS> &S)
{
    const LevelArgs &A = F.L;
    constexpr int PER = PART_PER;
    constexpr int PART_BS = PART_THREADS * PART_PER;
    constexpr int WARPS = PART_THREADS / 32;
    constexpr int GROUPS = PER * WARPS;         // runs of 32 entries per tile
    constexpr int GPL = GROUPS / 32;            // groups per lane of the scanning warp
    int &s_ok = S.s_ok;
    int *gp = S.gp, *gq = S.gq;
    int &s_ep = S.s_ep, &s_eq = S.s_eq;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    // Striped: entry j of the thread is tile entry j * PART_THREADS +
    // threadIdx.x, so that group g = j * WARPS + w is a run of 32 consecutive
    // entries, loaded and stored by one warp instruction each.  A flag's rank
    // inside its group comes from a ballot; the flags stay in two bit masks
    // and the entries' values are read again for the scatter.
    const int base = tile * PART_BS + threadIdx.x;
    int eo[PER], es[PER];
    unsigned fbits = 0, gbits = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * PART_THREADS;
        eo[j] = es[j] = 0;
        int fp = 0, fq = 0;
        if (i < A.k) {
            node_of(i, A.level, A.k, eo[j], es[j]);
            const int h = es[j] >> 1;
            fp = A.P[i] < h;
            fq = A.Q[i] < h;
        }
        const unsigned mp = __ballot_sync(FULL_MASK, fp), mq = __ballot_sync(FULL_MASK, fq);
        if (lane == 0) {
            gp[j * WARPS + w] = __popc(mp);
            gq[j * WARPS + w] = __popc(mq);
        }
        fbits |= unsigned(fp) << j;
        gbits |= unsigned(fq) << j;
    }
    __syncthreads();
    // Warp 0 scans the group counts (lane l: groups GPL l .. GPL l + GPL - 1),
    // publishes the tile's counts and looks back over its predecessors 32 at
    // a time: lane l reads tile (front - 1 - l); the window's nearest INCL
    // ends the look-back, otherwise its 32 AGG counts are added and the
    // window moves back.  A window with a tile that has not published yet is
    // read again (bounded by %globaltimer).
    if (w == 0) {
        int cp[GPL], cq[GPL], sp = 0, sq = 0;
#pragma unroll
        for (int t = 0; t < GPL; ++t) {
            cp[t] = gp[GPL * lane + t];
            cq[t] = gq[GPL * lane + t];
            sp += cp[t];
            sq += cq[t];
        }
        int xp = sp, xq = sq;
        for (int off = 1; off < 32; off <<= 1) {
            const int yp = __shfl_up_sync(FULL_MASK, xp, off), yq = __shfl_up_sync(FULL_MASK, xq, off);
            if (lane >= off) {
                xp += yp;
                xq += yq;
            }
        }
        const int tp = __shfl_sync(FULL_MASK, xp, 31), tq = __shfl_sync(FULL_MASK, xq, 31);
        int rp = xp - sp, rq = xq - sq;
#pragma unroll
        for (int t = 0; t < GPL; ++t) {
            gp[GPL * lane + t] = rp;
            gq[GPL * lane + t] = rq;
            rp += cp[t];
            rq += cq[t];
        }
        int ep = 0, eq = 0;
        bool ok = true;
        if (local) {
            // Every node of the level lies inside one tile: node-relative
            // counts need only the tile's own scan (no look-back).
        } else if (tile == 0) {
            if (lane == 0) st_release_u64(F.tiles, pack_counts(TILE_INCL, tp, tq));
        } else {
            if (lane == 0) st_release_u64(F.tiles + tile, pack_counts(TILE_AGG, tp, tq));
            int front = tile; // the window covers tiles [front - 32, front)
            uint64_t t0 = 0;
            while (front > 0) {
                const int j = front - 1 - lane;
                const unsigned long long v = j >= 0 ? ld_acquire_u64(F.tiles + j) : TILE_INCL;
                if (__any_sync(FULL_MASK, (v & (TILE_AGG | TILE_INCL)) == 0)) {
                    // a predecessor has not counted yet: read the window again
                    int stop = 0;
                    if (lane == 0) {
                        const uint64_t now = globaltimer_ns();
                        if (ld_relaxed_gpu(F.err)) {
                            stop = 1;
                        } else if (t0 == 0) {
                            t0 = now;
                        } else if (now - t0 > PART_WAIT_NS) {
                            atomicExch(F.err, 1);
                            raise_status(F.status, DEV_ERR_TIMEOUT);
                            stop = 1;
                        }
                    }
                    if (__shfl_sync(FULL_MASK, stop, 0)) {
                        ok = false;
                        break;
                    }
                    __nanosleep(64);
                    continue;
                }
                const unsigned incl = __ballot_sync(FULL_MASK, (v & TILE_INCL) != 0);
                const int first = incl ? __ffs(incl) - 1 : 32; // nearest INCL in the window
                int cp_ = lane <= first && j >= 0 ? int(v & TILE_COUNT_MASK) : 0;
                int cq_ = lane <= first && j >= 0 ? int((v >> 31) & TILE_COUNT_MASK) : 0;
                for (int off = 16; off; off >>= 1) {
                    cp_ += __shfl_xor_sync(FULL_MASK, cp_, off);
                    cq_ += __shfl_xor_sync(FULL_MASK, cq_, off);
                }
                ep += cp_;
                eq += cq_;
                if (incl) break;
                front -= 32;
            }
            if (ok && lane == 0) st_release_u64(F.tiles + tile, pack_counts(TILE_INCL, ep + tp, eq + tq));
        }
        if (lane == 0) {
            if (!ok) s_ok = 0;
            s_ep = ep;
            s_eq = eq;
        }
    }
    __syncthreads();
    if (!s_ok) return false;
    // The exclusive scan value of an entry over the whole level; only a
    // node's first entry stores it (the scatter needs node-relative counts).
    const int ep0 = s_ep, eq0 = s_eq;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * PART_THREADS;
        const unsigned mp = __ballot_sync(FULL_MASK, (fbits >> j) & 1u);
        const unsigned mq = __ballot_sync(FULL_MASK, (gbits >> j) & 1u);
        if (i < A.k && i == eo[j]) {
            A.scanP[i] = ep0 + gp[j * WARPS + w] + __popc(mp & below);
            A.scanQ[i] = eq0 + gq[j * WARPS + w] + __popc(mq & below);
        }
    }
    __threadfence();
    __syncthreads();
    // Node starts inside the tile are written; the one node that can start in
    // an earlier tile is the node of the tile's first entry: wait for that
    // tile's `done`.
    if (threadIdx.x == 0) {
        st_release_gpu(F.done + tile, 1);
        int o, sz;
        node_of(tile * PART_BS, A.level, A.k, o, sz);
        const int t_o = o / PART_BS;
        if (t_o < tile && !wait_done(F, t_o)) s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) return false;
    // Scan values at the node starts: written before the barrier above (this
    // tile) or before a done flag thread 0 acquired (an earlier tile); read
    // through L2, the point of coherence.
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * PART_THREADS;
        const unsigned mp = __ballot_sync(FULL_MASK, (fbits >> j) & 1u);
        const unsigned mq = __ballot_sync(FULL_MASK, (gbits >> j) & 1u);
        if (i >= A.k) continue;
        const int o = eo[j], sz = es[j];
        const int h = sz >> 1;
        const int p = A.P[i], q = A.Q[i];
        const int bp = ep0 + gp[j * WARPS + w] + __popc(mp & below) - __ldcg(A.scanP + o);
        const int bq = eq0 + gq[j * WARPS + w] + __popc(mq & below) - __ldcg(A.scanQ + o);
        const int local = i - o;
        const int pp = p < h ? o + bp : o + h + (local - bp);
        const int pq = q < h ? o + bq : o + h + (local - bq);
        // A destination outside the node can only come from a wrong scan
        // value: report it and store nothing.
        if (unsigned(pp - o) >= unsigned(sz) || unsigned(pq - o) >= unsigned(sz)) {
            atomicExch(F.err, 1);
            raise_status(F.status, DEV_ERR_BOUNDS);
            continue;
        }
        A.Pn[pp] = p < h ? p : p - h;
        A.pmap[pp] = local;
        A.Qn[pq] = q < h ? q : q - h;
        A.qmap[pq] = local;
    }
    return true;
}

template <int PART_THREADS, int N>
__global__ void __launch_bounds__(PART_THREADS) part_levels_kernel(const __grid_constant__ Many<PartAllArgs, N> M)
{
    const PartAllArgs &G = M.of[blockIdx.z];
    constexpr int PART_BS = PART_THREADS * PART_PER;
    __shared__ PartSmem<PART_THREADS> S;
    __shared__ int s_ticket;
    const size_t kk = size_t(G.k);
    for (;;) {
        __syncthreads(); // the previous tile is done with the shared arrays
        if (threadIdx.x == 0) {
            s_ticket = atomicAdd(G.ticket, 1);
            S.s_ok = !ld_relaxed_gpu(G.err);
            const int lv = s_ticket / G.kb, tl = s_ticket % G.kb;
            if (S.s_ok && lv > 0 && lv < G.levels) {
                // This tile's input is written by the tiles of the level above
                // that hold a node overlapping the tile: when the parent nodes
                // are at most two tiles long (power-of-two k), those tiles
                // only; otherwise every tile of the level.
                const int ps = G.k >> (lv - 1); // parent node size (power-of-two k)
                const bool near = G.pow2 && ps <= 2 * PART_BS;
                const int32_t *ctr = G.level_done + lv - 1;
                int want = G.kb, ta = 0, tb = 0;
                if (near) {
                    ta = (tl * PART_BS) / ps * ps / PART_BS;
                    tb = min(G.kb - 1, ((tl * PART_BS + PART_BS - 1) / ps * ps + ps - 1) / PART_BS);
                    want = 1;
                }
                for (int u = ta; u <= tb && S.s_ok; ++u) {
                    if (near) ctr = G.scat + size_t(lv - 1) * G.kb + u;
                    uint64_t t0 = 0;
                    while (ld_acquire_gpu(ctr) < want) {
                        if (ld_relaxed_gpu(G.err)) {
                            S.s_ok = 0;
                            break;
                        }
                        const uint64_t now = globaltimer_ns();
                        if (t0 == 0) {
                            t0 = now;
                        } else if (now - t0 > PART_WAIT_NS) {
                            atomicExch(G.err, 1);
                            raise_status(G.status, DEV_ERR_TIMEOUT);
                            S.s_ok = 0;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
            }
        }
        __syncthreads();
        const int t = s_ticket;
        if (!S.s_ok || t >= G.levels * G.kb) return;
        const int lv = t / G.kb, tile = t % G.kb;
        int32_t *in = G.PQ + ((lv & 1) ? 2 * kk : 0), *nx = G.PQ + ((lv & 1) ? 0 : 2 * kk);
        int32_t *mp = G.maps + 2 * kk * size_t(lv + 1);
        FusedArgs F{LevelArgs{in, in + kk, nx, nx + kk, mp, mp + kk, G.scanP, G.scanQ, G.k, lv,
                              G.err},
                    G.tiles + size_t(lv) * G.kb, G.done + size_t(lv) * G.kb, G.err, G.status};
        const bool local = G.pow2 && (G.k >> lv) <= PART_BS; // the level's nodes fit inside tiles
        if (!part_tile<PART_THREADS>(F, tile, local, S)) return;
        __syncthreads(); // every thread of the tile has scattered
        if (threadIdx.x == 0) {
            __threadfence();
            st_release_gpu(G.scat + size_t(lv) * G.kb + tile, 1);
            atomicAdd(G.level_done + lv, 1);
        }
    }
}



// ---------------------------------------------------------------------------
// the ant walk (ant_passage, src/braid_multiplication.hpp:123-189)
// ---------------------------------------------------------------------------
// A node's glued state as packed words: the word of row r holds the column of
// its point, the word of column c the row of its point, each with bit 31 set
// when the point comes from the hi half.
//
// The reference keeps two dominance counts (dom_sum_count, 39-119) and moves
// right while hi-above-left minus lo-below-right is negative, up while it is
// zero.  Only that difference, delta(r, c) = #{hi: row < r, col < c} -
// #{lo: row >= r, col >= c}, decides anything, and one step changes it by the
// contribution of a single row or column:
__device__ __forceinline__ int word_inc(int w, int lim)
{
    const int p = w & INT_MAX;
    return w < 0 ? int(p < lim) : int(p >= lim);
}

// Walks from the point (dr, dc) with delta = delta(dr, dc) while dr >= 0,
// dc <= s and the diagonal dc - dr stays <= last; put(r, c) records a fresh
// point (the reference's test at 171-181: delta left of the point negative,
// delta below it positive).  rw(r) / cw(c) read row / column words.
//
// This general form serves starts with any delta.  On the walk itself delta
// only takes the values -1 and 0: a right move (delta < 0) adds 0 or 1, an
// up move (delta == 0) subtracts 0 or 1.  ant_walk below uses that.
template <typename RowW, typename ColW, typename Put>
__device__ __forceinline__ void ant_walk_general(int dr, int dc, int delta, int s, int last, RowW rw, ColW cw, Put put)
{
    while (dr >= 0 && dc <= s && dc - dr <= last) {
        if (dc > 0 && delta - word_inc(cw(dc - 1), dr) < 0 && delta + word_inc(rw(dr), dc) > 0) put(dr, dc - 1);
        if (delta < 0) {
            if (dc + 1 <= s) delta += word_inc(cw(dc), dr);
            ++dc;
        } else if (delta == 0) {
            if (dr - 1 >= 0) delta -= word_inc(rw(dr - 1), dc);
            --dr;
        } else {
            break;
        }
    }
}

// The walk as a two-state machine (up: delta == 0, right: delta == -1).  A
// step needs the words of rows dr, dr-1 and columns dc-1, dc, which it keeps
// in registers; it loads the two words either move could need next before
// deciding, and moves by selects.  The trip count only bounds the walk (each
// step moves dc - dr up by one, and the walk leaves the box after at most
// dr + s - dc + 1 steps), so the loop carries no data-dependent branch.
// (A variant that also precomputed the four flip values of the step after
// next ran slower: a lone walking warp is bound by the instructions it
// issues per step as much as by their dependency chain.)
template <typename RowW, typename ColW, typename Put>
__device__ __forceinline__ void ant_walk(int dr, int dc, int delta, int s, int last, RowW rw, ColW cw, Put put)
{
    if (delta != 0 && delta != -1) {
        ant_walk_general(dr, dc, delta, s, last, rw, cw, put);
        return;
    }
    bool up = delta == 0;
    bool alive = dr >= 0 && dc <= s && dc - dr <= last;
    if (!alive) return;
    int r0 = rw(dr);                                // row dr
    int r1 = dr >= 1 ? rw(dr - 1) : 0;              // row dr - 1
    int cm = dc >= 1 ? cw(dc - 1) : 0;              // column dc - 1
    int c0 = dc < s ? cw(dc) : 0;                   // column dc
    const int trips = int(min(int64_t(last) - (dc - dr), int64_t(dr) + s - dc)) + 1;
#pragma unroll 4
    for (int t = 0; t < trips; ++t) {
        const int r2 = dr >= 2 ? rw(dr - 2) : 0;
        const int c1 = dc + 1 < s ? cw(dc + 1) : 0;
        if (alive && up && dc > 0 && word_inc(cm, dr) && word_inc(r0, dc)) put(dr, dc - 1);
        const int inc_right = (dc + 1 <= s) ? word_inc(c0, dr) : 0;
        const int inc_up = dr >= 1 ? word_inc(r1, dc) : 0;
        const bool mv_up = alive && up, mv_right = alive && !up;
        const bool flip = up ? inc_up : inc_right;
        dc += mv_right;
        dr -= mv_up;
        cm = mv_right ? c0 : cm;
        c0 = mv_right ? c1 : c0;
        r0 = mv_up ? r1 : r0;
        r1 = mv_up ? r2 : r1;
        up = alive ? (up != flip) : up;
        alive = alive && dr >= 0 && dc <= s && dc - dr <= last;
    }
}

// The same walk by a whole warp, as alternating runs: an up run climbs while
// the row above adds nothing (delta stays 0), a right run moves while the
// column adds nothing (delta stays -1), and the move that adds one ends the
// run and turns the walk.  A fresh point can only lie where an up run starts:
// every later position of the run was reached by a move whose row word added
// nothing, and the test needs that word to add one.  Each run is found 32
// moves at a time, lane l testing the word of the run's (t + 1 + l)-th move;
// the first lane whose move turns the walk (or leaves the box) ends it.  (A
// lone thread walking runs with branches was slower than the two-state step
// above: lanes walking different nodes diverge.)  Lanes may read up
// to 31 words past the walk's last move; rw / cw must accept any index
// there (the window readers clamp), and their answers are not used.  Every
// lane returns with the same state; lane 0 writes the fresh points.
template <typename RowW, typename ColW, typename Put>
__device__ __forceinline__ void ant_walk_warp(int dr, int dc, int delta, int s, int last, RowW rw, ColW cw, Put put,
                                              int lane)
{
    if (delta != 0 && delta != -1) {
        if (lane == 0) ant_walk_general(dr, dc, delta, s, last, rw, cw, put);
        return;
    }
    if (!(dr >= 0 && dc <= s && dc - dr <= last)) return;
    int left = int(min(int64_t(last) - (dc - dr), int64_t(dr) + s - dc)) + 1;
    bool up = delta == 0;
    while (left > 0) {
        int t = 0;
        unsigned hit = 0;
        if (up) {
            if (lane == 0 && dc > 0 && word_inc(cw(dc - 1), dr) && word_inc(rw(dr), dc)) put(dr, dc - 1);
            while (t < left) {
                const int r = dr - (t + 1 + lane);
                hit = __ballot_sync(FULL_MASK, r < 0 || word_inc(rw(r), dc) != 0);
                if (hit) break;
                t += 32;
            }
            if (!hit) return;
            t += __ffs(hit);
            if (t > left || dr - t < 0) return; // out of steps, or it left the box upwards
            dr -= t;
        } else {
            while (t < left) {
                const int c = dc + t + lane;
                hit = __ballot_sync(FULL_MASK, c >= s || word_inc(cw(c), dr) != 0);
                if (hit) break;
                t += 32;
            }
            if (!hit) return;
            t += __ffs(hit);
            if (t > left || dc + t > s) return; // out of steps, or it left the box to the right
            dc += t;
        }
        left -= t;
        up = !up;
    }
}

// The walk's rows side by side: on its way up the walk leaves row r at
// c*(r), the first column with delta(r, c) = 0, whatever way it came, so a
// segment's rows need not wait for one another.  Lane t of a group takes row
// dr - t: delta(dr - t, dc) is the start's minus the increments of the rows
// between (a warp scan), and c* is where the increments of the columns from dc
// on have made up for it (counted from shared memory, every lane reading the
// same column).  Rows and columns beyond the segment's last diagonal belong to
// later segments, so the counts form a triangle of B^2 / 2.  A fresh point can
// only lie at (r, c* - 1).  Needs -1 <= delta <= 0 and, unless dc is 0,
// delta(dr, dc - 1) < 0, as on every start of a segment; col holds last + 1 -
// (dc - dr) entries.
template <typename RowW, typename ColW, typename Put>
__device__ __forceinline__ void walk_rows(int dr, int dc, int delta, int last, int s, RowW rw, ColW cw, Put put,
                                          int2 *col, int lane)
{
    const int most = last - (dc - dr); // row dr - t looks at columns dc to dc + most - t
    if (most < 0) return;
    for (int j = lane; j < most; j += 32) {
        const int w = dc + j < s ? cw(dc + j) : 0;
        col[j] = make_int2(w & INT_MAX, w < 0 ? 0 : -1);
    }
    __syncwarp();
    int carry = -delta;
    for (int t0 = 0; t0 <= min(most, dr); t0 += 32) {
        const int t = t0 + lane, r = dr - t;
        const int w = r >= 0 ? rw(r) : 0;
        int need = t > 0 && r >= 0 ? word_inc(w, dc) : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, need, off);
            if (lane >= off) need += y;
        }
        need += carry;
        carry = __shfl_sync(FULL_MASK, need, 31);
        int c = dc;
        const int cols = most - t0;
#pragma unroll 8
        for (int j = 0; j < cols; ++j) {
            const int2 p = col[j];
            c += need > 0;
            need += ((p.x - r) ^ p.y) >> 31; // hi: row above r; lo: row r or below
        }
        if (r >= 0 && need <= 0 && c - r <= last && c > 0 && word_inc(w, c)) put(r, c - 1);
    }
}

// ---------------------------------------------------------------------------
// nodes at or below the cutoff
// ---------------------------------------------------------------------------
struct NodeArgs {
    const int32_t *P; // level lc arrays (global): P's rows by column, Q's columns by row
    const int32_t *Q;
    int32_t *res;     // level lc result (global), node-local r2c
    int k, lc;
    const int32_t *bad;
};

// One round element of a node: P's row that ends on middle position j in the
// high half, the complement of the column where Q's row j ends in the low half.
__device__ __forceinline__ uint32_t pass_low(uint32_t l, uint32_t r) { return l > r ? __vminu2(l, r) : l; }
__device__ __forceinline__ uint32_t pass_high(uint32_t l, uint32_t r) { return l > r ? __vmaxu2(l, r) : r; }
__device__ __forceinline__ void pass_pair(uint32_t &l, uint32_t &r)
{
    const uint32_t low = pass_low(l, r);
    r = l + r - low; // both halves keep their sums
    l = low;
}

// One block multiplies one node of level lc (size S <= NODE_MAX) by passing
// P's crossings into Q one by one, without any recursion.  Odd-even
// transposition sorts P's strands along the middle: every exchange is one
// crossing of a reduced word of P taken off P's right end, and
// sigma_j . R exchanges rows j and j + 1 of R unless those two strands have
// crossed already.  With R's columns complemented both exchanges take the
// smaller half to the left, so one packed minimum does them (4 instructions a
// pair).  S rounds of S / 2 independent pairs: S^2 / 2 pairs in all, against
// S log S steps of a recursion, whose walks and scans are serial chains.  A
// 1024-entry node took 183 us as a shared-memory recursion and takes 32 us
// here, bound by the ALU pipe (30 of its 40 instructions a lane per round run
// at half rate); products of k = 1003 231 -> 75 us, 32768 486 -> 334 us
// (MEASURED).  Larger nodes lose to one more level of the recursion: 2048
// entries 93 us, against two of 1024 side by side and a level of about 45 us.
//
// A lane holds NODE_E consecutive entries: rounds of even pairs stay in the
// lane, odd ones cross one lane boundary (two shuffles, both sides compute
// their half).  With several warps each warp owns 30 lanes, and its outer two
// lanes repeat the neighbours' edge lanes: a round spoils one more of their
// entries from the outside, so NODE_E rounds pass before the edges are
// exchanged through shared memory at one barrier.  NODE_E = 10 gives a
// 1024-entry node four warps, one on each SM sub-partition (8 gave it five:
// whole product of k = 1024 76 us against 67).
constexpr int NODE_E = 10;
constexpr int NODE_OWN = 30 * NODE_E; // entries a warp owns when a block has several
constexpr int NODE_MAX = 1200;
constexpr int NODE_WARPS = (NODE_MAX + NODE_OWN - 1) / NODE_OWN;
inline int node_warps(int smax) { return smax <= 32 * NODE_E ? 1 : (smax + NODE_OWN - 1) / NODE_OWN; }

template <bool ONE_WARP, int N>
__global__ void __launch_bounds__(ONE_WARP ? 32 : NODE_WARPS * 32)
    node_kernel(const __grid_constant__ Many<NodeArgs, N> M)
{
    const NodeArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    __shared__ uint16_t half[2 * (ONE_WARP ? 32 * NODE_E : NODE_MAX)]; // entry j: column half, row half
    __shared__ __align__(8) uint32_t edge[ONE_WARP ? 1 : 2][ONE_WARP ? 1 : NODE_WARPS][2][NODE_E];
    // node of this block: descend lc levels following the bits of blockIdx.x
    int o = 0, S = A.k;
    for (int d = 0; d < A.lc; ++d) {
        const int h = S >> 1;
        if ((blockIdx.x >> (A.lc - 1 - d)) & 1) {
            o += h;
            S -= h;
        } else {
            S = h;
        }
    }
    for (int i = threadIdx.x; i < S; i += blockDim.x) {
        const int p = A.P[o + i], q = A.Q[o + i];
        if (unsigned(p) < unsigned(S)) half[2 * p + 1] = uint16_t(i);
        if (unsigned(q) < unsigned(S)) half[2 * q] = uint16_t(0xFFFF - i);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int warp = ONE_WARP ? 0 : int(threadIdx.x >> 5), warps = ONE_WARP ? 1 : int(blockDim.x >> 5);
    const int base = (ONE_WARP ? lane : warp * 30 + lane - 1) * NODE_E;
    uint32_t x[NODE_E];
#pragma unroll
    for (int e = 0; e < NODE_E; ++e) {
        const int j = base + e; // outside the node: words no neighbour exchanges with
        x[e] = j < 0 ? 0u : j >= S ? 0xFFFFFFFFu : (uint32_t(half[2 * j + 1]) << 16 | half[2 * j]);
    }
    for (int t = 0; t < S; t += NODE_E) {
#pragma unroll
        for (int u = 0; u < NODE_E; u += 2) {
#pragma unroll
            for (int e = 0; e < NODE_E; e += 2) pass_pair(x[e], x[e + 1]);
            uint32_t next = __shfl_down_sync(FULL_MASK, x[0], 1);
            uint32_t prev = __shfl_up_sync(FULL_MASK, x[NODE_E - 1], 1);
            if (ONE_WARP) {
                if (lane == 31) next = 0xFFFFFFFFu;
                if (lane == 0) prev = 0u;
            }
#pragma unroll
            for (int e = 1; e + 1 < NODE_E; e += 2) pass_pair(x[e], x[e + 1]);
            x[NODE_E - 1] = pass_low(x[NODE_E - 1], next);
            x[0] = pass_high(prev, x[0]);
        }
        if (!ONE_WARP) {
            const int buf = (t / NODE_E) & 1;
            if (lane == 1 || lane == 30) {
                uint2 *to = reinterpret_cast<uint2 *>(edge[buf][warp][lane == 30]);
#pragma unroll
                for (int e = 0; e < NODE_E; e += 2) to[e / 2] = make_uint2(x[e], x[e + 1]);
            }
            __syncthreads();
            const int from = lane == 0 ? warp - 1 : warp + 1;
            if ((lane == 0 || lane == 31) && from >= 0 && from < warps) {
                const uint2 *in = reinterpret_cast<const uint2 *>(edge[buf][from][lane == 0]);
#pragma unroll
                for (int e = 0; e < NODE_E; e += 2) {
                    const uint2 w = in[e / 2];
                    x[e] = w.x;
                    x[e + 1] = w.y;
                }
            }
        }
    }
    if (!ONE_WARP && (lane == 0 || lane == 31)) return;
#pragma unroll
    for (int e = 0; e < NODE_E; ++e)
        if (base + e < S) A.res[o + base + e] = int32_t(0xFFFFu - (x[e] & 0xFFFFu));
}

// ---------------------------------------------------------------------------
// upward levels above the cutoff
// ---------------------------------------------------------------------------
struct GlueArgs {
    const int32_t *child_res; // level l+1 results
    const int32_t *pmap;      // level l+1 maps
    const int32_t *qmap;
    int32_t *CW, *RW;         // packed words: row r -> its column | hi << 31, column c -> its row | hi << 31
    int32_t *res;             // level l result
    int k, level;
    const int32_t *bad;
    // Block counts of the level's delta tables, counted as the points are
    // glued: (G+1)^2 per node and table, G = node size / B.
    int32_t *cnt_hi, *cnt_lo;
    int B, stride;
    // The next level's tables: the other of the two table buffers, free since
    // the walk one level down read it; zeroed here for that level's glue
    // (instead of a memset launch per level).
    int32_t *clear;
    long long nclear;
};

template <int N>
__global__ void __launch_bounds__(256) glue_kernel(const __grid_constant__ Many<GlueArgs, N> M)
{
    const GlueArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < A.nclear;
         i += (long long)gridDim.x * blockDim.x)
        A.clear[i] = 0;
    const bool pow2 = (A.k & (A.k - 1)) == 0;
    int lg = 0; // log2 k for a power of two
    while (pow2 && (1 << lg) < A.k) ++lg;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.k; i += gridDim.x * blockDim.x) {
        // parent node (offset, size, index) and child node of entry i: for a
        // power-of-two k every node of a level has size k >> level
        int po = 0, ps = A.k, nd = 0;
        if (pow2) {
            ps = A.k >> A.level;
            nd = i >> (lg - A.level);
            po = nd * ps;
        } else {
            for (int d = 0; d < A.level; ++d) {
                const int h = ps >> 1;
                nd <<= 1;
                if (i < po + h) {
                    ps = h;
                } else {
                    po += h;
                    ps -= h;
                    nd |= 1;
                }
            }
        }
        const int co = i < po + (ps >> 1) ? po : po + (ps >> 1);
        const int prow = A.pmap[i];
        const int pcol = A.qmap[co + A.child_res[i]];
        const int32_t hi = co != po ? INT_MIN : 0;
        A.CW[po + prow] = pcol | hi;
        A.RW[po + pcol] = prow | hi;
        A.res[po + prow] = pcol; // the union of both halves; the walk adds the fresh points
        if (A.cnt_hi) {
            const int G = ps / A.B;
            const int bi = min(prow / A.B, G), bj = min(pcol / A.B, G);
            int32_t *t = (hi ? A.cnt_hi : A.cnt_lo) + size_t(nd) * A.stride * A.stride;
            atomicAdd(t + bi * A.stride + bj, 1);
        }
    }
}


// ---------------------------------------------------------------------------
// concurrent walk of large nodes
//
// delta(r, c) = #{hi points with row < r, col < c} - #{lo points with row >= r,
// col >= c} is non-decreasing in r and in c, changes by 0 or 1 per unit step,
// and the reference's walk turns right where it is negative and up where it
// is zero.  Each step moves to the next diagonal e = col - row, and the walk's
// row on diagonal e is r*(e-1) - 1 with r*(e) the first row of diagonal e whose
// delta is >= 0.  A level therefore tabulates delta at the grid points that
// are multiples of B (per node, a (G+1)^2 table from block counts), and walk
// segment q, which owns diagonals (E, E+B] for E a multiple of B, finds r*(E)
// by a binary search over the table and a warp scan inside one block, then
// walks its B diagonals alone.  Every segment writes its fresh points.
// ---------------------------------------------------------------------------
constexpr int WALK_GMAX = 1024; // grid lines per node and dimension, at most
constexpr int WALK_BMIN = 64;   // smallest grid spacing

struct TableArgs {
    const int32_t *__restrict__ CW; // row words (column | hi << 31)
    int32_t *cnt_hi; // (G+1)^2 per node, becomes the delta table
    int32_t *cnt_lo;
    int k, level, B, stride; // stride = Gmax+1 for the level
    const int32_t *bad;
};

__device__ __forceinline__ void node_by_index(int nd, int level, int k, int &o, int &s)
{
    o = 0;
    s = k;
    for (int e = 0; e < level; ++e) {
        const int h = s >> 1;
        if ((nd >> (level - 1 - e)) & 1) {
            o += h;
            s -= h;
        } else {
            s = h;
        }
    }
}

// One warp per (node, row block): exclusive prefix of the hi counts and
// inclusive suffix of the lo counts along the row, the two scans side by side
// (hi from the left, lo from the right), ROW_STEPS groups of 32 columns at a
// time: a lone warp's row is bound by the latency of its reads and shuffles,
// so the groups' scans run side by side and the next ones' words are read before
// them (one group at a time: products of overlap 32768 187 -> 183 us, 131072
// 331 -> 316; eight: 183 and 320).
constexpr int ROW_STEPS = 4;
template <int N>
__global__ void __launch_bounds__(256) table_rows_kernel(const __grid_constant__ Many<TableArgs, N> M, int nodes)
{
    const TableArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    const int lane = threadIdx.x & 31;
    const long wid = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (wid >= long(nodes) * A.stride) return;
    const int nd = int(wid / A.stride), bi = int(wid % A.stride);
    int o, s;
    node_by_index(nd, A.level, A.k, o, s);
    const int G = s / A.B;
    if (bi > G) return;
    int32_t *hi = A.cnt_hi + size_t(nd) * A.stride * A.stride + size_t(bi) * A.stride;
    int32_t *lo = A.cnt_lo + size_t(nd) * A.stride * A.stride + size_t(bi) * A.stride;
    const int nch = G / 32 + 1; // steps of 32 columns over 0..G
    int nh[ROW_STEPS], nl[ROW_STEPS];
    auto load = [&](int c0) {
#pragma unroll
        for (int u = 0; u < ROW_STEPS; ++u) {
            const int jh = (c0 + u) * 32 + lane, jl = (nch - 1 - c0 - u) * 32 + lane;
            nh[u] = jh <= G ? hi[jh] : 0;
            nl[u] = jl >= 0 && jl <= G ? lo[jl] : 0;
        }
    };
    load(0);
    int carry_h = 0, carry_l = 0;
    for (int c0 = 0; c0 < nch; c0 += ROW_STEPS) {
        int vh[ROW_STEPS], xh[ROW_STEPS], xl[ROW_STEPS]; // xl becomes the sum over lanes >= lane
#pragma unroll
        for (int u = 0; u < ROW_STEPS; ++u) {
            vh[u] = xh[u] = nh[u];
            xl[u] = nl[u];
        }
        if (c0 + ROW_STEPS < nch) load(c0 + ROW_STEPS);
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
#pragma unroll
            for (int u = 0; u < ROW_STEPS; ++u) {
                const int yh = __shfl_up_sync(FULL_MASK, xh[u], off);
                const int yl = __shfl_down_sync(FULL_MASK, xl[u], off);
                if (lane >= off) xh[u] += yh;
                if (lane + off < 32) xl[u] += yl;
            }
#pragma unroll
        for (int u = 0; u < ROW_STEPS; ++u) {
            const int jh = (c0 + u) * 32 + lane, jl = (nch - 1 - c0 - u) * 32 + lane;
            if (jh <= G) hi[jh] = carry_h + xh[u] - vh[u];
            if (jl >= 0 && jl <= G) lo[jl] = carry_l + xl[u];
            carry_h += __shfl_sync(FULL_MASK, xh[u], 31);
            carry_l += __shfl_sync(FULL_MASK, xl[u], 0);
        }
    }
}

// One block per (node, COLS grid columns): a three-phase scan down the rows
// (CHUNKS row chunks per column; the chunk's words stay in registers between
// the phases) that finishes the 2D sums and stores delta(iB, jB) =
// hi-prefix - lo-suffix in the hi table.  Large tables (the top levels: one
// or two nodes of up to 1025 columns) take 4 columns x 64 row chunks per
// block, so that they still spread over all the SMs; small ones (many nodes
// of at most TCOL_SMALL_ROWS rows) 32 columns x 8 chunks.
constexpr int TCOL_PER = (WALK_GMAX + 1 + 63) / 64; // rows of a chunk, at most
constexpr int TCOL_SMALL_ROWS = 8 * TCOL_PER;
template <int COLS, int CHUNKS, int N>
__global__ void __launch_bounds__(COLS * CHUNKS) table_cols_kernel(const __grid_constant__ Many<TableArgs, N> M, int nodes)
{
    const TableArgs &A = M.of[blockIdx.z];
    constexpr int TCOL_COLS = COLS, TCOL_CHUNKS = CHUNKS;
    if (*A.bad) return;
    const int colblocks = (A.stride + TCOL_COLS - 1) / TCOL_COLS;
    const int nd = blockIdx.x / colblocks, jb = blockIdx.x % colblocks;
    int o, s;
    node_by_index(nd, A.level, A.k, o, s);
    const int G = s / A.B;
    const int tx = threadIdx.x % TCOL_COLS, ty = threadIdx.x / TCOL_COLS;
    const int j = jb * TCOL_COLS + tx;
    const bool col_ok = j <= G;
    const int rows = G + 1, per = (rows + TCOL_CHUNKS - 1) / TCOL_CHUNKS;
    const int i0 = min(rows, ty * per), i1 = min(rows, i0 + per);
    int32_t *hi = A.cnt_hi + size_t(nd) * A.stride * A.stride + j;
    const int32_t *lo = A.cnt_lo + size_t(nd) * A.stride * A.stride + j;
    __shared__ int Hs[TCOL_CHUNKS][TCOL_COLS + 1], Ls[TCOL_CHUNKS][TCOL_COLS + 1];
    int vh[TCOL_PER], vl[TCOL_PER];
    int hs = 0, ls = 0;
    {
        const int32_t *ph = hi + size_t(i0) * A.stride, *pl = lo + size_t(i0) * A.stride;
        const int n = col_ok ? i1 - i0 : 0;
#pragma unroll
        for (int u = 0; u < TCOL_PER; ++u) {
            vh[u] = u < n ? ph[u * A.stride] : 0;
            vl[u] = u < n ? pl[u * A.stride] : 0;
            hs += vh[u];
            ls += vl[u];
        }
    }
    Hs[ty][tx] = hs;
    Ls[ty][tx] = ls;
    __syncthreads();
    int hoff = 0, loff = 0;
    for (int t = 0; t < ty; ++t) hoff += Hs[t][tx];
    for (int t = ty + 1; t < TCOL_CHUNKS; ++t) loff += Ls[t][tx];
    if (!col_ok) return;
    int run_h = hoff, run_l = loff + ls; // #lo points with row >= i0 + u, col >= jB
    int32_t *ph = hi + size_t(i0) * A.stride;
    const int n = i1 - i0;
#pragma unroll
    for (int u = 0; u < TCOL_PER; ++u) {
        if (u < n) ph[u * A.stride] = run_h - run_l; // delta(iB, jB)
        run_h += vh[u];
        run_l -= vl[u];
    }
}

// Levels whose tables have at most SMALL_TABLE entries: one block per node
// finishes the whole table in shared memory (row pass, then column pass):
// delta(iB, jB) = #{hi blocks above-left} - #{lo blocks at or below-right}.
constexpr int SMALL_TABLE = 4096;
template <int N>
__global__ void __launch_bounds__(256) table_small_kernel(const __grid_constant__ Many<TableArgs, N> M, int nodes)
{
    const TableArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    __shared__ int32_t hs[SMALL_TABLE], ls[SMALL_TABLE];
    const int nd = blockIdx.x;
    if (nd >= nodes) return;
    int o, s;
    node_by_index(nd, A.level, A.k, o, s);
    const int G = s / A.B, W = A.stride, n = (G + 1) * W;
    int32_t *hi = A.cnt_hi + size_t(nd) * W * W, *lo = A.cnt_lo + size_t(nd) * W * W;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        hs[t] = hi[t];
        ls[t] = lo[t];
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= G; i += blockDim.x) { // rows: hi exclusive prefix, lo inclusive suffix
        int run = 0;
        for (int j = 0; j <= G; ++j) {
            const int v = hs[i * W + j];
            hs[i * W + j] = run;
            run += v;
        }
        run = 0;
        for (int j = G; j >= 0; --j) {
            run += ls[i * W + j];
            ls[i * W + j] = run;
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j <= G; j += blockDim.x) { // columns, then delta into the hi table
        int run = 0;
        for (int i = G; i >= 0; --i) {
            run += ls[i * W + j];
            ls[i * W + j] = run;
        }
        run = 0;
        for (int i = 0; i <= G; ++i) {
            const int v = hs[i * W + j];
            hi[i * W + j] = run - ls[i * W + j];
            run += v;
        }
    }
}

struct SegArgs {
    const int32_t *__restrict__ CW; // row words (column | hi << 31)
    const int32_t *__restrict__ RW; // column words (row | hi << 31)
    const int32_t *T; // delta tables
    int32_t *res;
    int k, level, B, stride, nseg; // nseg: segments per node
    const int32_t *bad;
};

// delta(r+1, c) - delta(r, c): the point of row r joins the hi count or
// leaves the lo count.
__device__ __forceinline__ int rowinc(const SegArgs &A, int o, int r, int c)
{
    return word_inc(__ldg(A.CW + o + r), c);
}
// delta(r, c+1) - delta(r, c)
__device__ __forceinline__ int colinc(const SegArgs &A, int o, int c, int r)
{
    return word_inc(__ldg(A.RW + o + c), r);
}

// Rows and columns a walk segment can touch, staged per warp in shared
// memory (packed: position | hi flag in bit 31) before lane 0 walks.
// Per warp two arrays of `win` words, win = min(B + 12, WALK_WIN) for the
// level (dynamic shared memory, so that levels with short segments keep many
// warps resident).
constexpr int WALK_WIN = 1040;
constexpr int WALK_LANE_B = 256;
constexpr int WALK_ROW_B = 128; // segments up to this long walk their rows side by side
__host__ __device__ inline int walk_win(int B) { return B + 12 < WALK_WIN ? B + 12 : WALK_WIN; }

template <int N>
__global__ void __launch_bounds__(128) walk_segments_kernel(const __grid_constant__ Many<SegArgs, N> M, int nodes)
{
    const SegArgs &A = M.of[blockIdx.z];
    extern __shared__ int32_t walk_smem[];
    if (*A.bad) return;
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= nodes * A.nseg) return;
    const int nd = w / A.nseg, q = w % A.nseg;
    int o, s;
    node_by_index(nd, A.level, A.k, o, s);
    if (s <= 1) return;
    const int B = A.B;
    const int G = s / B;
    const int32_t *T = A.T + size_t(nd) * A.stride * A.stride;
    const int jmin = -((s + B - 1) / B); // floor(-s / B)
    const int E = (jmin + q) * B;
    const int e0 = -(s - 1);
    if (E > s || E + B < e0) return;
    int dr, dc, delta;
    if (E < e0) {
        dr = s - 1;
        dc = 0;
        delta = __ldg(A.CW + o + s - 1) < 0 ? 0 : -1;
    } else {
        const int rlo = max(0, -E), rhi = min(s, s - E);
        if (rlo > rhi) return;
        const int jj = E / B;
        const int ilo = rlo / B, ihi = rhi / B;
        // First grid point of diagonal E with delta >= 0 (delta does not
        // decrease along a diagonal): the warp probes 32 evenly spaced points
        // of the range at once and keeps the stretch where the test turns.
        int lo_i = ilo, hi_i = ihi + 1;
        while (lo_i < hi_i) {
            const int step = (hi_i - lo_i + 31) >> 5;
            const int pi = lo_i + lane * step;
            const bool ge = pi < hi_i && T[pi * A.stride + pi + jj] >= 0;
            const unsigned inside = __ballot_sync(FULL_MASK, pi < hi_i);
            const unsigned hit = __ballot_sync(FULL_MASK, ge);
            if (hit & 1u) {
                hi_i = lo_i; // the first point already passes
                break;
            }
            if (hit) {
                const int f = __ffs(hit) - 1;
                const int nlo = lo_i + (f - 1) * step + 1;
                hi_i = lo_i + f * step;
                lo_i = nlo;
            } else {
                lo_i = lo_i + (31 - __clz(inside)) * step + 1; // past the last probe inside the range
            }
        }
        const int istar = hi_i;
        int rstar;
        int dstart = T[ilo * A.stride + ilo + jj]; // delta(rlo, rlo + E): a grid point
        if (istar == ilo) {
            rstar = rlo;
        } else {
            int rb = (istar - 1) * B;
            int dval = T[(istar - 1) * A.stride + (istar - 1) + jj];
            const int rend = min(istar * B, rhi);
            rstar = rhi + 1;
            // The increments of the next 32 rows are loaded before this
            // chunk is scanned, so that their latency overlaps the scan.
            auto inc_at = [&](int r) {
                return r < rend ? colinc(A, o, r + E, r) + rowinc(A, o, r, r + E + 1) : 0;
            };
            int inc_next = inc_at(rb + lane);
            for (; rb < rend; rb += 32) {
                const int r = rb + lane;
                const int inc = inc_next;
                inc_next = inc_at(r + 32);
                int pre = inc;
                for (int off = 1; off < 32; off <<= 1) {
                    const int y = __shfl_up_sync(FULL_MASK, pre, off);
                    if (lane >= off) pre += y;
                }
                const unsigned hit = __ballot_sync(FULL_MASK, r < rend && dval + pre >= 0);
                if (hit) {
                    rstar = rb + __ffs(hit); // lane f (1-based) reaches row rb + f
                    dstart = dval + __shfl_sync(FULL_MASK, pre, __ffs(hit) - 1);
                    break;
                }
                dval += __shfl_sync(FULL_MASK, pre, 31);
            }
        }
        dr = rstar - 1;
        dc = rstar + E;
        if (rstar > rhi || dr < 0 || dc > s) return;
        // dstart = delta(r*, r* + E); one row up the point of row r* - 1 leaves
        delta = dstart - rowinc(A, o, dr, dc);
    }
    (void)G;
    if (B <= WALK_ROW_B) {
        int2 *col = reinterpret_cast<int2 *>(walk_smem) + size_t(threadIdx.x >> 5) * B;
        walk_rows(
            dr, dc, delta, E + B, s, [&](int r) { return __ldg(A.CW + o + r); },
            [&](int c) { return __ldg(A.RW + o + c); }, [&](int r, int c) { A.res[o + r] = c; }, col, lane);
        return;
    }
    // The segment walks at most B + 1 steps, each one row up or one column
    // right: rows [dr - B - 6, dr] and columns [dc - 1, dc + B + 5] cover
    // them.  The warp stages them (coalesced), then walks in shared memory.
    const int wi = threadIdx.x >> 5;
    const int win = walk_win(B);
    int32_t *wr_s = walk_smem + size_t(wi) * 2 * win, *wc_s = wr_s + win;
    const int rb = max(0, dr - B - 6), nr = min(max(dr - rb + 1, 0), win);
    const int cb = max(0, dc - 1), nc = min(max(min(s, dc + B + 6) - cb, 0), win);
#pragma unroll 4
    for (int t = lane; t < nr; t += 32) wr_s[t] = __ldg(A.CW + o + rb + t);
#pragma unroll 4
    for (int t = lane; t < nc; t += 32) wc_s[t] = __ldg(A.RW + o + cb + t);
    __syncwarp();
    const int32_t *wr = wr_s, *wc = wc_s;
    if (B + 12 <= WALK_WIN) {
        // The window holds every row and column the walk's moves read (see
        // above): shared memory only.  The index is clamped to the window,
        // which changes nothing for those reads and keeps the lanes' reads
        // past the walk's end inside the warp's own slice.
        const unsigned rmax = unsigned(win - 1);
        ant_walk_warp(
            dr, dc, delta, s, E + B, [&](int r) { return wr[min(unsigned(r - rb), rmax)]; },
            [&](int c) { return wc[min(unsigned(c - cb), rmax)]; }, [&](int r, int c) { A.res[o + r] = c; }, lane);
        return;
    }
    // Grids coarser than the window (k beyond 2^20): outside it, global
    // memory (the walk reads rows in [0, dr] and columns in [dc - 1, s) only).
    ant_walk_warp(
        dr, dc, delta, s, E + B,
        [&](int r) {
            const unsigned t = unsigned(r - rb);
            return t < unsigned(nr) ? wr[t] : __ldg(A.CW + o + r);
        },
        [&](int c) {
            const unsigned t = unsigned(c - cb);
            return t < unsigned(nc) ? wc[t] : __ldg(A.RW + o + c);
        },
        [&](int r, int c) { A.res[o + r] = c; }, lane);
}

// Many short segments (B <= WALK_LANE_B, more of them than the device keeps
// WALK_WARPS warps per SM for): one lane per segment, all steps straight from
// global memory (L2), so that a warp advances 32 walks at once instead of one.
// While every segment's warp is resident the warp's staged walk wins, since a
// lane waits for L2 at most steps.  Whole products, MEASURED lanes -> warps
// (combed strands / random permutations): k = 32768 334 -> 285 / 333 -> 312 us,
// 131072 555 -> 476 / 555 -> 535, 524288 932 -> 853 / 1097 -> 1109 with the
// levels of at most 10000 segments on warps; with all of its levels on warps
// 905 / 1288.
constexpr int WALK_WARPS = 64;

template <int N>
__global__ void __launch_bounds__(256) walk_lanes_kernel(const __grid_constant__ Many<SegArgs, N> M, int nodes)
{
    const SegArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    const long gid = long(blockIdx.x) * blockDim.x + threadIdx.x;
    if (gid >= long(nodes) * A.nseg) return;
    const int nd = int(gid / A.nseg), q = int(gid % A.nseg);
    int o, s;
    node_by_index(nd, A.level, A.k, o, s);
    if (s <= 1) return;
    const int B = A.B;
    const int32_t *T = A.T + size_t(nd) * A.stride * A.stride;
    const int jmin = -((s + B - 1) / B);
    const int E = (jmin + q) * B;
    const int e0 = -(s - 1);
    if (E > s || E + B < e0) return;
    int dr, dc, delta;
    if (E < e0) {
        dr = s - 1;
        dc = 0;
        delta = __ldg(A.CW + o + s - 1) < 0 ? 0 : -1;
    } else {
        const int rlo = max(0, -E), rhi = min(s, s - E);
        if (rlo > rhi) return;
        const int jj = E / B;
        const int ilo = rlo / B, ihi = rhi / B;
        // first grid point of diagonal E with delta >= 0: three probes per
        // round (read together), then halving
        int lo_i = ilo, hi_i = ihi + 1;
        while (hi_i - lo_i > 3) {
            const int w = hi_i - lo_i;
            const int q1 = lo_i + w / 4, q2 = lo_i + w / 2, q3 = lo_i + 3 * w / 4;
            const bool g1 = T[q1 * A.stride + q1 + jj] >= 0, g2 = T[q2 * A.stride + q2 + jj] >= 0,
                       g3 = T[q3 * A.stride + q3 + jj] >= 0;
            if (g1) {
                hi_i = q1;
            } else if (g2) {
                lo_i = q1 + 1;
                hi_i = q2;
            } else if (g3) {
                lo_i = q2 + 1;
                hi_i = q3;
            } else {
                lo_i = q3 + 1;
            }
        }
        while (lo_i < hi_i) {
            const int mid = (lo_i + hi_i) >> 1;
            if (T[mid * A.stride + mid + jj] >= 0) hi_i = mid;
            else lo_i = mid + 1;
        }
        int rstar = rlo;
        int dval = T[ilo * A.stride + ilo + jj]; // delta(rlo, rlo + E): a grid point
        if (lo_i != ilo) {
            dval = T[(lo_i - 1) * A.stride + (lo_i - 1) + jj];
            const int rend = min(lo_i * B, rhi);
            rstar = rhi + 1;
            // Four rows at a time: their words are read before any is tested,
            // so that the reads' latency is paid once per four rows.
            for (int r = (lo_i - 1) * B; r < rend && rstar > rhi; r += 4) {
                int inc[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    inc[u] = r + u < rend ? colinc(A, o, r + u + E, r + u) + rowinc(A, o, r + u, r + u + E + 1) : 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (r + u < rend && rstar > rhi) {
                        dval += inc[u];
                        if (dval >= 0) rstar = r + u + 1;
                    }
                }
            }
        }
        dr = rstar - 1;
        dc = rstar + E;
        if (rstar > rhi || dr < 0 || dc > s) return;
        // dval = delta(r*, r* + E); one row up the point of row r* - 1 leaves
        delta = dval - rowinc(A, o, dr, dc);
    }
    ant_walk(
        dr, dc, delta, s, E + B, [&](int r) { return __ldg(A.CW + o + r); },
        [&](int c) { return __ldg(A.RW + o + c); }, [&](int r, int c) { A.res[o + r] = c; });
}

// ---------------------------------------------------------------------------
// staggered multiplication around the steady ant
// ---------------------------------------------------------------------------
// Pc = inverse of P (p entries) and Qc = inverse of Q (q entries), one
// launch; an entry outside [0, n) raises *bad.  A column that no entry hits
// keeps whatever Pc / Qc held: slice_count_kernel detects it (a repeat in
// the input leaves some column unhit).
struct InverseArgs {
    const int32_t *P;
    int32_t *Pc;
    const int32_t *Q;
    int32_t *Qc;
    int p, q;
    int32_t *bad;
};
template <int N>
__global__ void __launch_bounds__(256) inverse_pair_kernel(const __grid_constant__ Many<InverseArgs, N> M)
{
    const InverseArgs &A = M.of[blockIdx.z];
    const int32_t *P = A.P, *Q = A.Q;
    int32_t *Pc = A.Pc, *Qc = A.Qc, *bad = A.bad;
    const int p = A.p, q = A.q;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < p + q; t += gridDim.x * blockDim.x) {
        const bool in_p = t < p;
        const int i = in_p ? t : t - p, n = in_p ? p : q;
        const int c = in_p ? P[i] : Q[i];
        if (c < 0 || c >= n) *bad = 1;
        else (in_p ? Pc : Qc)[c] = i;
    }
}

// Slices of P (rows whose column lies in [c0, c0+k), row order) and of Q
// (columns whose row lies in [r0, r0+k), column order) by one stable
// compaction each, using the level-0 scan machinery over max(p, q) entries.
struct SliceArgs {
    const int32_t *P_r2c;
    const int32_t *Q_c2r;
    const int32_t *P_c2r, *Q_r2c; // for the permutation check
    int p, q, k, c0, r0;
    int32_t *p_red;  // level-0 P (r2c, local)
    int32_t *q_red;  // level-0 Q (c2r, local)
    int32_t *map_row, *map_col;
    int32_t *bsumP, *bsumQ;
    int n; // max(p, q)
    int32_t *bad;
    int32_t *fan_cnt; // counts for fan_kernel (null: not used), of lc levels
    int lc;
};

__device__ __forceinline__ void slice_flags(const SliceArgs &A, int i, int &fp, int &fq)
{
    fp = i < A.p && A.P_r2c[i] >= A.c0 && A.P_r2c[i] < A.c0 + A.k;
    fq = i < A.q && A.Q_c2r[i] >= A.r0 && A.Q_c2r[i] < A.r0 + A.k;
}

template <int N>
__global__ void __launch_bounds__(256) slice_count_kernel(const __grid_constant__ Many<SliceArgs, N> M)
{
    const SliceArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    constexpr int PER = SCAN_BS / 256;
    const int base = blockIdx.x * SCAN_BS + threadIdx.x;
    int cp = 0, cq = 0;
    bool wrong = false;
    int rp[PER], rq[PER]; // all reads of a kind in flight at once
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * 256;
        rp[j] = i < A.p ? A.P_c2r[i] : 0;
        rq[j] = i < A.q ? A.Q_c2r[i] : 0;
    }
    // Column i of P (row i of Q) must be the image of the row its
    // inverse names: otherwise no entry hit it and the input repeats one.
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j * 256;
        if (i < A.p) wrong |= unsigned(rp[j]) >= unsigned(A.p) || A.P_r2c[rp[j]] != i;
        if (i < A.q) wrong |= unsigned(rq[j]) >= unsigned(A.q) || A.Q_r2c[rq[j]] != i;
        int fp, fq;
        slice_flags(A, i, fp, fq);
        cp += fp;
        cq += fq;
    }
    if (wrong) *A.bad = 1;
    __shared__ int sp[8], sq[8];
    for (int off = 16; off; off >>= 1) {
        cp += __shfl_xor_sync(FULL_MASK, cp, off);
        cq += __shfl_xor_sync(FULL_MASK, cq, off);
    }
    if ((threadIdx.x & 31) == 0) {
        sp[threadIdx.x >> 5] = cp;
        sq[threadIdx.x >> 5] = cq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int tp = 0, tq = 0;
        for (int w = 0; w < 8; ++w) {
            tp += sp[w];
            tq += sq[w];
        }
        A.bsumP[blockIdx.x] = tp;
        A.bsumQ[blockIdx.x] = tq;
    }
}

template <int N>
__global__ void __launch_bounds__(256) slice_write_kernel(const __grid_constant__ Many<SliceArgs, N> M)
{
    const SliceArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    constexpr int PER = SCAN_BS / 256;
    const int base = blockIdx.x * SCAN_BS + threadIdx.x * PER;
    int fp[PER], fq[PER], cp = 0, cq = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j;
        if (i < A.n) slice_flags(A, i, fp[j], fq[j]);
        else fp[j] = fq[j] = 0;
        cp += fp[j];
        cq += fq[j];
    }
    int xp = cp, xq = cq;
    for (int off = 1; off < 32; off <<= 1) {
        int yp = __shfl_up_sync(FULL_MASK, xp, off), yq = __shfl_up_sync(FULL_MASK, xq, off);
        if ((threadIdx.x & 31) >= off) {
            xp += yp;
            xq += yq;
        }
    }
    __shared__ int wp[8], wq[8], before[2];
    if ((threadIdx.x & 31) == 31) {
        wp[threadIdx.x >> 5] = xp;
        wq[threadIdx.x >> 5] = xq;
    }
    int op, oq;
    if (gridDim.x <= SLICE_DIRECT) { // the block adds its predecessors' counts itself
        int bp = 0, bq = 0;
        for (unsigned t = threadIdx.x; t < blockIdx.x; t += 256) {
            bp += A.bsumP[t];
            bq += A.bsumQ[t];
        }
        if (threadIdx.x < 2) before[threadIdx.x] = 0;
        __syncthreads();
        bp = __reduce_add_sync(FULL_MASK, bp);
        bq = __reduce_add_sync(FULL_MASK, bq);
        if ((threadIdx.x & 31) == 0 && (bp | bq)) {
            atomicAdd(before, bp);
            atomicAdd(before + 1, bq);
        }
        __syncthreads();
        op = before[0];
        oq = before[1];
    } else {
        __syncthreads();
        op = A.bsumP[blockIdx.x];
        oq = A.bsumQ[blockIdx.x];
    }
    for (int w = 0; w < (threadIdx.x >> 5); ++w) {
        op += wp[w];
        oq += wq[w];
    }
    op += xp - cp;
    oq += xq - cq;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = base + j;
        if (fp[j]) {
            A.map_row[op] = i;
            const int v = A.P_r2c[i] - A.c0;
            A.p_red[op] = v;
            if (A.fan_cnt) atomicAdd(A.fan_cnt + ((op / FAN_TILE) << A.lc) + leaf_of(v, A.lc, A.k), 1);
            ++op;
        }
        if (fq[j]) {
            A.map_col[oq] = i;
            const int v = A.Q_c2r[i] - A.r0;
            A.q_red[oq] = v;
            if (A.fan_cnt)
                atomicAdd(A.fan_cnt + ((fan_tiles(A.k) + oq / FAN_TILE) << A.lc) + leaf_of(v, A.lc, A.k), 1);
            ++oq;
        }
    }
}

// ---------------------------------------------------------------------------
// every level's partition at once
//
// An entry's place at level l is its node's start plus the number of earlier
// entries in the same node, and its node follows from its value alone (nodes
// are the same ranges of values as of places).  So no level needs the one
// above: slice_write counts the entries of every (tile, node of level lc);
// here a block of one tile adds the earlier tiles' counts and its own warps'
// into prefix sums over the nodes of level lc, of which the count of any
// level's node before a warp is a difference of two, and __match_any_sync
// ranks a warp's entries within their node, level by level.  No block waits
// for another.  At an overlap of 32768 (5 levels) the level-by-level
// partitions took 59 us, waiting for one another; this takes 6 (MEASURED).
// The counts grow with the tiles times the nodes, and the sums take 132 bytes of
// shared memory a node, so products of more than FAN_LEAVES nodes keep the
// level-by-level form (256 nodes instead of 128: 262144 569 -> 478 us).
// ---------------------------------------------------------------------------
struct FanArgs {
    const int32_t *in; // level 0: P then Q (k entries each)
    int32_t *out;      // level lc, node-local: P then Q
    int32_t *maps;     // level l at maps + 2 k l: P's map, then Q's (levels 1 to lc)
    const int32_t *cnt; // (P or Q, tile, node of level lc)
    int k, lc;
    const int32_t *bad;
};

template <int N>
__global__ void __launch_bounds__(FAN_TILE) fan_kernel(const __grid_constant__ Many<FanArgs, N> M)
{
    const FanArgs &A = M.of[blockIdx.z];
    if (*A.bad) return;
    __shared__ int sums[FAN_TILE / 32][FAN_LEAVES + 1]; // per warp: entries before it, by node, then prefix sums
    __shared__ int before[FAN_LEAVES];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int side = blockIdx.y, tile = blockIdx.x, tiles = gridDim.x;
    const int nl = 1 << A.lc;
    const int i = tile * FAN_TILE + threadIdx.x;
    const bool here = i < A.k;
    const int v = here ? A.in[size_t(side) * A.k + i] : 0;
    const int leaf = here ? leaf_of(v, A.lc, A.k) : -1;
    for (int t = lane; t <= nl; t += 32) sums[warp][t] = 0;
    if (threadIdx.x < nl) before[threadIdx.x] = 0;
    __syncthreads();
    {
        const unsigned same = __match_any_sync(FULL_MASK, leaf);
        if (here && lane == __ffs(same) - 1) sums[warp][leaf] = __popc(same);
        const int32_t *cnt = A.cnt + ((size_t(side) * tiles) << A.lc);
        int sum = 0;
        for (int t = threadIdx.x >> A.lc; t < tile; t += FAN_TILE >> A.lc)
            sum += cnt[(size_t(t) << A.lc) + (threadIdx.x & (nl - 1))];
        if (sum) atomicAdd(before + (threadIdx.x & (nl - 1)), sum);
    }
    __syncthreads();
    if (threadIdx.x < nl) {
        int run = before[threadIdx.x];
        for (int w = 0; w < FAN_TILE / 32; ++w) {
            const int c = sums[w][threadIdx.x];
            sums[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int base = 0, carry = 0; base <= nl; base += 32) { // exclusive prefix sums of the warp's row
        const int t = base + lane, c = t < nl ? sums[warp][t] : 0;
        int x = c;
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(FULL_MASK, x, off);
            if (lane >= off) x += y;
        }
        if (t <= nl) sums[warp][t] = carry + x - c;
        carry += __shfl_sync(FULL_MASK, x, 31);
    }
    __syncwarp();
    int o = 0, s = A.k, local = i; // the entry's node of level l and its place there
    for (int l = 1; l <= A.lc; ++l) {
        const int h = s >> 1;
        if (v < o + h) {
            s = h;
        } else {
            o += h;
            s -= h;
        }
        const int nd = leaf >> (A.lc - l);
        const unsigned same = __match_any_sync(FULL_MASK, nd);
        if (here) {
            const int first = nd << (A.lc - l);
            const int place = sums[warp][first + (1 << (A.lc - l))] - sums[warp][first] +
                              __popc(same & ((1u << lane) - 1));
            A.maps[size_t(2) * A.k * l + size_t(side) * A.k + o + place] = local;
            local = place;
        }
    }
    if (here) A.out[size_t(side) * A.k + o + local] = v - o;
}

struct AssembleArgs {
    const int32_t *P_r2c, *P_c2r, *Q_r2c;
    const int32_t *res; // steady-ant product (r2c, k x k)
    const int32_t *map_row, *map_col;
    int32_t *out;       // product r2c
    int p, q, k;
    bool row_glue;
    const int32_t *bad;
    uint32_t *status;   // device status word: DEV_ERR_INPUT when the product failed
};

template <int N>
__global__ void __launch_bounds__(256) assemble_kernel(const __grid_constant__ Many<AssembleArgs, N> M)
{
    const AssembleArgs &A = M.of[blockIdx.z];
    if (*A.bad) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(A.status, DEV_ERR_INPUT);
        return;
    }
    const int tot = A.p + A.q; // work items: k reduced points + p columns + q rows
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tot + A.k; t += gridDim.x * blockDim.x) {
        if (t < A.k) {
            const int cur_row = A.map_row[t], cur_col = A.map_col[A.res[t]];
            if (A.row_glue) A.out[A.q - A.k + cur_row] = cur_col;
            else A.out[cur_row] = cur_col + A.p - A.k;
        } else if (t < A.k + A.p) {
            const int j = t - A.k; // column j of P
            const int row = A.P_c2r[j];
            if (A.row_glue) {
                if (j >= A.k) A.out[row + A.q - A.k] = j + A.q - A.k;
            } else {
                if (j < A.p - A.k) A.out[row] = j;
            }
        } else {
            const int i = t - A.k - A.p; // row i of Q
            const int col = A.Q_r2c[i];
            if (A.row_glue) {
                if (i < A.q - A.k) A.out[i] = col;
            } else {
                if (i >= A.k) A.out[i - A.k + A.p] = col - A.k + A.p;
            }
        }
    }
}

__global__ void __launch_bounds__(256) direct_sum_kernel(const int32_t *P, const int32_t *Q, int p, int q, bool row_glue,
                                                         int32_t *out)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < p + q; t += gridDim.x * blockDim.x) {
        if (t < p) {
            out[row_glue ? t + q : t] = row_glue ? P[t] + q : P[t];
        } else {
            const int i = t - p;
            out[row_glue ? i : i + p] = row_glue ? Q[i] : Q[i] + p;
        }
    }
}

inline int blocks_for(long n, int threads) { return int(std::min<long>((n + threads - 1) / threads, 148L * 16)); }


} // namespace

// Grid spacing and table stride of the concurrent walk at `level` (nodes of at
// most smax entries).
// Grid spacing of a level's delta tables: at most WALK_GMAX lines per node and
// about 2^21 table entries per level over all its nodes (the tables are
// rebuilt every level, and a segment walk of B steps is cheap in shared memory).
static void walk_grid(int k, int level, int &B, int &stride)
{
    int smax = k;
    for (int d = 0; d < level; ++d) smax = smax - (smax >> 1);
    const double per_node = double(1 << 21) / double(1u << std::min(level, 30));
    const int gmax = std::max(1, std::min(WALK_GMAX, int(std::sqrt(per_node)) - 1));
    B = std::max(WALK_BMIN, (smax + gmax - 1) / gmax);
    stride = smax / B + 1;
}

// First level whose nodes are at most `cutoff` entries.
static int cutoff_level(int k, int cutoff)
{
    int lc = 0;
    for (int s = k; s > cutoff; s = s - (s >> 1)) ++lc;
    return lc;
}

static size_t table_ints(int k, int cutoff)
{
    size_t best = 0;
    const int lc = cutoff_level(k, cutoff);
    for (int l = 0; l < lc; ++l) {
        int B, stride;
        walk_grid(k, l, B, stride);
        best = std::max(best, (size_t(1) << l) * size_t(stride) * size_t(stride));
    }
    return best;
}

slcs_status braid_workspace_bytes(int p, int q, int k, int cutoff, size_t *bytes)
{
    const int n = std::max(p, q);
    const size_t kk = size_t(std::max(k, 1));
    if (cutoff <= 0) cutoff = NODE_MAX;
    if (cutoff > NODE_MAX) cutoff = NODE_MAX;
    const int lc = cutoff_level(k, cutoff);
    size_t b = 0;
    b += 4 * table_ints(k, cutoff) * sizeof(int32_t) + 512; // delta tables (hi, lo), two buffers
    b += 4 * kk * sizeof(int32_t);                         // P/Q ping-pong
    b += 2 * kk * size_t(lc + 2) * sizeof(int32_t);    // maps per level
    b += kk * size_t(lc + 2) * sizeof(int32_t);        // results per level
    b += 2 * kk * sizeof(int32_t);                         // row and column words
    b += 2 * size_t(std::max(n, k)) * sizeof(int32_t);     // scans
    b += 2 * (size_t(std::max(n, k)) / SCAN_BS + 2) * sizeof(int32_t);
    b += size_t(p) * sizeof(int32_t) + size_t(q) * sizeof(int32_t); // inverses
    b += 2 * kk * sizeof(int32_t);                         // map_row, map_col
    b += 64 * 256 + 256;                                    // alignment slack, flag
    b += size_t(2 * fan_tiles(std::min(k, FAN_LEAVES * NODE_MAX))) * FAN_LEAVES * sizeof(int32_t); // the fan's counts
    b += size_t(lc + 1) * ((size_t(std::max(k, 1)) + 256 * PART_PER - 1) / (256 * PART_PER)) * 16 + 512; // partition tiles
    *bytes = (b + 255) / 256 * 256;
    return SLCS_OK;
}

namespace {

// Products jobs[0..count) of one overlap k >= 1, each with ws_bytes of
// workspace one after another: every step of them in one launch.
template <int N>
slcs_status launch_many(const BraidJob *jobs, int count, int k, bool row_glue, int cutoff, void *ws, size_t ws_bytes,
                        cudaStream_t st)
{
    if (cutoff <= 0 || cutoff > NODE_MAX) cutoff = NODE_MAX;
    int pmax = 0, qmax = 0; // one layout for all: of the largest sizes
    for (int z = 0; z < count; ++z) {
        pmax = std::max(pmax, jobs[z].p);
        qmax = std::max(qmax, jobs[z].q);
    }
    const int n = std::max(pmax, qmax);
    const int lc = cutoff_level(k, cutoff); // first level whose nodes fit a block
    const size_t kk = size_t(k);
    char *cur = static_cast<char *>(ws);
    auto take = [&](size_t bytes) {
        char *r = cur;
        cur += (bytes + 255) / 256 * 256;
        return r;
    };
    auto take_ints = [&](size_t n) { return reinterpret_cast<int32_t *>(take(n * sizeof(int32_t))); };
    // The first product's arrays; another's lie a multiple of ws_bytes further.
    int32_t *PQ0 = take_ints(4 * kk);
    int32_t *maps0 = take_ints(2 * kk * size_t(lc + 2));
    int32_t *res0 = take_ints(kk * size_t(lc + 2));
    int32_t *C0 = take_ints(kk), *Rr0 = take_ints(kk);
    const size_t nscan = size_t(std::max(n, k));
    int32_t *scanP0 = take_ints(nscan), *scanQ0 = take_ints(nscan);
    const int nbs = int((nscan + SCAN_BS - 1) / SCAN_BS);
    int32_t *bsP0 = take_ints(size_t(nbs + 1)), *bsQ0 = take_ints(size_t(nbs + 1));
    int32_t *P_c2r0 = take_ints(size_t(pmax)), *Q_c2r0 = take_ints(size_t(qmax));
    int32_t *map_row0 = take_ints(kk), *map_col0 = take_ints(kk);
    // Error flag, then the partitions' tile words (one per tile and level),
    // their done flags, the ticket and the levels' done counts, or the fan's
    // counts: zeroed by one memset.
    const int part_bs = part_threads(k) * PART_PER;
    const int kb = int((kk + part_bs - 1) / part_bs);
    const bool fan = lc > 0 && lc < 31 && (1 << lc) <= FAN_LEAVES;
    const size_t tile_words = fan ? 0 : size_t(lc) * size_t(kb);
    const size_t fan_words = fan ? size_t(2 * fan_tiles(k)) << lc : 0;
    const size_t sync_bytes = 256 + tile_words * 8 + tile_words * 4 + 256 + tile_words * 4 + fan_words * 4;
    char *sync0 = take(sync_bytes);
    const size_t tints = table_ints(k, cutoff);
    // Two table buffers, each a level's hi then lo counts; levels alternate.
    int32_t *tabs0 = take_ints(4 * tints);
    if (size_t(cur - static_cast<char *>(ws)) > ws_bytes) return fail(SLCS_ERR_ALLOC, "braid workspace too small");

    const unsigned nz = unsigned(count);
    auto at = [&](auto *p, int z) { return reinterpret_cast<decltype(p)>(reinterpret_cast<char *>(p) + ws_bytes * size_t(z)); };
    auto bad_of = [&](int z) { return reinterpret_cast<int32_t *>(at(sync0, z)); };
    // Level l's tables: entries of each of the two, and place in the buffer
    // of its parity.
    auto level_tables = [&](int l, size_t *tentries) {
        int B, stride;
        walk_grid(k, l, B, stride);
        *tentries = (size_t(1) << l) * size_t(stride) * size_t(stride);
        return tabs0 + size_t(l & 1) * 2 * tints;
    };
    auto zero = [&](void *p, size_t bytes) {
        if (count > 1 && ws_bytes < (size_t(1) << 30)) // within the pitch limit
            return cudaMemset2DAsync(p, ws_bytes, 0, bytes, size_t(count), st);
        cudaError_t e = cudaSuccess;
        for (int z = 0; z < count && e == cudaSuccess; ++z)
            e = cudaMemsetAsync(static_cast<char *>(p) + ws_bytes * size_t(z), 0, bytes, st);
        return e;
    };
    SLCS_CUDA(zero(sync0, sync_bytes));
    if (lc > 0) { // the deepest level's tables; each level's glue clears the next level's
        size_t te = 0;
        int32_t *t0 = level_tables(lc - 1, &te);
        SLCS_CUDA(zero(t0, 2 * te * sizeof(int32_t)));
    }
    {
        Many<InverseArgs, N> I{};
        Many<SliceArgs, N> S{};
        Many<BsumArgs, N> U{};
        for (int z = 0; z < count; ++z) {
            const BraidJob &j = jobs[z];
            int32_t *P_c2r = at(P_c2r0, z), *Q_c2r = at(Q_c2r0, z), *PQ = at(PQ0, z);
            I.of[z] = InverseArgs{j.P, P_c2r, j.Q, Q_c2r, j.p, j.q, bad_of(z)};
            int32_t *fan_cnt = reinterpret_cast<int32_t *>(at(sync0, z) + 512);
            S.of[z] = SliceArgs{j.P, Q_c2r, P_c2r, j.Q, j.p, j.q, k, row_glue ? 0 : j.p - k, row_glue ? j.q - k : 0,
                                PQ, PQ + kk, at(map_row0, z), at(map_col0, z), at(bsP0, z), at(bsQ0, z),
                                std::max(j.p, j.q), bad_of(z), fan ? fan_cnt : nullptr, lc};
            U.of[z] = BsumArgs{at(bsP0, z), at(bsQ0, z)};
        }
        inverse_pair_kernel<N><<<dim3(unsigned(blocks_for(long(pmax) + qmax, 256)), 1, nz), 256, 0, st>>>(I);
        slice_count_kernel<N><<<dim3(unsigned(nbs), 1, nz), 256, 0, st>>>(S);
        if (nbs > SLICE_DIRECT) part_bsum_kernel<N><<<dim3(1, 1, nz), 1024, 0, st>>>(U, nbs);
        slice_write_kernel<N><<<dim3(unsigned(nbs), 1, nz), 256, 0, st>>>(S);
    }
    // Levels above the cutoff: device-wide partitions, all in one launch
    // (level by level, level l reads the even or odd pair of PQ's arrays and
    // writes the other).
    int32_t *cur0 = PQ0; // P then Q of level lc
    if (fan) {
        Many<FanArgs, N> G{};
        for (int z = 0; z < count; ++z) {
            int32_t *PQ = at(PQ0, z);
            G.of[z] = FanArgs{PQ, PQ + 2 * kk, at(maps0, z), reinterpret_cast<int32_t *>(at(sync0, z) + 512), k, lc,
                              bad_of(z)};
        }
        fan_kernel<N><<<dim3(unsigned(fan_tiles(k)), 2, nz), FAN_TILE, 0, st>>>(G);
        cur0 = PQ0 + 2 * kk;
    } else if (lc > 0) {
        Many<PartAllArgs, N> G{};
        for (int z = 0; z < count; ++z) {
            char *sync_area = at(sync0, z);
            int32_t *ticket = reinterpret_cast<int32_t *>(sync_area + 256 + tile_words * 12);
            G.of[z] = PartAllArgs{at(PQ0, z), at(maps0, z), at(scanP0, z), at(scanQ0, z), k, lc, kb,
                                  (k & (k - 1)) == 0, reinterpret_cast<unsigned long long *>(sync_area + 256),
                                  reinterpret_cast<int32_t *>(sync_area + 256 + tile_words * 8), ticket,
                                  ticket + 1, // lc counts (lc <= 31 fits these 256 bytes)
                                  reinterpret_cast<int32_t *>(sync_area + 256 + tile_words * 12 + 256), bad_of(z),
                                  device_status_word()};
        }
        const int threads = part_threads(k);
        const long grid = std::min<long>(long(lc) * kb, long(sm_count()) * (2048 / threads));
        if (threads == 1024) part_levels_kernel<1024, N><<<dim3(unsigned(grid), 1, nz), 1024, 0, st>>>(G);
        else part_levels_kernel<256, N><<<dim3(unsigned(grid), 1, nz), 256, 0, st>>>(G);
        if (lc & 1) cur0 = PQ0 + 2 * kk;
    }
    // Nodes of level lc: one block each.
    {
        int smax = k; // largest node of level lc (floor/ceil halving)
        for (int l = 0; l < lc; ++l) smax = smax - (smax >> 1);
        Many<NodeArgs, N> G{};
        for (int z = 0; z < count; ++z)
            G.of[z] = NodeArgs{at(cur0, z), at(cur0, z) + kk, at(res0, z) + kk * size_t(lc), k, lc, bad_of(z)};
        const int warps = node_warps(smax);
        const dim3 grid(1u << lc, 1, nz);
        if (warps == 1) node_kernel<true, N><<<grid, 32, 0, st>>>(G);
        else node_kernel<false, N><<<grid, warps * 32, 0, st>>>(G);
    }
    // Levels above: glue, union, walk.
    for (int l = lc - 1; l >= 0; --l) {
        int B, stride;
        walk_grid(k, l, B, stride);
        const int nodes = 1 << l;
        int smax = k;
        for (int d = 0; d < l; ++d) smax = smax - (smax >> 1);
        const int nseg = 2 * ((smax + B - 1) / B) + 2;
        // hi and lo counts of the level side by side (zeroed by the memset
        // above or by the glue one level down), filled by the glue as it
        // places the points
        size_t tentries = 0, next_entries = 0;
        int32_t *tab0 = level_tables(l, &tentries);
        int32_t *next0 = l > 0 ? level_tables(l - 1, &next_entries) : nullptr;
        Many<GlueArgs, N> G{};
        Many<TableArgs, N> TA{};
        Many<SegArgs, N> SA{};
        for (int z = 0; z < count; ++z) {
            int32_t *C = at(C0, z), *Rr = at(Rr0, z), *tab = at(tab0, z), *lo = tab + tentries;
            int32_t *maps = at(maps0, z) + 2 * kk * size_t(l + 1), *res = at(res0, z) + kk * size_t(l);
            G.of[z] = GlueArgs{res + kk, maps, maps + kk, C, Rr, res, k, l, bad_of(z), tab, lo, B, stride,
                               next0 ? at(next0, z) : nullptr, (long long)(2 * next_entries)};
            TA.of[z] = TableArgs{C, tab, lo, k, l, B, stride, bad_of(z)};
            SA.of[z] = SegArgs{C, Rr, tab, res, k, l, B, stride, nseg, bad_of(z)};
        }
        glue_kernel<N><<<dim3(unsigned(blocks_for(k, 256)), 1, nz), 256, 0, st>>>(G);
        if (size_t(stride) * stride <= size_t(SMALL_TABLE)) {
            table_small_kernel<N><<<dim3(unsigned(nodes), 1, nz), 256, 0, st>>>(TA, nodes);
        } else {
            const int rows = nodes * stride;
            table_rows_kernel<N><<<dim3(unsigned((long(rows) * 32 + 255) / 256), 1, nz), 256, 0, st>>>(TA, nodes);
            if (stride <= TCOL_SMALL_ROWS)
                table_cols_kernel<32, 8, N><<<dim3(unsigned(nodes * ((stride + 31) / 32)), 1, nz), 256, 0, st>>>(TA, nodes);
            else
                table_cols_kernel<4, 64, N><<<dim3(unsigned(nodes * ((stride + 3) / 4)), 1, nz), 256, 0, st>>>(TA, nodes);
        }
        const long warps = long(nodes) * nseg;
        if (B <= WALK_LANE_B && warps * count > long(WALK_WARPS) * sm_count()) {
            walk_lanes_kernel<N><<<dim3(unsigned((warps + 255) / 256), 1, nz), 256, 0, st>>>(SA, nodes);
        } else {
            const size_t wsm = size_t(4) * 2 * (B <= WALK_ROW_B ? B : walk_win(B)) * sizeof(int32_t);
            walk_segments_kernel<N><<<dim3(unsigned((warps * 32 + 127) / 128), 1, nz), 128, wsm, st>>>(SA, nodes);
        }
    }
    Many<AssembleArgs, N> A{};
    for (int z = 0; z < count; ++z) {
        const BraidJob &j = jobs[z];
        A.of[z] = AssembleArgs{j.P, at(P_c2r0, z), j.Q, at(res0, z), at(map_row0, z), at(map_col0, z), j.out, j.p, j.q,
                               k, row_glue, bad_of(z), device_status_word()};
    }
    assemble_kernel<N><<<dim3(unsigned(blocks_for(long(pmax) + qmax + k, 256)), 1, nz), 256, 0, st>>>(A);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

} // namespace

slcs_status launch_braids(const BraidJob *jobs, int count, int k, bool row_glue, int cutoff, void *ws, size_t ws_bytes,
                          cudaStream_t st)
{
    if (k == 0) {
        for (int z = 0; z < count; ++z) {
            const BraidJob &j = jobs[z];
            direct_sum_kernel<<<blocks_for(j.p + j.q, 256), 256, 0, st>>>(j.P, j.Q, j.p, j.q, row_glue, j.out);
        }
        SLCS_CUDA(cudaGetLastError());
        return SLCS_OK;
    }
    if (count == 1) return launch_many<1>(jobs, 1, k, row_glue, cutoff, ws, ws_bytes, st);
    return launch_many<BRAID_MANY>(jobs, count, k, row_glue, cutoff, ws, ws_bytes, st);
}

} // namespace slcs
