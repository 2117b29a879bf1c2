// couples.cu -- two pairs per register: the short pairs of a batch.
//
// A couple of pairs (A, B) is combed together, one instruction for two cells
// (cell16, cell.cuh).
//
// A warp combs a bundle: couples side by side, each on as many lanes as its
// rows need at TM rows per lane, all started in the same step and of about the
// same length, so that every lane of the warp runs the same straight line from
// the first step to the last.  Lanes before or past their couple's columns
// comb masked ones.  The plan deals the bundles out to the SM sub-partitions
// (one block per SM; warp w of a block runs on sub-partition w % 4), whose
// integer pipe bounds the comb; up to COUPLE_DEPTH warps of a block take a
// sub-partition's bundles longest first.  (Claimed by all warps from one
// counter, the longest bundles met on the SMs that started first: the busiest
// sub-partition issued 1.85 times the average.)
// (The design before, couples streamed through segments one after another, saved
// the fill of a couple but had every lane change couples in a step of its own:
// divergent code every other step, and a scoreboard that makes a lane wait for
// what its neighbour loaded a step ago.  It combed the 20,000 reads in 202 us.)
//
// A warp expands the columns of its bundle into shared memory first (ready
// registers, masked where a pair has no column), replaces their strands there
// as they leave the last lane, and writes them out after the last step, so
// that a step knows nothing of pairs, ids, lengths or alignment and waits for
// no global memory.  Couples too long for that are staged in global memory the
// same way by two more launches, pack_couples_kernel and unpack_couples_kernel.
// (Staging every couple so took 139 us: 25 in those launches, and steps waiting
// for L2.)
#include <algorithm>
#include <climits>

#include "cell.cuh"
#include "couples.cuh"
#include "occupancy.cuh"

namespace slcs {

namespace {

// Symbols c .. c + 3 of one pair as two packed words' low halves would hold
// them: s[0..3], `mask` past n.  Whole-word loads where they are aligned.
__device__ __forceinline__ void four_symbols(const uint8_t *p, int c, int n, uint32_t mask, uint32_t (&s)[4])
{
    if (c + 4 <= n && (reinterpret_cast<uintptr_t>(p + c) & 3) == 0) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(p + c));
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = (w >> (8 * j)) & 0xFFu;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = c + j < n ? uint32_t(__ldg(p + c + j)) : mask;
    }
}

// Symbols of rows or columns 4 q .. 4 q + 3 of both pairs.
__device__ __forceinline__ uint4 couple_symbols(const uint8_t *pa, int na, const uint8_t *pb, int nb, int q, uint32_t mask)
{
    uint32_t lo[4], hi[4];
    four_symbols(pa, 4 * q, na, mask & 0xFFFFu, lo);
    four_symbols(pb, 4 * q, nb, mask & 0xFFFFu, hi);
    return make_uint4(lo[0] | hi[0] << 16, lo[1] | hi[1] << 16, lo[2] | hi[2] << 16, lo[3] | hi[3] << 16);
}
// h strands of rows 4 q .. (id + 1: the rows left) and v strands of columns 4 q ..
__device__ __forceinline__ uint4 couple_h(const CoupleDev &C, int q)
{
    const int ra = C.a.m - 4 * q, rb = C.b.m - 4 * q;
    uint32_t x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = uint32_t(max(ra - j, 0)) | (uint32_t(max(rb - j, 0)) << 16);
    return make_uint4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ uint4 couple_v(const CoupleDev &C, int q)
{
    uint32_t x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = 4 * q + j;
        x[j] = (c < C.a.n ? uint32_t(C.a.m + c + 1) : 0x7FFFu) | ((c < C.b.n ? uint32_t(C.b.m + c + 1) : 0x7FFFu) << 16);
    }
    return make_uint4(x[0], x[1], x[2], x[3]);
}

// One warp per staged couple, four rows or columns per lane and round.
constexpr int COUPLES_PER_BLOCK = 4;
__global__ void __launch_bounds__(32 * COUPLES_PER_BLOCK) pack_couples_kernel(const CouplesLaunch L)
{
    const int k = blockIdx.x * COUPLES_PER_BLOCK + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= L.nstaged) return;
    const CoupleDev C = L.couples[k];
    uint4 *sym = L.stage + C.off, *h = sym + C.rows / 4;
    for (int q = lane; q < C.rows / 4; q += 32) {
        sym[q] = couple_symbols(L.a_blob + C.a.a_off, C.a.m, L.a_blob + C.b.a_off, C.b.m, q, MASKED_ROW16);
        h[q] = couple_h(C, q);
    }
    sym = h + C.rows / 4;
    uint4 *v = sym + C.nb;
    for (int q = lane; q < C.nb; q += 32) {
        sym[q] = couple_symbols(L.b_blob + C.a.b_off, C.a.n, L.b_blob + C.b.b_off, C.b.n, q, MASKED_COLUMN16);
        v[q] = couple_v(C, q);
    }
}

// Strand x (id + 1) of one pair to entry i of its output.
__device__ __forceinline__ void put(const CouplesLaunch &L, int64_t i, uint32_t x)
{
    if (L.out16) L.out16[i] = int16_t(int(x) - 1);
    else L.out[i] = int32_t(x) - 1;
}
__device__ __forceinline__ void put_h(const CouplesLaunch &L, const CoupleDev &C, int r, uint32_t x)
{
    if (r < C.a.m) put(L, C.a.out_off + C.a.m - 1 - r, x & 0xFFFFu);
    if (r < C.b.m) put(L, C.b.out_off + C.b.m - 1 - r, x >> 16);
}
__device__ __forceinline__ void put_v(const CouplesLaunch &L, const CoupleDev &C, int c, uint32_t x)
{
    if (c < C.a.n) put(L, C.a.out_off + C.a.m + c, x & 0xFFFFu);
    if (c < C.b.n) put(L, C.b.out_off + C.b.m + c, x >> 16);
}

__global__ void __launch_bounds__(32 * COUPLES_PER_BLOCK) unpack_couples_kernel(const CouplesLaunch L)
{
    const int k = blockIdx.x * COUPLES_PER_BLOCK + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= L.nstaged) return;
    const CoupleDev C = L.couples[k];
    const uint32_t *h = reinterpret_cast<const uint32_t *>(L.stage + C.off) + C.rows;
    const uint32_t *v = h + C.rows + 4 * C.nb;
    for (int r = lane; r < C.rows; r += 32) put_h(L, C, r, h[r]);
#pragma unroll 4
    for (int c = lane; c < 4 * C.nb; c += 32) put_v(L, C, c, v[c]);
}

__device__ __forceinline__ uint4 ld_if(bool on, const uint4 *p, uint4 x)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+r"(x.x), "+r"(x.y), "+r"(x.z), "+r"(x.w)
                 : "l"(p), "r"(int(on))
                 : "memory");
    return x;
}
__device__ __forceinline__ void st_shared_if(bool on, uint4 *p, const uint32_t (&x)[4])
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.shared.v4.u32 [%1], {%2, %3, %4, %5};\n\t}"
                 ::"r"(int(on)), "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(x[0]), "r"(x[1]),
                 "r"(x[2]), "r"(x[3])
                 : "memory");
}
__device__ __forceinline__ void st_if(bool on, uint4 *p, const uint32_t (&x)[4])
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %0, 0;\n\t@q st.global.v4.u32 [%1], {%2, %3, %4, %5};\n\t}"
                 ::"r"(int(on)), "l"(p), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3])
                 : "memory");
}

template <int TM>
__device__ __forceinline__ void split(const uint4 &x, uint32_t (&r)[TM], int q)
{
    r[4 * q] = x.x, r[4 * q + 1] = x.y, r[4 * q + 2] = x.z, r[4 * q + 3] = x.w;
}

// A step of one lane: its block's symbols are c, its strands come from the lane
// before it, or (the first lane of a couple) are f.
template <int TM>
__device__ __forceinline__ void couple_step(const uint4 &c, const uint4 &f, bool first, const uint32_t (&ap)[TM],
                                            uint32_t (&hp)[TM], uint32_t (&vc)[4])
{
    uint32_t vi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) vi[j] = __shfl_up_sync(FULL_MASK, vc[j], 1);
    vi[0] = first ? f.x : vi[0], vi[1] = first ? f.y : vi[1];
    vi[2] = first ? f.z : vi[2], vi[3] = first ? f.w : vi[3];
    const uint32_t bp[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t v = vi[j];
#pragma unroll
        for (int r = 0; r < TM; ++r) cell16(ap[r], bp[j], hp[r], v);
        vc[j] = v;
    }
}

// Bundles whose columns are in shared memory.
struct BundleColumns { // of one warp; the last block is a masked one
    uint4 symbols[BUNDLE_BLOCKS + 1];
    uint4 strands[BUNDLE_BLOCKS + 1];
};
struct BundleHead {
    int32_t ticket[4]; // next bundle of each sub-partition's list
};
constexpr size_t SM_SMEM = 227 * 1024; // what one block may have of an SM's
constexpr size_t bundle_smem_bytes(int depth) { return sizeof(BundleHead) + 4 * depth * sizeof(BundleColumns); }

template <int TM>
__global__ void __launch_bounds__(4 * COUPLE_DEPTH * 32) bundle_kernel(const CouplesLaunch L)
{
    extern __shared__ __align__(16) unsigned char bundle_smem[];
    constexpr int Q = TM / 4;
    const int lane = threadIdx.x & 31;
    const int w = __shfl_sync(FULL_MASK, int(threadIdx.x) >> 5, 0); // warp-uniform for the compiler
    BundleHead &H = *reinterpret_cast<BundleHead *>(bundle_smem);
    BundleColumns &W = reinterpret_cast<BundleColumns *>(bundle_smem + sizeof(BundleHead))[w];
    if (threadIdx.x < 4) {
        const int list = blockIdx.x * 4 + threadIdx.x;
        H.ticket[threadIdx.x] = list < L.nlists ? L.list_off[list] : INT_MAX;
    }
    __syncthreads();
    const int list = blockIdx.x * 4 + (w & 3);
    if (list >= L.nlists) return;
    const int end = L.list_off[list + 1];
    if (lane == 0) {
        W.symbols[BUNDLE_BLOCKS] = make_uint4(MASKED_COLUMN16, MASKED_COLUMN16, MASKED_COLUMN16, MASKED_COLUMN16);
        W.strands[BUNDLE_BLOCKS] = make_uint4(0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu);
    }
    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(&H.ticket[w & 3], 1);
        k = __shfl_sync(FULL_MASK, k, 0);
        if (k >= end) break;
        const BundleLane e = L.bundles[(L.nstaged_bundles + k) * 32 + lane];
        const int steps = __shfl_sync(FULL_MASK, e.steps, 0); // warp-uniform for the compiler
        const bool busy = e.couple >= 0;
        CoupleDev C{};
        if (busy) C = L.couples[e.couple];
        const int nb = C.nb, sl = e.sl;
        const bool first = sl == 0, last = sl == e.lanes - 1;
        uint32_t ap[TM], hp[TM], vc[4];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            split<TM>(couple_symbols(L.a_blob + C.a.a_off, C.a.m, L.a_blob + C.b.a_off, C.b.m, sl * Q + q, MASKED_ROW16),
                      ap, q);
            split<TM>(couple_h(C, sl * Q + q), hp, q);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) vc[j] = 0x7FFF7FFFu;
        for (int q = sl; q < nb; q += e.lanes) {
            W.symbols[e.base + q] =
                couple_symbols(L.b_blob + C.a.b_off, C.a.n, L.b_blob + C.b.b_off, C.b.n, q, MASKED_COLUMN16);
            W.strands[e.base + q] = couple_v(C, q);
        }
        __syncwarp();
        auto at = [&](int t) { // this lane's block in step t
            const int i = t - sl;
            return unsigned(i) < unsigned(nb) ? e.base + i : BUNDLE_BLOCKS;
        };
        int x = at(0);
        uint4 c = W.symbols[x], f = W.strands[x];
#pragma unroll 2
        for (int t = 0; t < steps; ++t) {
            const int xn = at(t + 1);
            const uint4 cn = W.symbols[xn], fn = W.strands[xn]; // only the first lane's f counts
            couple_step<TM>(c, f, first, ap, hp, vc);
            st_shared_if(last && x < BUNDLE_BLOCKS, &W.strands[x], vc);
            x = xn;
            c = cn;
            f = fn;
        }
        __syncwarp();
        if (busy) {
#pragma unroll
            for (int r = 0; r < TM; ++r) put_h(L, C, sl * TM + r, hp[r]);
            const uint32_t *v = reinterpret_cast<const uint32_t *>(&W.strands[e.base]);
#pragma unroll 4
            for (int i = sl; i < 4 * nb; i += e.lanes) put_v(L, C, i, v[i]);
        }
        __syncwarp();
    }
}

// Bundles of staged couples.
constexpr int AHEAD = 4; // steps (each about 350 cycles, an L2 hit about two of them)
constexpr int STAGED_WARPS = 4;
template <int TM>
__global__ void __launch_bounds__(STAGED_WARPS * 32) staged_bundle_kernel(const CouplesLaunch L)
{
    uint4 *const S = L.stage;
    constexpr int Q = TM / 4;
    const int lane = threadIdx.x & 31;
    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(L.ticket, 1);
        k = __shfl_sync(FULL_MASK, k, 0);
        if (k >= L.nstaged_bundles) break;
        const BundleLane e = L.bundles[k * 32 + lane];
        const int steps = __shfl_sync(FULL_MASK, e.steps, 0); // warp-uniform for the compiler
        const int nb = e.couple >= 0 ? L.couples[e.couple].nb : 0, off = e.couple >= 0 ? L.couples[e.couple].off : 0;
        const int sl = e.sl, rowq = e.lanes * Q;
        const bool first = sl == 0, last = sl == e.lanes - 1;
        uint32_t ap[TM], hp[TM], vc[4];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            uint4 a = make_uint4(MASKED_ROW16, MASKED_ROW16, MASKED_ROW16, MASKED_ROW16), h = make_uint4(0, 0, 0, 0);
            if (nb > 0) {
                a = S[off + sl * Q + q];
                h = S[off + rowq + sl * Q + q];
            }
            split<TM>(a, ap, q);
            split<TM>(h, hp, q);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) vc[j] = 0x7FFF7FFFu;
        const int cols = off + 2 * rowq; // symbols of block 0; strands nb further
        // Symbols (and for the first lane the fresh strands) of step t, loaded
        // AHEAD steps before.
        uint4 code[AHEAD], fresh[AHEAD] = {};
        auto load = [&](int t, uint4 &c, uint4 &f) {
            const int i = t - sl;
            const bool in = unsigned(i) < unsigned(nb);
            const uint4 *p = S + (in ? cols + i : 0);
            c = __ldg(p);
            f = ld_if(first, p + (in ? nb : 1), f);
        };
#pragma unroll
        for (int x = 0; x < AHEAD; ++x) load(x, code[x], fresh[x]);
        for (int t = 0; t < steps; t += AHEAD) {
#pragma unroll
            for (int x = 0; x < AHEAD; ++x) {
                const uint4 c = code[x], f = fresh[x];
                load(t + x + AHEAD, code[x], fresh[x]);
                couple_step<TM>(c, f, first, ap, hp, vc);
                const int i = t + x - sl;
                st_if(last && unsigned(i) < unsigned(nb), S + cols + nb + i, vc);
            }
        }
        if (nb > 0) {
#pragma unroll
            for (int q = 0; q < Q; ++q)
                S[off + rowq + sl * Q + q] = make_uint4(hp[4 * q], hp[4 * q + 1], hp[4 * q + 2], hp[4 * q + 3]);
        }
    }
}

template <int TM>
slcs_status launch_bundles(const CouplesLaunch &L, int depth, bool alone, int sms, cudaStream_t stream)
{
    int occ = 1, socc = 1;
    slcs_status s = occupancy_of<bundle_kernel<TM>>(4 * COUPLE_DEPTH * 32, &occ, SM_SMEM);
    if (s == SLCS_OK) s = occupancy_of<staged_bundle_kernel<TM>>(STAGED_WARPS * 32, &socc);
    if (s != SLCS_OK || stream == PREPARE_ONLY) return s;
    depth = depth > 0 ? std::min(depth, COUPLE_DEPTH) : COUPLE_DEPTH;
    if (L.nstaged > 0) {
        const int blocks = (L.nstaged + COUPLES_PER_BLOCK - 1) / COUPLES_PER_BLOCK;
        pack_couples_kernel<<<blocks, 32 * COUPLES_PER_BLOCK, 0, stream>>>(L);
        SLCS_CUDA(cudaGetLastError());
        const int want = (L.nstaged_bundles + STAGED_WARPS - 1) / STAGED_WARPS;
        staged_bundle_kernel<TM><<<std::min(want, sms * std::min(socc, depth)), STAGED_WARPS * 32, 0, stream>>>(L);
        SLCS_CUDA(cudaGetLastError());
        unpack_couples_kernel<<<blocks, 32 * COUPLES_PER_BLOCK, 0, stream>>>(L);
        SLCS_CUDA(cudaGetLastError());
    }
    if (L.nlists > 0) {
        // Alone: the rest of an SM's shared memory keeps other blocks off it.
        const size_t smem = alone ? SM_SMEM : bundle_smem_bytes(depth);
        bundle_kernel<TM><<<(L.nlists + 3) / 4, 4 * depth * 32, smem, stream>>>(L);
        SLCS_CUDA(cudaGetLastError());
    }
    return SLCS_OK;
}

} // namespace

bool packed16_supported(int tm, int seg) { return (tm == 4 || tm == 8 || tm == 12 || tm == 16) && seg == 16; }

slcs_status launch_couples(const CouplesLaunch &L, int tm, int depth, bool alone, int sms, cudaStream_t stream)
{
    switch (tm) {
    case 4: return launch_bundles<4>(L, depth, alone, sms, stream);
    case 8: return launch_bundles<8>(L, depth, alone, sms, stream);
    case 12: return launch_bundles<12>(L, depth, alone, sms, stream);
    case 16: return launch_bundles<16>(L, depth, alone, sms, stream);
    default: return fail(SLCS_ERR_UNSUPPORTED, "couples need 4, 8, 12 or 16 rows per lane");
    }
}

} // namespace slcs
