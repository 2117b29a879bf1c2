// queries.cu -- semi-local LCS queries answered from the strands.
//
// The strands of a comb are the semi-local solution: the reference computes
// them for every procedure and checks the whole-string LCS against its
// prefix DP (src/lcs_reference.hpp:71-132).  A v strand that enters at the
// top of column s leaves either at the bottom of some column k >= s or on
// the right edge; v_strands[k] holds the id (m + s for a v strand, < m for an
// h strand) of the strand leaving at the bottom of column k.  For a
// substring b[i, j) of b, the columns of b[i, j) that stay unmatched by any
// alignment with a are exactly the strands that enter and leave inside
// [i, j), so
//     LLCS(a, b[i, j)) = (j - i) - #{k in [i, j) : v_strands[k] >= m + i}
// (the whole-string case i = 0, j = n is the identity the oracle tests
// against the DP).
//
// Few or short queries are counted directly, one warp each.  For others the
// columns and the start positions s (a strand's id is m + s) are cut into
// blocks, and a table holds how many strands leave in the first x column
// blocks and start in position block y or later; a query then is two entries
// of the table, the columns before and after its whole blocks, and the
// positions between its start and the next block, looked up where they leave.
// Only the device sees how long the queries are, so the first of the table's
// launches decides: it answers them itself, and the others return at once, or
// it clears what the others fill.
#include <algorithm>

#include "queries.cuh"

namespace slcs {

namespace {

// Sum of x over the warp, in every lane.
__device__ __forceinline__ int warp_sum(int x)
{
    for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(FULL_MASK, x, off);
    return x;
}

// Strands of columns [k0, k1) with ids of at least lim, this lane's share.
__device__ __forceinline__ int count_columns(const int32_t *__restrict__ v, int k0, int k1, int lim, int lane)
{
    int cnt = 0;
    const int32_t *p = v + k0 + lane;
    const int rounds = int((unsigned(k1 - k0) + 31u - unsigned(lane)) / 32u);
#pragma unroll 4
    for (int t = 0; t < rounds; ++t, p += 32) cnt += __ldg(p) >= lim;
    return cnt;
}

// The table of one v array.  Its blocks are `block` wide in both directions.
struct Table {
    unsigned block;
    int rows, bins;  // column blocks, position blocks
    int32_t *count;  // (rows + 1) x (bins + 1): [x][y] as above
    int32_t *leave;  // n: the column where the strand of position s leaves, -1: on the right edge
    int32_t *state;  // [0] the table is made, [1] it holds: cleared when two columns have the same id (not strands of a comb)
};
constexpr int TABLE_MAX = 1024; // rows and bins, at most
constexpr int TABLE_THREADS = 256;

// Whether the table answers the queries sooner than a warp each does, in
// microseconds fitted to one B200: a warp takes 1.1 ns a column, all of them
// 2.2e-7 us, and a query at least 1.4e-4; the table 8 us, 2.3e-5 per column and
// 1e-5 per entry, and a query then 3.7e-4.  The lengths are those of at most 64
// queries, evenly spaced, so that deciding takes one round of reads (128 took
// the 20,000 queries of 100 columns 10.2 us, 32 8.5, 64 9.2).  Device time in us
// of the direct kernel alone, of the table, and as chosen here, n = 50,001: 64
// queries of 100 columns 2.4, 10.3, 4.8, of random ones 39, 12.4, 12.0; 20,000
// of 1,000 columns 8.9, 19.6, 14.3, of random ones 75, 19.6, 20.3; n = 2^24: 64
// of 2,000 columns 5.0, 398, 8.2, of random ones 20,697, 513, 440.
constexpr int SAMPLES = 2; // per lane
__device__ __forceinline__ bool table_pays(const int32_t *qb, const int32_t *qe, int32_t nq, int32_t n,
                                           const Table &T)
{
    constexpr unsigned MOST = SAMPLES * 32;
    float sum = 0.0f, longest = 0.0f;
#pragma unroll
    for (int x = 0; x < SAMPLES; ++x) {
        const unsigned t = x * 32 + (threadIdx.x & 31);
        if (t >= unsigned(nq)) continue;
        const unsigned q = unsigned(nq) <= MOST ? t : unsigned(nq) / MOST * t;
        const int i = __ldg(qb + q), j = __ldg(qe + q);
        const float len = i >= 0 && j > i && j <= n ? float(j - i) : 0.0f;
        sum += len;
        longest = fmaxf(longest, len);
    }
    for (int off = 16; off; off >>= 1) {
        sum += __shfl_xor_sync(FULL_MASK, sum, off);
        longest = fmaxf(longest, __shfl_xor_sync(FULL_MASK, longest, off));
    }
    if (unsigned(nq) > MOST) sum *= float(nq) / MOST;
    const float direct = fmaxf(1.1e-3f * longest, 2.2e-7f * sum + 1.4e-4f * nq);
    return direct > 8.0f + 2.3e-5f * n + 1e-5f * T.rows * T.bins + 3.7e-4f * nq;
}

// One warp per query (coalesced loads, the warp sums the counts).
template <bool TABLE>
__device__ __forceinline__ void answer_queries(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                               const int32_t *__restrict__ qb, const int32_t *__restrict__ qe,
                                               int32_t nq, int32_t *__restrict__ out, uint32_t *status, const Table &T)
{
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * (blockDim.x >> 5);
    const bool table = TABLE && T.state[1] != 0;
    for (long q = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; q < nq; q += warps) {
        const int i = __ldg(qb + q), j = __ldg(qe + q);
        if (i < 0 || j < i || j > n) { // bad query: -1, and the status word says so
            if (lane == 0) {
                out[q] = -1;
                raise_status(status, DEV_ERR_INPUT);
            }
            continue;
        }
        const int lim = m + i;
        int cnt = 0;
        const unsigned x0 = table ? (unsigned(i) + T.block - 1) / T.block : 0, x1 = table ? unsigned(j) / T.block : 0;
        if (TABLE && x0 < x1) {
            const int k0 = int(x0 * T.block), k1 = int(x1 * T.block); // the whole column blocks
            cnt = count_columns(v, i, k0, lim, lane) + count_columns(v, k1, j, lim, lane);
            // Position blocks start where column blocks do: from k0 on in the table.
            for (int s = i + lane; s < k0; s += 32) {
                const int k = T.leave[s];
                cnt += k >= k0 && k < k1;
            }
            if (lane == 0)
                cnt += T.count[int64_t(x1) * (T.bins + 1) + x0] - T.count[int64_t(x0) * (T.bins + 1) + x0];
        } else {
            cnt = count_columns(v, i, j, lim, lane);
        }
        cnt = warp_sum(cnt);
        if (lane == 0) out[q] = (j - i) - cnt;
    }
}

// The launches of the table follow each other closely: each may start while the
// one before it ends, and waits for its results before it does anything.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_last() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Decides; without the table this launch answers the queries, with it it
// clears the positions.
__global__ void __launch_bounds__(256, 8) first_queries_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                                               const int32_t *__restrict__ qb,
                                                               const int32_t *__restrict__ qe, int32_t nq,
                                                               int32_t *__restrict__ out, uint32_t *status, Table T)
{
    let_next_start();
    const bool pays = table_pays(qb, qe, nq, n, T);
    if (blockIdx.x == 0 && threadIdx.x == 0) T.state[0] = T.state[1] = pays;
    if (!pays) {
        answer_queries<false>(v, m, n, qb, qe, nq, out, status, T);
        return;
    }
    int4 *leave = reinterpret_cast<int4 *>(T.leave); // its space is a multiple of 16 bytes
    for (unsigned x = blockIdx.x * 256 + threadIdx.x; x < (unsigned(n) + 3) / 4; x += gridDim.x * 256)
        leave[x] = make_int4(-1, -1, -1, -1);
}

// One block per column block: its strands by position block, summed from the
// last one down; row x + 1 of the table before its rows are added up.
__global__ void __launch_bounds__(TABLE_THREADS) table_rows_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                                                   Table T)
{
    let_next_start();
    wait_for_last();
    if (!T.state[0]) return;
    __shared__ int hist[TABLE_MAX + 1];
    __shared__ int part[TABLE_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int y = threadIdx.x; y <= T.bins; y += TABLE_THREADS) hist[y] = 0;
    __syncthreads();
    const unsigned k1 = min(unsigned(n), (blockIdx.x + 1) * T.block);
    for (unsigned k = blockIdx.x * T.block + threadIdx.x; k < k1; k += TABLE_THREADS) {
        const int id = __ldg(v + k);
        if (id < m) continue; // an h strand
        const int s = id - m;
        atomicAdd(&hist[s < n ? unsigned(s) / T.block : T.bins], 1);
        if (s < n) T.leave[s] = int(k);
    }
    __syncthreads();
    // Suffix sums, a run of entries per thread, the last run first.
    const int run = (T.bins + TABLE_THREADS) / TABLE_THREADS;
    const int y1 = T.bins + 1 - int(threadIdx.x) * run, y0 = max(0, y1 - run);
    int own = 0;
    for (int y = y0; y < y1; ++y) own += hist[y];
    int sum = own; // of the runs up to this one
    for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(FULL_MASK, sum, off);
        if (lane >= off) sum += x;
    }
    if (lane == 31) part[w] = sum;
    __syncthreads();
    for (int x = 0; x < w; ++x) sum += part[x];
    int32_t *row = T.count + int64_t(blockIdx.x + 1) * (T.bins + 1);
    int acc = sum - own;
    for (int y = y1 - 1; y >= y0; --y) {
        acc += hist[y];
        row[y] = acc;
    }
}

// Blocks below `sums`: add the table's rows up, 32 columns of it per block,
// the rows in 32 chunks side by side.  The others check that every position
// leaves where it was found.
__global__ void __launch_bounds__(1024) table_sums_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n, Table T,
                                                          int sums)
{
    let_next_start();
    wait_for_last();
    if (!T.state[0]) return;
    if (int(blockIdx.x) >= sums) {
        const int64_t stride = int64_t(gridDim.x - sums) * blockDim.x;
        for (int64_t k = int64_t(blockIdx.x - sums) * blockDim.x + threadIdx.x; k < n; k += stride) {
            const int id = __ldg(v + k);
            if (id >= m && id - m < n && T.leave[id - m] != k) T.state[1] = 0;
        }
        return;
    }
    __shared__ int part[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int y = blockIdx.x * 32 + lane, per = (T.rows + 31) / 32;
    const int x0 = 1 + w * per, x1 = min(T.rows + 1, x0 + per);
    const bool in = y <= T.bins;
    int sum = 0;
    if (in)
        for (int x = x0; x < x1; ++x) sum += T.count[int64_t(x) * (T.bins + 1) + y];
    part[w][lane] = sum;
    __syncthreads();
    int acc = 0;
    for (int x = 0; x < w; ++x) acc += part[x][lane];
    if (!in) return;
    if (w == 0) T.count[y] = 0;
    for (int x = x0; x < x1; ++x) {
        int32_t *c = T.count + int64_t(x) * (T.bins + 1) + y;
        acc += *c;
        *c = acc;
    }
}

template <bool TABLE>
__global__ void __launch_bounds__(256) substring_llcs_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                                             const int32_t *__restrict__ qb,
                                                             const int32_t *__restrict__ qe, int32_t nq,
                                                             int32_t *__restrict__ out, uint32_t *status, Table T)
{
    if (TABLE) {
        wait_for_last();
        if (!T.state[0]) return;
    }
    answer_queries<TABLE>(v, m, n, qb, qe, nq, out, status, T);
}

} // namespace

slcs_status launch_substring_llcs(const int32_t *v, int32_t m, int32_t n, const int32_t *qb, const int32_t *qe,
                                  int32_t nq, int32_t *out, cudaStream_t st)
{
    if (nq <= 0) return SLCS_OK;
    const int blocks = int(std::min<long>((long(nq) + 7) / 8, long(sm_count()) * 16));
    // Below these sizes the table never pays (one B200, random queries, us
    // direct and by table: n = 20,000: 500 queries 21 and 31, 20,000 35 and 31,
    // 100,000 136 and 54; n = 5,000: 100,000 44 and 52).  Queries that the
    // answers overwrite are left to one kernel, which reads each before.
    auto apart = [&](const int32_t *q) {
        const uintptr_t x = reinterpret_cast<uintptr_t>(q), y = reinterpret_cast<uintptr_t>(out);
        const uintptr_t size = sizeof(int32_t) * uintptr_t(nq);
        return x + size <= y || y + size <= x;
    };
    Table T{};
    size_t leave_bytes = 0;
    char *ws = nullptr; // [state | leave | count]
    if ((n >= 32768 || (n >= 16384 && int64_t(nq) * n >= 300000000)) && apart(qb) && apart(qe)) {
        T.block = TABLE_THREADS * ((unsigned(n) + TABLE_THREADS * TABLE_MAX - 1) / (TABLE_THREADS * TABLE_MAX));
        T.rows = T.bins = int((unsigned(n) + T.block - 1) / T.block); // all below 2^32
        leave_bytes = (sizeof(int32_t) * size_t(n) + 15) / 16 * 16;
        const size_t count_bytes = sizeof(int32_t) * size_t(T.rows + 1) * size_t(T.bins + 1);
        if (cudaMallocAsync(reinterpret_cast<void **>(&ws), 16 + leave_bytes + count_bytes, st) !=
            cudaSuccess) {
            cudaGetLastError(); // no room: as without the table
            ws = nullptr;
        }
    }
    if (!ws) {
        substring_llcs_kernel<false><<<blocks, 256, 0, st>>>(v, m, n, qb, qe, nq, out, device_status_word(), T);
        SLCS_CUDA(cudaGetLastError());
        return SLCS_OK;
    }
    T.state = reinterpret_cast<int32_t *>(ws);
    T.leave = T.state + 4;
    T.count = reinterpret_cast<int32_t *>(ws + 16 + leave_bytes);
    uint32_t *status = device_status_word();
    const int clears = int(std::min<unsigned>((unsigned(n) + 4095) / 4096, unsigned(sm_count()) * 8));
    // (Resident blocks: more of them decide more often, and launch for nothing.)
    first_queries_kernel<<<std::max(std::min(blocks, sm_count() * 8), clears), 256, 0, st>>>(v, m, n, qb, qe, nq, out, status, T);
    cudaError_t e = cudaGetLastError();
    auto then = [&](auto kernel, int grid, int threads, auto... args) {
        cudaLaunchConfig_t c{};
        cudaLaunchAttribute close{};
        close.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        close.val.programmaticStreamSerializationAllowed = 1;
        c.gridDim = dim3(unsigned(grid));
        c.blockDim = dim3(unsigned(threads));
        c.stream = st;
        c.attrs = &close;
        c.numAttrs = 1;
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&c, kernel, args...);
    };
    const int sums = T.bins / 32 + 1, checks = int(std::min<unsigned>((unsigned(n) + 1023) / 1024, 64));
    then(table_rows_kernel, T.rows, TABLE_THREADS, v, m, n, T);
    then(table_sums_kernel, sums + checks, 1024, v, m, n, T, sums);
    then(substring_llcs_kernel<true>, std::min(blocks, sm_count() * 6), 256, v, m, n, qb, qe, nq, out, status, T);
    const cudaError_t f = cudaFreeAsync(ws, st);
    if (e != cudaSuccess) return cuda_fail(e, "substring queries");
    SLCS_CUDA(f);
    return SLCS_OK;
}

} // namespace slcs
