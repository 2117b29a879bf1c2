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
// Few or short queries are counted directly, one warp each.  Otherwise the
// columns and the start positions s (a strand's id is m + s) are cut into
// blocks, and a table holds how many strands leave in the first x column
// blocks and start in position block y or later; a query then is two entries
// of the table, the columns before and after its whole blocks, and the
// positions between its start and the next block, looked up where they leave.
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
    for (int k = k0 + lane; k < k1; k += 32) cnt += __ldg(v + k) >= lim;
    return cnt;
}

// The table of one v array.  Its blocks are `block` wide in both directions.
struct Table {
    int block, rows, bins;    // column blocks, position blocks
    int32_t *count;           // (rows + 1) x (bins + 1): [x][y] as above
    int32_t *leave;           // n: the column where the strand of position s leaves, -1: on the right edge
    int32_t *sound;           // -1; cleared when two columns hold the same id (not strands of a comb)
};
constexpr int TABLE_MAX = 1024; // rows and bins, at most
constexpr int TABLE_THREADS = 256;

// One block per column block: its strands by position block, summed from the
// last one down; row x + 1 of the table before its rows are added up.
__global__ void __launch_bounds__(TABLE_THREADS) table_rows_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                                                   Table T)
{
    __shared__ int hist[TABLE_MAX + 1];
    __shared__ int part[TABLE_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int y = threadIdx.x; y <= T.bins; y += TABLE_THREADS) hist[y] = 0;
    __syncthreads();
    const int k1 = min(n, int(blockIdx.x + 1) * T.block);
    for (int k = blockIdx.x * T.block + threadIdx.x; k < k1; k += TABLE_THREADS) {
        const int s = __ldg(v + k) - m;
        if (s < 0) continue; // an h strand
        atomicAdd(&hist[s < n ? s / T.block : T.bins], 1);
        if (s < n) T.leave[s] = k;
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
    if (int(blockIdx.x) >= sums) {
        const int stride = (gridDim.x - sums) * blockDim.x;
        for (int k = (blockIdx.x - sums) * blockDim.x + threadIdx.x; k < n; k += stride) {
            const int s = __ldg(v + k) - m;
            if (s >= 0 && s < n && T.leave[s] != k) *T.sound = 0;
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

// One warp per query (coalesced loads, the warp sums the counts).
template <bool TABLE>
__global__ void __launch_bounds__(256) substring_llcs_kernel(const int32_t *__restrict__ v, int32_t m, int32_t n,
                                                             const int32_t *__restrict__ qb,
                                                             const int32_t *__restrict__ qe, int32_t nq,
                                                             int32_t *__restrict__ out, uint32_t *status, Table T)
{
    const int lane = threadIdx.x & 31;
    const long warps = long(gridDim.x) * (blockDim.x >> 5);
    const bool table = TABLE && *T.sound != 0;
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
        const int x0 = TABLE ? (i + T.block - 1) / T.block : 0, x1 = TABLE ? j / T.block : 0;
        if (table && x0 < x1) {
            const int k0 = x0 * T.block, k1 = x1 * T.block; // the whole column blocks
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

} // namespace

slcs_status launch_substring_llcs(const int32_t *v, int32_t m, int32_t n, const int32_t *qb, const int32_t *qe,
                                  int32_t nq, int32_t *out, cudaStream_t st)
{
    if (nq <= 0) return SLCS_OK;
    const int blocks = int(std::min<long>((long(nq) + 7) / 8, long(sm_count()) * 16));
    // A warp reads 32 columns a round and waits for them, the table takes four
    // launches.  One B200, random queries, us direct and by table: n = 20,000:
    // 500 queries 21 and 31, 20,000 35 and 31, 100,000 136 and 54; n = 50,001:
    // 64 queries 42 and 24, 20,000 79 and 30; n = 262,144: 64 queries 308 and 34,
    // 100,000 2,469 and 75; n = 5,000: 100,000 44 and 52.
    const bool by_table = n >= 32768 || (n >= 16384 && int64_t(nq) * n >= 300000000);
    if (!by_table) {
        substring_llcs_kernel<false><<<blocks, 256, 0, st>>>(v, m, n, qb, qe, nq, out, device_status_word(), Table{});
        SLCS_CUDA(cudaGetLastError());
        return SLCS_OK;
    }
    Table T{};
    T.block = TABLE_THREADS * ((n + TABLE_THREADS * TABLE_MAX - 1) / (TABLE_THREADS * TABLE_MAX));
    T.rows = T.bins = (n + T.block - 1) / T.block;
    const size_t count_bytes = sizeof(int32_t) * size_t(T.rows + 1) * size_t(T.bins + 1);
    char *ws = nullptr; // [sound | leave | count]
    SLCS_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&ws), 16 + sizeof(int32_t) * size_t(n) + count_bytes, st));
    T.sound = reinterpret_cast<int32_t *>(ws);
    T.leave = T.sound + 4;
    T.count = T.leave + n;
    cudaError_t e = cudaMemsetAsync(ws, 0xff, 16 + sizeof(int32_t) * size_t(n), st);
    if (e == cudaSuccess) {
        table_rows_kernel<<<T.rows, TABLE_THREADS, 0, st>>>(v, m, n, T);
        const int sums = T.bins / 32 + 1;
        table_sums_kernel<<<sums + std::min((n + 1023) / 1024, 64), 1024, 0, st>>>(v, m, n, T, sums);
        substring_llcs_kernel<true><<<blocks, 256, 0, st>>>(v, m, n, qb, qe, nq, out, device_status_word(), T);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(ws, st);
    if (e != cudaSuccess) return cuda_fail(e, "substring queries");
    SLCS_CUDA(f);
    return SLCS_OK;
}

} // namespace slcs
