// strips.cu -- one pair combed as tiles, then merged by braid multiplication.
//
// a is cut into R row bands a_1..a_R and b into S column strips b_1..b_S.
// Every tile (a_r, b_s) is an independent comb (one persistent wavefront
// launch over all tiles), its strands become the permutation P(a_r, b_s)
// (src/permutation_matrix.hpp:88-115), and balanced trees of sticky-braid
// products glue them (src/braid_multiplication.hpp:273-407):
//   staggered_multiply<false>(P(a_r, x), P(a_r, y), |a_r|) == P(a_r, x y)
//   staggered_multiply<true>(P(x, b), P(y, b), |b|)       == P(x y, b)
// first the strips of every band, then the bands.  The last product is turned
// back into strands, so the caller sees exactly what the direct comb returns.
//
// This is the reference's tiled decomposition (tiles combed apart, then their
// permutations multiplied) at a coarse granularity.  Why it pays on the GPU:
// the stripes of one tile form a chain (stripe t starts about 32 column
// blocks after stripe t-1), so a tall pair spends the chain length in
// pipeline fill and drain.  Bands cut the chain into R shorter ones that fill
// at once; strips multiply the chains of a short pair, so that they fill the
// GPU.  Column strips are also the per-GPU unit of the multi-GPU split.
#include <algorithm>
#include <mutex>
#include <vector>

#include "braid.cuh"
#include "comb.cuh"
#include "strips.cuh"

namespace slcs {

namespace {

// row_to_col of P(a, b) (size m + n) -> strands: row i leaves at column c;
// c < n is the bottom exit of v strand c, c >= n the right exit of h strand c - n.
__global__ void perm_to_strands_kernel(const int32_t *__restrict__ r2c, int32_t m, int32_t n, int32_t *h,
                                       int32_t *v)
{
    const int64_t size = int64_t(m) + n;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < size; i += int64_t(gridDim.x) * blockDim.x) {
        const int32_t c = r2c[i];
        if (c >= 0 && c < n)
            v[c] = int32_t(i);
        else if (c >= n && int64_t(c) < size)
            h[c - n] = int32_t(i);
    }
}

// The tiles of a comb, numbered band by band, and its schedule, written on the
// device (a copy from the call's own memory would be read again, long after
// that memory is gone, by every replay of a graph that the call was captured in).
struct Tiles {
    int32_t m, n, bands, strips;
    int32_t stripe_rows, stripes; // rows of a stripe, stripes of a
    int32_t per;                  // stripes of a task: 1, or a relay group's
    int32_t base;                 // columns of every strip but the last
    int64_t hand;                 // entries of a band's scratch or hand-down rows; 0: no tile needs one

    __host__ __device__ int64_t row(int64_t r) const // first row of band r
    {
        const int64_t x = int64_t(stripes) * r / bands * stripe_rows;
        return r < bands && x < m ? x : m;
    }
    __host__ __device__ int64_t column(int64_t s) const { return s < strips ? s * base : n; }
    __host__ __device__ int64_t tasks(int64_t r) const // of one tile of band r
    {
        const int64_t count = int64_t(stripes) * (r + 1) / bands - int64_t(stripes) * r / bands;
        return (count + per - 1) / per;
    }
    __host__ __device__ int64_t tasks_before(int64_t r) const // of all tiles of the bands above r
    {
        if (per == 1) return int64_t(stripes) * r / bands * strips;
        int64_t t = 0;
        for (int64_t x = 0; x < r; ++x) t += tasks(x);
        return t * strips;
    }
    __host__ __device__ PairDev tile(int64_t r, int64_t s) const
    {
        const int64_t a0 = row(r), b0 = column(s), h = row(r + 1) - a0;
        return PairDev{a0, b0, strips * a0 + r * n + s * h + b0, int32_t(h), int32_t(column(s + 1) - b0)};
    }
};

// One block per tile.
__global__ void __launch_bounds__(128) tiles_kernel(const Tiles G, PairDev *pairs, int2 *tasks, int64_t *hand_off)
{
    const int t = blockIdx.x, r = t / G.strips, s = t % G.strips;
    const int64_t count = G.tasks(r), first = G.tasks_before(r) + s * count;
    if (threadIdx.x == 0) {
        pairs[t] = G.tile(r, s);
        hand_off[t] = r * G.hand + (G.hand > 0 ? G.column(s) : 0); // strips start at multiples of 16
    }
    for (int64_t k = threadIdx.x; k < count; k += blockDim.x) tasks[first + k] = make_int2(t, int(k));
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Batches of products of one tree level (bands of unequal heights, more
// products than a batch takes) run side by side on a small pool of streams per
// device (created once, never destroyed), each with its own braid workspace,
// forked from and joined back to the caller's stream with events.
constexpr int MAX_SIDE = 4;
std::mutex g_side_mu;
std::vector<cudaStream_t> g_side[64];

slcs_status side_streams(int count, cudaStream_t *out)
{
    int dev = 0;
    SLCS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(SLCS_ERR_UNSUPPORTED, "device index out of range");
    std::lock_guard<std::mutex> g(g_side_mu);
    auto &v = g_side[dev];
    while (int(v.size()) < count) {
        cudaStream_t t = nullptr;
        SLCS_CUDA(cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking));
        v.push_back(t);
    }
    for (int i = 0; i < count; ++i) out[i] = v[size_t(i)];
    return SLCS_OK;
}

// A permutation in one of the two strand buffers.
struct Perm {
    int64_t off, size;
};

// One level of a merge tree: in every job's list, neighbours are multiplied
// and an odd last entry is copied; each list is replaced by its results, laid
// one after another in the other buffer.  Products of one overlap go into the
// same launches, BRAID_MANY at most.
struct Level {
    struct Job {
        std::vector<Perm> *list;
        int32_t k;     // overlap of every product of the list
        bool row_glue; // staggered_multiply<true> (bands) or <false> (strips)
    };
    struct Batch {
        int32_t k;
        bool row_glue;
        std::vector<Perm> p, q, out;
    };
    std::vector<Batch> batches;
    std::vector<Perm> copy_from, copy_to;

    explicit Level(std::vector<Job> &&jobs)
    {
        int64_t off = 0;
        for (Job &J : jobs) {
            std::vector<Perm> out, &lv = *J.list;
            for (size_t i = 0; i < lv.size(); i += 2) {
                if (i + 1 < lv.size()) {
                    if (batches.empty() || batches.back().k != J.k || batches.back().row_glue != J.row_glue ||
                        batches.back().p.size() >= size_t(BRAID_MANY))
                        batches.push_back(Batch{J.k, J.row_glue, {}, {}, {}});
                    Batch *it = &batches.back();
                    out.push_back({off, lv[i].size + lv[i + 1].size - J.k});
                    it->p.push_back(lv[i]);
                    it->q.push_back(lv[i + 1]);
                    it->out.push_back(out.back());
                } else {
                    out.push_back({off, lv[i].size});
                    copy_from.push_back(lv[i]);
                    copy_to.push_back(out.back());
                }
                off += out.back().size;
            }
            lv.swap(out);
        }
    }
    // Workspace of one product of a batch.
    static size_t product_bytes(const Batch &B, int cutoff)
    {
        int64_t p = 0, q = 0;
        for (const Perm &x : B.p) p = std::max(p, x.size);
        for (const Perm &x : B.q) q = std::max(q, x.size);
        size_t bytes = 0;
        braid_workspace_bytes(int(p), int(q), B.k, cutoff, &bytes);
        return bytes;
    }
};

// Runs the levels: a level of one batch on the caller's stream, the batches
// of others round robin on the side streams (forked from and joined back to
// the caller's), each stream with its own workspace.
struct Merger {
    cudaStream_t st;
    cudaStream_t *side;
    int par;
    int cutoff;
    char *ws;
    size_t ws_bytes; // of one side stream
    cudaEvent_t fork = nullptr;
    cudaEvent_t join[MAX_SIDE] = {};

    slcs_status create()
    {
        if (par < 2) return SLCS_OK;
        SLCS_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
        for (int j = 0; j < par; ++j) SLCS_CUDA(cudaEventCreateWithFlags(&join[j], cudaEventDisableTiming));
        return SLCS_OK;
    }
    void destroy()
    {
        if (fork) cudaEventDestroy(fork);
        for (int j = 0; j < par; ++j)
            if (join[j]) cudaEventDestroy(join[j]);
    }
    slcs_status batch(const Level::Batch &B, const int32_t *src, int32_t *dst, int slot, cudaStream_t t)
    {
        BraidJob jobs[BRAID_MANY];
        const int count = int(B.p.size());
        for (int z = 0; z < count; ++z)
            jobs[z] = BraidJob{src + B.p[size_t(z)].off, int(B.p[size_t(z)].size), src + B.q[size_t(z)].off,
                               int(B.q[size_t(z)].size), dst + B.out[size_t(z)].off};
        return launch_braids(jobs, count, B.k, B.row_glue, cutoff, ws + ws_bytes * size_t(slot),
                             Level::product_bytes(B, cutoff), t);
    }
    // On an error the streams already forked are still joined back, so that
    // the caller's stream does not run ahead of (and free the workspace of)
    // products still in flight.
    slcs_status level(const Level &L, const int32_t *src, int32_t *dst)
    {
        slcs_status s = SLCS_OK;
        auto cu = [&](cudaError_t e, const char *what) {
            if (s == SLCS_OK && e != cudaSuccess) s = cuda_fail(e, what);
        };
        const bool forked = L.batches.size() > 1;
        int used = 0;
        if (forked) cu(cudaEventRecord(fork, st), "fork");
        for (size_t i = 0; i < L.batches.size() && s == SLCS_OK; ++i) {
            const int j = forked ? int(i) % par : 0;
            if (forked && j >= used) {
                cu(cudaStreamWaitEvent(side[j], fork, 0), "fork wait");
                used = j + 1;
            }
            if (s == SLCS_OK) s = batch(L.batches[i], src, dst, j, forked ? side[j] : st);
        }
        for (size_t i = 0; i < L.copy_from.size(); ++i)
            cu(cudaMemcpyAsync(dst + L.copy_to[i].off, src + L.copy_from[i].off,
                               sizeof(int32_t) * size_t(L.copy_from[i].size), cudaMemcpyDeviceToDevice, st),
               "odd part copy");
        for (int j = 0; j < used; ++j) {
            const cudaError_t e1 = cudaEventRecord(join[j], side[j]);
            const cudaError_t e2 = e1 == cudaSuccess ? cudaStreamWaitEvent(st, join[j], 0) : e1;
            if (e2 != cudaSuccess) {
                cu(e2, "join");
                cudaStreamSynchronize(side[j]); // could not order the streams: wait here
            }
        }
        return s;
    }
};

} // namespace

int strip_count(const slcs_config *cfg, int32_t n)
{
    int s = (cfg && cfg->strips > 0) ? cfg->strips : 8;
    s = std::min(s, std::max(1, int(n / 64)));
    return std::max(1, s);
}

int band_count(const slcs_config *cfg, int32_t m, int tm)
{
    int r = (cfg && cfg->bands > 0) ? cfg->bands : 1;
    r = std::min(r, std::max(1, int(stripes_of(m, tm))));
    return std::max(1, r);
}

std::vector<int32_t> strip_widths(int32_t n, int strips)
{
    std::vector<int32_t> w(size_t(strips), 0);
    if (strips <= 0) return w;
    // Strips start on 16-byte boundaries of b (whole-word symbol loads).
    const int32_t base = std::max<int32_t>(16, n / strips / 16 * 16);
    int32_t left = n;
    for (int s = 0; s < strips; ++s) {
        w[size_t(s)] = s + 1 < strips ? std::min(base, left) : left;
        left -= w[size_t(s)];
    }
    return w;
}

std::vector<int32_t> band_heights(int32_t m, int bands, int tm)
{
    std::vector<int32_t> h(size_t(bands), 0);
    if (bands <= 0) return h;
    // Bands are whole stripes (the last takes the rest), as equal in stripes
    // as the stripe count allows.
    const int64_t rows = 32 * int64_t(tm);
    const int64_t stripes = stripes_of(m, tm);
    int64_t left = m;
    for (int r = 0; r < bands; ++r) {
        const int64_t want = (stripes * (r + 1) / bands - stripes * r / bands) * rows;
        h[size_t(r)] = int32_t(r + 1 < bands ? std::min(want, left) : left);
        left -= h[size_t(r)];
    }
    return h;
}

slcs_status perm_to_strands(const int32_t *r2c, int32_t m, int32_t n, int32_t *h, int32_t *v, cudaStream_t st)
{
    const int64_t size = int64_t(m) + n;
    if (size <= 0) return SLCS_OK;
    int blocks = int(std::min<int64_t>((size + 255) / 256, int64_t(sm_count()) * 8));
    perm_to_strands_kernel<<<blocks, 256, 0, st>>>(r2c, m, n, h, v);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

slcs_status comb_strips(const uint8_t *a, int32_t m, const uint8_t *b, int32_t n, int32_t *h_out, int32_t *v_out,
                        const slcs_config *cfg, int tm, int warps, const RelayShape *relay, cudaStream_t st)
{
    if (relay) tm = relay->tm;
    const int R = band_count(cfg, m, tm);
    const int S = strip_count(cfg, n);
    const std::vector<int32_t> hgt = band_heights(m, R, tm);
    const std::vector<int32_t> w = strip_widths(n, S);
    // Tile (r, s) = (band r of a, strip s of b), numbered r * S + s; the tasks
    // of the comb are the stripes (relay: groups of stripes) of every tile,
    // tile after tile, so that a task's producer is the one before it.
    const int T = R * S;
    Tiles G{m, n, R, S, 32 * tm, stripes_of(m, tm), relay ? relay->warps : 1, w[0], 0};
    const int64_t total = int64_t(S) * m + int64_t(R) * n; // strands
    const int64_t ntasks = G.tasks_before(R);
    if (ntasks > T) // int32 of the wavefront's scratch, int2 of the relay's rows; whole 32-byte sectors
        G.hand = G.column(S - 1) + (int64_t(w[size_t(S - 1)]) + 7) / 8 * 8;
    const int64_t scr_elems = R * G.hand;
    const int cutoff = (cfg && cfg->braid_cutoff > 0) ? cfg->braid_cutoff : 0;
    // The merge tree: strips of every band glue with overlap = band height
    // (column glue), all bands side by side; then the bands glue with overlap
    // n (row glue).  Each level writes into the buffer the previous one did not.
    std::vector<Level> levels;
    std::vector<Perm> col;
    {
        std::vector<std::vector<Perm>> rows(static_cast<size_t>(R));
        for (int t = 0; t < T; ++t) {
            const PairDev d = G.tile(t / S, t % S);
            rows[size_t(t / S)].push_back({d.out_off, int64_t(d.m) + d.n});
        }
        while (rows[0].size() > 1) {
            std::vector<Level::Job> jobs;
            for (int r = 0; r < R; ++r) jobs.push_back({&rows[size_t(r)], hgt[size_t(r)], false});
            levels.emplace_back(std::move(jobs));
        }
        for (int r = 0; r < R; ++r) col.push_back(rows[size_t(r)][0]);
        while (col.size() > 1) levels.emplace_back(std::vector<Level::Job>{{&col, n, true}});
    }
    size_t braid_bytes = 0, most = 1; // workspace of a side stream; batches of a level
    for (const Level &L : levels) {
        most = std::max(most, L.batches.size());
        for (const Level::Batch &B : L.batches)
            braid_bytes = std::max(braid_bytes, Level::product_bytes(B, cutoff) * B.p.size());
    }
    // Workspace: descriptors, tasks, scratch offsets, counters, scratch,
    // strands / permutations (two buffers of S*m+R*n), braid workspaces.
    const size_t o_pairs = 0;
    const size_t o_tasks = align256(o_pairs + sizeof(PairDev) * size_t(T));
    const size_t o_soff = align256(o_tasks + sizeof(int2) * size_t(ntasks));
    const size_t o_work = align256(o_soff + sizeof(int64_t) * size_t(T));
    // The counters and, after them, what must be zero with them: the
    // wavefront's progress or the relay's rows.
    const size_t scr_bytes = size_t(scr_elems) * (relay ? sizeof(int2) : sizeof(int32_t));
    const size_t work_bytes = align256(relay ? 16 + scr_bytes : sizeof(int32_t) * (4 + size_t(ntasks)));
    const size_t o_scr = o_work + work_bytes;
    const size_t o_x = align256(o_scr + (relay ? 0 : scr_bytes + 16));
    const size_t o_y = align256(o_x + sizeof(int32_t) * size_t(total));
    const size_t o_braid = align256(o_y + sizeof(int32_t) * size_t(total));
    const int par = int(std::min(size_t(MAX_SIDE), most));
    const size_t bytes = o_braid + braid_bytes * size_t(par);
    char *ws = nullptr;
    SLCS_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&ws), bytes, st));
    slcs_status s = SLCS_OK;
    auto cu = [&](cudaError_t e, const char *what) {
        if (s == SLCS_OK && e != cudaSuccess) s = cuda_fail(e, what);
    };
    tiles_kernel<<<T, 128, 0, st>>>(G, reinterpret_cast<PairDev *>(ws + o_pairs), reinterpret_cast<int2 *>(ws + o_tasks),
                                    reinterpret_cast<int64_t *>(ws + o_soff));
    cu(cudaGetLastError(), "tiles");
    cu(cudaMemsetAsync(ws + o_work, 0, work_bytes, st), "counters");
    int32_t *X = reinterpret_cast<int32_t *>(ws + o_x);
    int32_t *Y = reinterpret_cast<int32_t *>(ws + o_y);
    if (s == SLCS_OK && relay) {
        RelayLaunch L{};
        L.pairs = reinterpret_cast<const PairDev *>(ws + o_pairs);
        L.items = reinterpret_cast<const int2 *>(ws + o_tasks);
        L.nitems = int32_t(ntasks);
        L.a_blob = a;
        L.b_blob = b;
        L.out = X;
        L.counters = reinterpret_cast<int32_t *>(ws + o_work);
        L.rows = reinterpret_cast<int2 *>(ws + o_work + 16);
        L.row_off = reinterpret_cast<const int64_t *>(ws + o_soff);
        L.status = device_status_word();
        L.wait_ns = wait_limit_ns(cfg);
        s = launch_relay(L, *relay, sm_count(), st);
    } else if (s == SLCS_OK) {
        CombLaunch L{};
        L.pairs = reinterpret_cast<const PairDev *>(ws + o_pairs);
        L.tasks = reinterpret_cast<const int2 *>(ws + o_tasks);
        L.ntasks = int32_t(ntasks);
        L.a_blob = a;
        L.b_blob = b;
        L.out = X;
        L.scratch = reinterpret_cast<int32_t *>(ws + o_scr);
        L.scratch_off = reinterpret_cast<const int64_t *>(ws + o_soff);
        L.counters = reinterpret_cast<int32_t *>(ws + o_work);
        L.progress = L.counters + 4;
        L.status = device_status_word();
        L.wait_ns = wait_limit_ns(cfg);
        const int32_t tallest = *std::max_element(hgt.begin(), hgt.end());
        L.tw = pick_tw(tm, stripes_of(tallest, tm), *std::min_element(w.begin(), w.end()), b);
        L.wide = wide_ids(tallest, *std::max_element(w.begin(), w.end()), cfg);
        s = launch_comb(L, tm, warps, st, nullptr);
    }
    // Strands of every tile -> its permutation (row -> col) in Y.
    if (s == SLCS_OK)
        s = launch_batch_to_perm(reinterpret_cast<const PairDev *>(ws + o_pairs), T, total, X, Y, st);
    cudaStream_t side[MAX_SIDE] = {};
    if (s == SLCS_OK && par > 1) s = side_streams(par, side);
    Merger M{st, side, par, cutoff, ws + o_braid, braid_bytes};
    if (s == SLCS_OK) s = M.create();
    int32_t *src = Y, *dst = X;
    for (size_t l = 0; l < levels.size() && s == SLCS_OK; ++l) {
        s = M.level(levels[l], src, dst);
        std::swap(src, dst);
    }
    M.destroy();
    if (s == SLCS_OK) s = perm_to_strands(src + col[0].off, m, n, h_out, v_out, st);
    cudaFreeAsync(ws, st);
    return s;
}

} // namespace slcs
