// api.cu -- the C ABI of libslcs (declared in include/slcs.h).
//
// Host logic only: argument checks, schedules (task lists), scratch and
// workspace management, batch plans with optional CUDA-graph replay, and the
// synchronous host-pointer wrappers.  All combing runs in comb.cu.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <queue>
#include <string>
#include <type_traits>
#include <vector>

#include "braid.cuh"
#include "comb.cuh"
#include "couples.cuh"
#include "queries.cuh"
#include "relay.cuh"
#include "strips.cuh"

namespace slcs {

namespace {
thread_local std::string g_last_error;

struct DeviceState {
    uint32_t *host_status = nullptr;
    uint32_t *dev_status = nullptr;
    cudaMemPool_t plan_pool = nullptr; // of the batch plans' blocks; null: they come from cudaMalloc
    int sms = 0;
    bool init = false;
};
std::mutex g_dev_mu;
DeviceState g_dev[64];
constexpr uint64_t PLAN_POOL_KEPT = uint64_t(64) << 20;

DeviceState &dev_state()
{
    int d = 0;
    cudaGetDevice(&d);
    if (d < 0 || d >= 64) d = 0;
    std::lock_guard<std::mutex> g(g_dev_mu);
    DeviceState &s = g_dev[d];
    if (!s.init) {
        s.init = true;
        cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, d);
        if (s.sms <= 0) s.sms = 148;
        // Workspaces come from cudaMallocAsync on every call; by default the
        // process's pool returns freed memory to the driver at each
        // synchronisation, and mapping it again cost milliseconds per call.
        // Keep it in the pool (a setting of this process only).
        cudaMemPool_t pool = nullptr;
        if (cudaDeviceGetDefaultMemPool(&pool, d) == cudaSuccess) {
            uint64_t keep = UINT64_MAX;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        // Batch plans have a pool of their own, which keeps PLAN_POOL_KEPT and
        // gives the rest back when a plan is destroyed: their blocks can be
        // gigabytes and may never be wanted again.
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = d;
        if (cudaMemPoolCreate(&s.plan_pool, &props) == cudaSuccess) {
            uint64_t keep = PLAN_POOL_KEPT;
            cudaMemPoolSetAttribute(s.plan_pool, cudaMemPoolAttrReleaseThreshold, &keep);
        } else {
            s.plan_pool = nullptr;
        }
        cudaGetLastError();
        void *p = nullptr;
        if (cudaHostAlloc(&p, 64, cudaHostAllocMapped) == cudaSuccess) {
            s.host_status = static_cast<uint32_t *>(p);
            *s.host_status = 0;
            void *dp = nullptr;
            if (cudaHostGetDevicePointer(&dp, p, 0) == cudaSuccess) s.dev_status = static_cast<uint32_t *>(dp);
        } else {
            cudaGetLastError();
        }
    }
    return s;
}

} // namespace

// Rows per lane for pairs of about m_typical rows on a device of `sms` SMs.
int pick_tile_m_for(const slcs_config *cfg, int32_t m_typical, int sms)
{
    if (cfg && cfg->tile_m) return cfg->tile_m;
    if (m_typical >= (1 << 19)) {
        // All stripes of one long pair are resident at once and every warp
        // stays on one SM sub-partition (4 per SM), so the busiest
        // sub-partition sets the pace: pick the rows per lane that minimise
        // its rows, ceil(stripes / sub-partitions) * rows per stripe (2^20
        // rows: 14 -> 2341 stripes, 4 per sub-partition; 16 -> 2048 stripes,
        // still 4 on most).  Ties go to the taller stripe.
        const int64_t parts = 4 * int64_t(std::max(1, sms));
        int best = 16;
        int64_t best_rows = INT64_MAX;
        for (int tm : {16, 14, 12}) {
            const int64_t stripes = stripes_of(m_typical, tm);
            const int64_t rows = (stripes + parts - 1) / parts * tm;
            if (rows < best_rows) {
                best_rows = rows;
                best = tm;
            }
        }
        return best;
    }
    if (m_typical >= 262144) return 16; // >= 512 stripes of 512 rows: enough warps in flight
    if (m_typical >= 65536) return 8;
    if (m_typical >= 8192) return 4;
    if (m_typical <= 64) return 2;
    if (m_typical <= 128) return 4;
    return 8;
}

namespace {

int pick_tile_m(const slcs_config *cfg, int32_t m_typical, int64_t total_cells)
{
    (void)total_cells;
    // The SM count matters only to tall pairs; shorter ones need no device.
    const bool tall = !(cfg && cfg->tile_m) && m_typical >= (1 << 19);
    return pick_tile_m_for(cfg, m_typical, tall ? sm_count() : 1);
}

// Column strips for one pair when nothing is configured and no relay shape
// takes it (on 148 SMs below 2^19 rows only pairs of more than 2^30 ids), fitted
// to B200 timings of uniform {0..3} pairs.  One wavefront keeps few warps busy below
// about 2^19 rows (stripe t starts 32 column blocks after stripe t-1), while
// every strip adds a braid product with overlap m.  About n / sqrt(4096 m)
// strips (a power of two, rounded up from 2^(k+0.45); 1..64 strips of at
// least 4096 columns) balance the two; pairs of 2^17 and of 2^18 rows and
// more take at most 4 and 2 strips.
int auto_strips(int32_t m, int32_t n)
{
    if (m <= 0 || n < 8192 || m >= (1 << 19)) return 1;
    const double base = double(n) / std::sqrt(4096.0 * double(m));
    int S = base <= 1.0 ? 1 : 1 << int(std::floor(std::log2(base) + 0.55));
    if (n >= 32768) S = std::max(S, 2);
    if (m >= (1 << 17)) S = std::min(S, 4);
    if (m >= (1 << 18)) S = std::min(S, 2);
    S = std::min(S, 64);
    while (S > 1 && n / S < 4096) S /= 2;
    return S;
}

// Row bands for one tall pair (at least 2^19 rows) when nothing is configured
// and no relay shape takes it (on 148 SMs beyond 1,060,864 rows).  The stripes of a band form a chain that fills and drains in
// about 44 steps of 4 columns per stripe, so a pair combed in R bands spends
// about (n + 176 * stripes / R) / n times its cell time; every band adds
// row-glue products, about log2(R) * m + (R - 1) * n permutation entries in
// all.  The constants (3.5 Tcells/s, 1.5 ns per entry) are fitted to B200
// timings of the 2^20 x 2^20 pair (R = 1, 2, 4, 8, 16: 410, 348, 327, 324,
// 334 ms).
int auto_bands(int32_t m, int32_t n, int tm)
{
    if (m < (1 << 19) || n <= 0) return 1;
    const double stripes = double(stripes_of(m, tm));
    const double cells = double(m) * double(n);
    int best = 1;
    double best_t = 0;
    for (int R = 1; R <= 16 && R <= stripes; R *= 2) {
        const double fill = (double(n) + 176.0 * std::ceil(stripes / R)) / double(n);
        const double t = cells / 3.5e12 * fill + 1.5e-9 * (std::log2(double(R)) * m + double(R - 1) * n);
        if (R == 1 || t < best_t) {
            best = R;
            best_t = t;
        }
    }
    return best;
}

} // namespace

// Row bands of a pair combed as column strips (below 2^19 rows): a strip's
// stripes form a chain that spends about 176 columns per stripe filling, so
// from 2^16 rows on the strips are cut into bands of about 32768 rows (64
// stripes of 16 rows per lane), at most 8.  Measured on B200, the 131072 x
// 131072 mutated pair at 16 rows per lane and 4 strips: 1, 2, 4, 8 bands
// 17.1, 14.4, 13.0, 14.0 ms; 2 x 8 and 8 x 4 tiles 13.8 and 14.7 ms.
int strip_bands(int32_t m)
{
    if (m < (1 << 16)) return 1;
    return std::min(8, std::max(1, int(m / 32768)));
}

// 14 or 16 rows per lane leave room for 8 warps per block; the smaller tiles run 4.
int pick_warps(const slcs_config *cfg, int tm) { return (cfg && cfg->warps) ? cfg->warps : (tm >= 14 ? 8 : 4); }

namespace {

// Shapes of the relay kernel: rows per lane, columns per step, combing warps,
// and the cycles one step takes while a block has its SM to itself (B200,
// inside whole combs; a step is bound by the chain shuffle -> cells -> shuffle
// until 8 rows per lane, then by instruction issue).
struct RelayCost {
    RelayShape shape;
    double step;
};
const RelayCost RELAY_COSTS[] = {{{1, 4, 3}, 66.0},  {{2, 4, 3}, 79.0},  {{4, 2, 3}, 76.0},
                                 {{8, 2, 3}, 108.0}, {{8, 4, 4}, 212.0}, {{14, 4, 4}, 344.0},
                                 {{14, 4, 8}, 665.0}, {{14, 4, 16}, 1277.0}};
constexpr double RELAY_GHZ = 1.965;     // the clock those cycles were measured at
constexpr double RELAY_WARP_LAG = 40.0; // steps a warp starts after the warp above it
constexpr double RELAY_HOP_LAG = 45.0;  // more steps for the hand-down to the next block

// Microseconds of a merge level of `count` braid products of overlap k, which
// run in the same launches (B200): one product's time, and about 1.2 ns per
// entry that the others add to it.
double merge_us(double k, double count)
{
    static const double log2k[] = {6, 8, 10, 12, 14, 16, 17, 20};
    static const double us[] = {38, 44, 60, 113, 166, 246, 334, 1206};
    const double x = std::log2(std::max(k, 64.0));
    int i = 0;
    while (i < 6 && x >= log2k[i + 1]) ++i;
    return us[i] + (us[i + 1] - us[i]) * (x - log2k[i]) / (log2k[i + 1] - log2k[i]) + 0.0012 * k * (count - 1);
}

// The relay kernel's plan for one pair: shape, column strips and row bands
// with the least predicted time among those whose groups fit one to an SM
// (two blocks on one SM slow the whole chain: 342 groups of (4, 2, 3) on 148
// SMs combed 131072 x 131072 in 13.2 ms, 128 of (8, 4, 4) in 6.4 ms; 152 groups
// of (14, 4, 16) combed the 2^20 pair in 353 ms, 148 in 190).  Bands one after
// another would need no more SMs but are not planned: a pair past the tallest
// shape, 1,060,864 rows on 148 SMs, takes the wavefront kernel (1,060,865 x
// 30,000: 17.4 ms).
// relay.tm == 0: no shape fits.  Predicted: a chain's steps (columns, then
// the lags of its warps and blocks) at the shape's step time, and the merge
// levels.
struct RelayPlan {
    RelayShape relay{};
    int strips = 1, bands = 1;
    double us = 0;
};
RelayPlan plan_relay(int32_t m, int32_t n, int sms)
{
    RelayPlan best;
    for (const RelayCost &c : RELAY_COSTS)
        for (int R = 1; R <= 16 && (R == 1 || m / R >= 4096); R *= 2)
            for (int S = 1; S <= 64 && (S == 1 || n / S >= 4096); S *= 2) {
                const double stripes = std::ceil(std::ceil(double(m) / (32 * c.shape.tm)) / R);
                const double groups = std::ceil(stripes / c.shape.warps);
                if (groups * R * S > sms) continue;
                const double steps = double(n) / S / c.shape.tw + RELAY_WARP_LAG * stripes + RELAY_HOP_LAG * groups;
                double us = 6.0 + steps * c.step / (RELAY_GHZ * 1e3);
                if (R * S > 1) us += 20.0;
                for (int p = S; p > 1; p /= 2) us += merge_us(double(m) / R, double(R) * (p / 2));
                for (int p = R; p > 1; p /= 2) us += merge_us(double(n), p / 2);
                if (best.relay.tm == 0 || us < best.us) best = RelayPlan{c.shape, S, R, us};
            }
    return best;
}

// The shapes with two pairs per register, and their steps.
const RelayCost RELAY_DUO_COSTS[] = {{{2, 4, 3}, 92.0}, {{4, 4, 3}, 135.0}, {{8, 2, 3}, 160.0}, {{8, 4, 4}, 248.0}};

// Instructions a combing warp of a relay shape issues per step (about; B200,
// counted for (4, 4) and scaled by cells), the I/O warp about 12.
double relay_issue(const RelayShape &s) { return 4.3 * s.tm * s.tw + 10.0 + 3.0 * s.tw; }

// Pairs of a batch that the relay kernel combs: (m, n) each, or the larger m
// and n of two pairs that share a register.
using Sizes = std::vector<std::pair<int32_t, int32_t>>;

// Longest chain (steps) and issue slots of a shape.
struct RelayWork {
    double chain = 0, slots = 0;
    int64_t groups = 0;
};
RelayWork relay_work(const Sizes &sizes, const RelayShape &s)
{
    const double issue = relay_issue(s);
    RelayWork w;
    for (const auto &[m, n] : sizes) {
        const int32_t stripes = (m + 32 * s.tm - 1) / (32 * s.tm);
        const int32_t groups = (stripes + s.warps - 1) / s.warps;
        const double own = double(n) / s.tw + 31.0; // steps of one warp
        w.chain = std::max(w.chain, own + RELAY_WARP_LAG * stripes + RELAY_HOP_LAG * groups);
        w.slots += stripes * own * issue + groups * (own + RELAY_WARP_LAG * (s.warps - 1)) * 12.0;
        w.groups += groups;
    }
    return w;
}

// Microseconds the relay kernel takes for them, with the best shape: its
// longest chain plus its blocks' issue slots, spread over the SMs (on B200
// within a factor of 0.85 to 1.7 of sweeps from 64 reads to 1,000 pairs of
// 9000 x 100 rows and columns).
double batch_relay_us(const Sizes &sizes, int sms, RelayShape *shape)
{
    double best = -1.0;
    for (const RelayCost &c : RELAY_COSTS) {
        const RelayWork w = relay_work(sizes, c.shape);
        const double us = 8.0 + 1.2 * (w.chain * c.step + w.slots / (4.0 * sms)) / (RELAY_GHZ * 1e3);
        if (best < 0 || us < best) {
            best = us;
            *shape = c.shape;
        }
    }
    return best;
}

// The same with contention by blocks: alone on its SM a block keeps its step;
// on shared SMs each further block adds its issue to a chain's step, and with
// many the slots count.  With two pairs per register within 0.87 to 1.12 of
// thirteen batches (2 pairs of 600 x 8000 to 400 of 2000 x 2000), with one
// 0.73 to 1.06.
template <class Costs>
double relay_shared_us(const Sizes &sizes, const Costs &costs, int sms, RelayShape *shape)
{
    double best = -1.0;
    for (const RelayCost &c : costs) {
        const RelayWork w = relay_work(sizes, c.shape);
        const double blocks = std::ceil(double(w.groups) / sms);
        double cycles = w.chain * c.step;
        if (blocks > 1) {
            const double crowded = w.chain * (c.step + 1.1 * (blocks - 1) * relay_issue(c.shape) * c.shape.warps / 4.0);
            cycles = std::max(blocks <= 3 ? crowded : 0.0, cycles + 1.35 * w.slots / (4.0 * sms));
        }
        const double us = 8.0 + cycles / (RELAY_GHZ * 1e3);
        if (best < 0 || us < best) {
            best = us;
            *shape = c.shape;
        }
    }
    return best;
}

// How the relay kernel combs the pairs that `take` selects: one per register
// or, when every pair's ids fit 15 bits and it is predicted faster, two,
// neighbours in rows and then columns.  Two take half the instructions, but a
// step of a lone chain 1.2 to 1.8 times as long: 96 pairs of up to 2900 x 3300
// 309 -> 183 us, 30 of 9000 x 9000 1131 -> 542, 64 of 400 x 5000 112 -> 91;
// 2 of 4000 x 4000 147 -> 194, which stay apart.
struct BatchRelay {
    RelayShape shape{};
    std::vector<int2> duos; // empty: one pair per register
    double us = 0.0;
    int64_t groups = 0;
};
// With `budget_us`, the plan of fewest groups predicted to end within it, if any.
template <class Take>
BatchRelay plan_batch_relay(const slcs_pair_desc *pairs, int32_t npairs, bool may_two, int sms, Take take,
                            double budget_us = 0.0)
{
    BatchRelay B;
    std::vector<int32_t> ids;
    for (int32_t p = 0; p < npairs; ++p)
        if (take(p) && pairs[p].m > 0 && pairs[p].n > 0) {
            ids.push_back(p);
            may_two = may_two && int64_t(pairs[p].m) + pairs[p].n <= PACKED16_MAX_IDS;
        }
    Sizes sizes, both;
    std::vector<int2> duos;
    for (int32_t p : ids) sizes.emplace_back(pairs[p].m, pairs[p].n);
    B.us = batch_relay_us(sizes, sms, &B.shape);
    if (may_two && ids.size() > 1) {
        constexpr int32_t ROWS = 256; // pairs within so many rows are neighbours by columns
        std::sort(ids.begin(), ids.end(), [&](int32_t x, int32_t y) {
            const int32_t rx = pairs[x].m / ROWS, ry = pairs[y].m / ROWS;
            return rx != ry ? rx > ry : pairs[x].n != pairs[y].n ? pairs[x].n > pairs[y].n : x < y;
        });
        for (size_t i = 0; i < ids.size(); i += 2) {
            const slcs_pair_desc &x = pairs[ids[i]];
            const bool second = i + 1 < ids.size();
            duos.push_back(make_int2(ids[i], second ? ids[i + 1] : -1));
            both.emplace_back(second ? std::max(x.m, pairs[ids[i + 1]].m) : x.m,
                              second ? std::max(x.n, pairs[ids[i + 1]].n) : x.n);
        }
        RelayShape one{}, two{};
        const double us = relay_shared_us(both, RELAY_DUO_COSTS, sms, &two);
        if (us < relay_shared_us(sizes, RELAY_COSTS, sms, &one)) {
            B.us = us;
            B.shape = two;
            B.duos = duos;
        }
    }
    B.groups = relay_work(B.duos.empty() ? sizes : both, B.shape).groups;
    if (budget_us > 0) {
        auto fewer = [&](const Sizes &of, const RelayCost &c, const std::vector<int2> &d) {
            const RelayCost only[] = {c};
            RelayShape shape{};
            const double us = relay_shared_us(of, only, sms, &shape);
            const int64_t groups = relay_work(of, shape).groups;
            if (us <= budget_us && groups < B.groups) B = BatchRelay{shape, d, us, groups};
        };
        for (const RelayCost &c : RELAY_COSTS) fewer(sizes, c, {});
        for (const RelayCost &c : RELAY_DUO_COSTS)
            if (!duos.empty()) fewer(both, c, duos);
    }
    return B;
}

// How slcs_comb_pair combs one pair: the effective configuration (algo
// WAVEFRONT or STRIPS with tile_m, warps, strips, bands, braid_cutoff set),
// and the relay plan that takes its place when nothing is configured and the
// pair fits one.
struct PairPlan {
    slcs_config c;
    RelayPlan relay;
};

slcs_status plan_pair(int32_t m, int32_t n, const slcs_config *cfg, int sms, PairPlan *P)
{
    P->c = cfg ? *cfg : slcs_config{};
    slcs_config &c = P->c;
    const int tm = pick_tile_m_for(cfg, m, sms);
    if (!tile_m_supported(tm)) return fail(SLCS_ERR_UNSUPPORTED, "tile_m must be one of 2, 4, 8, 12, 14, 16");
    const bool auto_all = !cfg || (cfg->algo == SLCS_ALGO_AUTO && cfg->tile_m == 0 && cfg->warps == 0 &&
                                   cfg->strips == 0 && cfg->bands == 0);
    c.tile_m = tm;
    c.warps = pick_warps(cfg, tm);
    if (c.algo == SLCS_ALGO_STRIPS) {
        c.strips = strip_count(cfg, n);
        c.bands = band_count(cfg, m, tm);
        if (c.braid_cutoff <= 0) c.braid_cutoff = 1024;
        return SLCS_OK;
    }
    c.algo = SLCS_ALGO_WAVEFRONT;
    c.strips = 1;
    c.bands = 1;
    if (!auto_all) return SLCS_OK;
    if (!wide_ids(m, n, cfg)) P->relay = plan_relay(m, n, sms);
    int R = auto_bands(m, n, tm);
    const int S = R > 1 ? 1 : auto_strips(m, n);
    if (S > 1) R = strip_bands(m);
    if (R > 1 || S > 1) {
        c.algo = SLCS_ALGO_STRIPS;
        c.strips = S;
        c.bands = R;
        if (S > 1) { // short pairs: column strips of 16-row stripes, 4 warps per block
            c.tile_m = 16;
            c.warps = 4;
        }
        if (c.braid_cutoff <= 0) c.braid_cutoff = 256;
    }
    return SLCS_OK;
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

__global__ void identity_strands_kernel(int32_t *h, int32_t m, int32_t *v, int32_t n)
{
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m + n; i += gridDim.x * blockDim.x) {
        if (i < m) h[i] = i;
        else v[i - m] = i;
    }
}

// Host schedule of a batch: pairs ordered by cells (largest first).  Pairs of
// at most stream_rows rows (stream_rows > 0) are streamed; every other pair
// contributes its row stripes as consecutive wavefront tasks, with a scratch
// row when it has more than one stripe.
struct Schedule {
    std::vector<int32_t> order; // every pair, most cells first
    std::vector<int2> tasks;
    std::vector<int32_t> stream_pairs;
    std::vector<int64_t> scratch_off;
    int64_t scratch_elems = 0;
};

Schedule build_schedule(const slcs_pair_desc *pairs, int32_t npairs, int tm, int32_t stream_rows)
{
    Schedule S;
    std::vector<int32_t> &order = S.order;
    order.resize(npairs);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
        return int64_t(pairs[x].m) * pairs[x].n > int64_t(pairs[y].m) * pairs[y].n;
    });
    S.scratch_off.assign(npairs, 0);
    for (int32_t p : order) {
        if (pairs[p].m == 0 || pairs[p].n == 0) continue;
        if (pairs[p].m <= stream_rows) {
            S.stream_pairs.push_back(p);
            continue;
        }
        const int32_t st = stripes_of(pairs[p].m, tm);
        for (int32_t s = 0; s < st; ++s) S.tasks.push_back(make_int2(p, s));
        const int64_t e = scratch_elems(pairs[p].m, pairs[p].n, tm);
        if (e) {
            S.scratch_off[p] = S.scratch_elems;
            S.scratch_elems += e;
        }
    }
    return S;
}

slcs_status check_pairs(const slcs_pair_desc *pairs, int32_t npairs)
{
    if (npairs < 0) return fail(SLCS_ERR_INVALID, "npairs must be >= 0");
    if (npairs > 0 && !pairs) return fail(SLCS_ERR_INVALID, "pairs is null");
    for (int32_t p = 0; p < npairs; ++p) {
        const slcs_pair_desc &d = pairs[p];
        if (d.m < 0 || d.n < 0 || d.a_offset < 0 || d.b_offset < 0 || d.out_offset < 0)
            return fail(SLCS_ERR_INVALID, "pair " + std::to_string(p) + ": negative size or offset");
        if (int64_t(d.m) + d.n > INT32_MAX)
            return fail(SLCS_ERR_RANGE, "pair " + std::to_string(p) + ": m+n exceeds int32 strand ids");
    }
    return SLCS_OK;
}

} // namespace

void set_error(const std::string &msg) { g_last_error = msg; }
slcs_status fail(slcs_status s, const std::string &msg)
{
    g_last_error = msg;
    return s;
}
slcs_status cuda_fail(cudaError_t e, const char *what)
{
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return SLCS_ERR_DEVICE;
}
uint32_t *device_status_word() { return dev_state().dev_status; }
uint32_t *device_status_word_if_ready()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return nullptr;
    std::lock_guard<std::mutex> g(g_dev_mu);
    return g_dev[d].init ? g_dev[d].dev_status : nullptr;
}
int sm_count() { return dev_state().sms; }

// Pairs with an empty side have no cells: the strands keep their start ids.
static slcs_status write_identity(int32_t *h, int32_t m, int32_t *v, int32_t n, cudaStream_t st)
{
    if (m + n == 0) return SLCS_OK;
    identity_strands_kernel<<<(m + n + 255) / 256 < 1024 ? (m + n + 255) / 256 : 1024, 256, 0, st>>>(h, m, v, n);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

} // namespace slcs

using namespace slcs;

struct StreamClass {
    int tm, seg;  // rows per lane, lanes per segment
};

// Relative time of one step of a warp of a stream class (all its segments
// advance one column block), which sets how many warps the class gets.  A
// warp's pace is not its own instruction count: the warps of an SM
// sub-partition share its issue slots and integer pipe, so the classes differ
// less than their rows per lane do.  Fitted to B200 per-warp clocks of the
// 20,000 read/window pairs (4 columns per step): 32-lane classes of 12 and 16
// rows 1348 and 1500 ns.  Plans with 8 columns per step weigh every class
// alike (no measurements).
static double class_step_time(const StreamClass &k, int tns)
{
    if (tns != 4) return 1.0;
    if (k.seg == 32) return k.tm <= 12 ? 1348.0 : 1500.0;
    return 1000.0 + 30.0 * k.tm; // 16-lane classes: between the two above
}

// Head of a batch plan's work buffer: counters [0] wavefront ticket and [1]
// abort, [2] ticket of the staged bundles, [3] unused, then MAX_CLASSES pool
// tickets; the wavefront progress counters follow.
static constexpr int WORK_HEAD = 4 + MAX_CLASSES;

struct slcs_batch_plan {
    int device = 0;
    int tm = 8;      // rows per lane of the wavefront tasks
    int warps = 4;
    int stm = 0;     // rows per lane in stream mode (0: wavefront only)
    int seg = 16;    // lanes per stream segment
    int32_t npairs = 0;
    int32_t ntasks = 0;
    int32_t nstream = 0;
    int32_t npacked = 0; // stream pairs in packed classes
    int tns = 8;        // stream columns per step
    int blocks_per_sm = 0;
    std::vector<StreamClass> classes; // stream classes in preference order
    int32_t nclass = 0; // classes with warps
    int32_t class_warp_end[MAX_CLASSES] = {};
    int32_t class_code[MAX_CLASSES] = {};
    int32_t nwarps = 0; // warps with a stream class
    int grid = 0;       // blocks of the batch launch
    uint64_t wait_ns = DEFAULT_WAIT_NS;
    bool use_graph = false;
    char *d_block = nullptr; // every device array of the plan lies in it
    bool pooled = false;     // it is the plans' pool's
    PairDev *d_pairs = nullptr;
    int32_t *d_seg_off = nullptr;
    int32_t *d_seg_list = nullptr;
    int32_t *d_pool_list = nullptr;
    int32_t pool_off[MAX_CLASSES + 1] = {};
    int couple_tm = 0; // rows per lane of the packed pairs (0: none)
    int depth = 0;     // their warps per SM sub-partition (0: the default)
    CoupleDev *d_couples = nullptr;
    int32_t *d_others = nullptr; // pairs not in couples
    int32_t nothers = 0;
    int32_t nstaged = 0, ncouples = 0, nstaged_bundles = 0, nlists = 0;
    int32_t *d_list_off = nullptr; // of the bundles that are not staged
    uint4 *d_couple_stage = nullptr;
    BundleLane *d_bundles = nullptr;
    int pool_pct = 15;
    int2 *d_tasks = nullptr;
    int64_t *d_scr_off = nullptr;
    int32_t *d_scratch = nullptr;
    int32_t *d_work = nullptr; // [counters(4) | progress(ntasks)]
    size_t work_bytes = 0;
    // Pairs combed by the relay kernel: those too tall to stream (few of them
    // beside the couples, on a stream of their own and SMs left to them, else
    // after the others), or all of the plan.
    RelayShape relay{};
    bool relay_all = false;
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    int32_t nrelay = 0;         // groups of those pairs
    int32_t relay_sms = 0;      // SMs the couples leave to them
    int2 *d_relay = nullptr;    // (pair, group)
    int64_t *d_row_off = nullptr;
    int2 *d_duos = nullptr;         // the relay's pairs of pairs (two per register)
    int32_t nduos = 0;
    char *d_relay_ws = nullptr; // counters and hand-down rows, cleared by every run
    size_t relay_ws_bytes = 0;
    std::vector<slcs_pair_desc> empty_pairs; // pairs with m == 0 or n == 0
    cudaGraphExec_t gexec = nullptr;
    const void *g_a = nullptr, *g_b = nullptr, *g_out = nullptr;
    cudaStream_t cap_stream = nullptr;
    // Extents the descriptors reach (elements), checked by the host-pointer run.
    int64_t need_a = 0, need_b = 0, need_out = 0;
    bool wide = false;   // ids past the fast cell rule (wavefront launch only)
    int64_t max_ids = 0; // largest m + n of a pair (strand ids are below it)
    // Device int16 copy of the strands for slcs_batch_plan_run_host16, grown on demand.
    int16_t *d_out16 = nullptr;
    size_t out16_elems = 0;
    // Device staging of slcs_batch_plan_run_host, grown on demand.
    char *h_stage = nullptr;
    size_t h_stage_bytes = 0;
    // Host runs of large batches: the pairs in index order cut into chunks
    // with disjoint byte ranges of a, b and out, one sub-plan and one stream
    // each, so that one chunk's copies overlap another chunk's combing.
    struct Chunk {
        slcs_batch_plan *plan = nullptr;
        int64_t a_lo = 0, a_hi = 0, b_lo = 0, b_hi = 0, o_lo = 0, o_hi = 0;
        cudaStream_t stream = nullptr;
        cudaEvent_t done = nullptr;
    };
    std::vector<Chunk> chunks;
    cudaEvent_t chunk_start = nullptr;

    CombLaunch launch(const uint8_t *a, const uint8_t *b, int32_t *out) const
    {
        CombLaunch L{};
        L.pairs = d_pairs;
        L.tasks = d_tasks;
        L.ntasks = ntasks;
        L.a_blob = a;
        L.b_blob = b;
        L.out = out;
        L.scratch = d_scratch;
        L.scratch_off = d_scr_off;
        L.counters = d_work;
        L.progress = d_work + WORK_HEAD;
        L.status = device_status_word();
        L.wait_ns = wait_ns;
        L.wide = wide;
        return L;
    }

    // With out16 the couples' strands go there, as int16, and the others' to out.
    slcs_status enqueue(const uint8_t *a, const uint8_t *b, int32_t *out, int16_t *out16, cudaStream_t st) const
    {
        slcs_status s = SLCS_OK;
        if (relay_all) {
            s = enqueue_relay(a, b, out, st);
        } else if (!side) {
            s = enqueue_rest(a, b, out, out16, st);
            if (s == SLCS_OK) s = enqueue_relay(a, b, out, st);
        } else {
            SLCS_CUDA(cudaEventRecord(fork, st));
            SLCS_CUDA(cudaStreamWaitEvent(side, fork, 0));
            s = enqueue_relay(a, b, out, side);
            SLCS_CUDA(cudaEventRecord(join, side));
            if (s == SLCS_OK) s = enqueue_rest(a, b, out, out16, st);
            SLCS_CUDA(cudaStreamWaitEvent(st, join, 0));
        }
        if (s != SLCS_OK) return s;
        for (const auto &d : empty_pairs) {
            s = write_identity(out + d.out_offset, d.m, out + d.out_offset + d.m, d.n, st);
            if (s != SLCS_OK) return s;
        }
        return SLCS_OK;
    }

    slcs_status enqueue_relay(const uint8_t *a, const uint8_t *b, int32_t *out, cudaStream_t st) const
    {
        if (nrelay <= 0) return SLCS_OK;
        SLCS_CUDA(cudaMemsetAsync(d_relay_ws, 0, relay_ws_bytes, st));
        RelayLaunch L{};
        L.pairs = d_pairs;
        L.items = d_relay;
        L.nitems = nrelay;
        L.a_blob = a;
        L.b_blob = b;
        L.out = out;
        L.counters = reinterpret_cast<int32_t *>(d_relay_ws);
        L.rows = reinterpret_cast<int2 *>(d_relay_ws + 16);
        L.row_off = d_row_off;
        L.status = device_status_word();
        L.wait_ns = wait_ns;
        L.two = nduos > 0;
        L.duos = L.two ? d_duos : nullptr;
        return launch_relay(L, relay, sm_count(), st);
    }

    // The streamed pairs, or all pairs of a wavefront plan.
    slcs_status enqueue_rest(const uint8_t *a, const uint8_t *b, int32_t *out, int16_t *out16, cudaStream_t st) const
    {
        if (stm > 0 ? nstream <= 0 : ntasks <= 0) return SLCS_OK;
        if (stm <= 0 || nstaged > 0 || nwarps > 0) SLCS_CUDA(cudaMemsetAsync(d_work, 0, work_bytes, st));
        if (stm > 0) {
            CouplesLaunch C{a,      b,       out,            out16,           d_couples, nstaged, d_couple_stage,
                            d_bundles, nstaged_bundles, nlists, d_list_off, d_work + 2};
            if (ncouples > 0) {
                const slcs_status s = launch_couples(C, couple_tm, depth, relay_sms > 0, sm_count(), st);
                if (s != SLCS_OK) return s;
            }
            if (nwarps <= 0) return SLCS_OK;
            BatchLaunch B{launch(a, b, out), d_seg_off, d_seg_list, nwarps, grid, nclass, {}, {}};
            for (int c = 0; c < nclass; ++c) {
                B.class_warp_end[c] = class_warp_end[c];
                B.class_code[c] = class_code[c];
            }
            B.pool_list = d_pool_list;
            B.pool_ticket = d_work + 4;
            for (int c = 0; c <= MAX_CLASSES; ++c) B.pool_off[c] = pool_off[c];
            return launch_batch(B, tns, st, nullptr);
        }
        return launch_comb(launch(a, b, out), tm, warps, st, nullptr);
    }
};

extern "C" {

const char *slcs_last_error(void) { return g_last_error.c_str(); }

const char *slcs_status_string(slcs_status s)
{
    switch (s) {
    case SLCS_OK: return "ok";
    case SLCS_ERR_INVALID: return "invalid argument";
    case SLCS_ERR_ALLOC: return "allocation failed";
    case SLCS_ERR_DEVICE: return "CUDA error";
    case SLCS_ERR_TIMEOUT: return "device wait timed out";
    case SLCS_ERR_UNSUPPORTED: return "unsupported configuration";
    case SLCS_ERR_RANGE: return "size out of range";
    }
    return "unknown status";
}

int32_t slcs_version(void) { return 1; }

slcs_status slcs_set_device(int32_t device)
{
    SLCS_CUDA(cudaSetDevice(device));
    return SLCS_OK;
}

slcs_status slcs_device_name(int32_t device, char *buf, int32_t len)
{
    if (!buf || len <= 0) return fail(SLCS_ERR_INVALID, "null buffer");
    cudaDeviceProp prop;
    SLCS_CUDA(cudaGetDeviceProperties(&prop, device));
    std::strncpy(buf, prop.name, size_t(len) - 1);
    buf[len - 1] = '\0';
    return SLCS_OK;
}

void slcs_default_config(slcs_config *cfg)
{
    if (cfg) std::memset(cfg, 0, sizeof(*cfg));
}

slcs_status slcs_device_status(int32_t device, int32_t clear)
{
    int cur = 0;
    cudaGetDevice(&cur);
    if (device != cur) SLCS_CUDA(cudaSetDevice(device));
    DeviceState &s = dev_state();
    uint32_t bits = s.host_status ? __atomic_load_n(s.host_status, __ATOMIC_SEQ_CST) : 0;
    if (clear && s.host_status) __atomic_store_n(s.host_status, 0u, __ATOMIC_SEQ_CST);
    bits |= noalloc_status_bits(clear != 0);
    if (device != cur) cudaSetDevice(cur);
    if (bits & DEV_ERR_TIMEOUT) return fail(SLCS_ERR_TIMEOUT, "a device-side wait timed out");
    if (bits & DEV_ERR_INPUT) return fail(SLCS_ERR_INVALID, "a device-side input check failed (not a permutation)");
    if (bits) return fail(SLCS_ERR_DEVICE, "device status bits " + std::to_string(bits));
    return SLCS_OK;
}

static slcs_status comb_pair_relay(const uint8_t *a, int32_t m, const uint8_t *b, int32_t n, int32_t *h_out,
                                   int32_t *v_out, const RelayShape &shape, const slcs_config *cfg, cudaStream_t st)
{
    RelayLaunch L{};
    L.nitems = relay_groups(m, shape);
    L.a_blob = a;
    L.b_blob = b;
    L.out = h_out;
    L.v_single = v_out;
    L.status = device_status_word();
    L.wait_ns = wait_limit_ns(cfg);
    L.single.m = m;
    L.single.n = n;
    char *ws = nullptr;
    if (L.nitems > 1) { // one group hands nothing down
        const size_t bytes = 16 + sizeof(int2) * size_t(relay_row_elems(m, n, shape));
        SLCS_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&ws), bytes, st));
        const cudaError_t e = cudaMemsetAsync(ws, 0, bytes, st);
        if (e != cudaSuccess) {
            cudaFreeAsync(ws, st);
            return cuda_fail(e, "hand-down row");
        }
        L.counters = reinterpret_cast<int32_t *>(ws);
        L.rows = reinterpret_cast<int2 *>(ws + 16);
    }
    const slcs_status s = launch_relay(L, shape, sm_count(), st);
    if (ws) SLCS_CUDA(cudaFreeAsync(ws, st));
    return s;
}

slcs_status slcs_comb_pair(const uint8_t *a, int32_t m, const uint8_t *b, int32_t n, int32_t *h_out,
                           int32_t *v_out, const slcs_config *cfg, void *stream)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if ((m > 0 && (!a || !h_out)) || (n > 0 && (!b || !v_out)))
        return fail(SLCS_ERR_INVALID, "null pointer for a non-empty side");
    if (int64_t(m) + n > INT32_MAX) return fail(SLCS_ERR_RANGE, "m+n exceeds int32 strand ids");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (m == 0 || n == 0) return write_identity(h_out, m, v_out, n, st);
    (void)sm_count(); // per-device set-up (memory pool) before the first allocation
    PairPlan pp;
    const slcs_status ps = plan_pair(m, n, cfg, sm_count(), &pp);
    if (ps != SLCS_OK) return ps;
    if (pp.relay.relay.tm > 0) {
        if (pp.relay.strips * pp.relay.bands == 1)
            return comb_pair_relay(a, m, b, n, h_out, v_out, pp.relay.relay, cfg, st);
        slcs_config rc{};
        rc.strips = pp.relay.strips;
        rc.bands = pp.relay.bands;
        rc.braid_cutoff = cfg ? cfg->braid_cutoff : 0;
        rc.wait_ms = cfg ? cfg->wait_ms : 0;
        return comb_strips(a, m, b, n, h_out, v_out, &rc, 0, 0, &pp.relay.relay, st);
    }
    const int tm = pp.c.tile_m;
    if (pp.c.algo == SLCS_ALGO_STRIPS) return comb_strips(a, m, b, n, h_out, v_out, &pp.c, tm, pp.c.warps, nullptr, st);
    const int32_t ntasks = stripes_of(m, tm);
    const size_t work_bytes = align_up(sizeof(int32_t) * (4 + size_t(ntasks)), 256);
    const size_t scr_bytes = sizeof(int32_t) * size_t(scratch_elems(m, n, tm));
    void *ws = nullptr;
    SLCS_CUDA(cudaMallocAsync(&ws, work_bytes + scr_bytes + 16, st));
    int32_t *work = static_cast<int32_t *>(ws);
    SLCS_CUDA(cudaMemsetAsync(work, 0, work_bytes, st));
    CombLaunch L{};
    L.pairs = nullptr;
    L.tasks = nullptr;
    L.ntasks = ntasks;
    L.a_blob = a;
    L.b_blob = b;
    L.out = h_out;
    L.scratch = reinterpret_cast<int32_t *>(static_cast<char *>(ws) + work_bytes);
    L.scratch_off = nullptr;
    L.counters = work;
    L.progress = work + 4;
    L.status = device_status_word();
    L.wait_ns = wait_limit_ns(cfg);
    L.single.a_off = 0;
    L.single.b_off = 0;
    L.single.m = m;
    L.single.n = n;
    L.tw = pick_tw(tm, ntasks, n, b);
    L.wide = wide_ids(m, n, cfg);
    // h and v may live in separate allocations: address v relative to h.
    L.single.out_off = 0;
    slcs_status s;
    if (v_out == h_out + m) {
        s = launch_comb(L, tm, pp.c.warps, st, nullptr);
    } else {
        // Comb into a contiguous temporary, then copy v out.
        int32_t *tmp = nullptr;
        SLCS_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&tmp), sizeof(int32_t) * (size_t(m) + n), st));
        L.out = tmp;
        s = launch_comb(L, tm, pp.c.warps, st, nullptr);
        if (s == SLCS_OK) {
            SLCS_CUDA(cudaMemcpyAsync(h_out, tmp, sizeof(int32_t) * m, cudaMemcpyDeviceToDevice, st));
            SLCS_CUDA(cudaMemcpyAsync(v_out, tmp + m, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st));
        }
        SLCS_CUDA(cudaFreeAsync(tmp, st));
    }
    SLCS_CUDA(cudaFreeAsync(ws, st));
    return s;
}

// A stream and a page-locked buffer for one host-pointer call at a time.  A
// call takes an idle one (or makes one) and gives it back; at most LANES_KEPT
// stay.  (A stream made and destroyed per call, and pageable copies one by one,
// cost a small pair about 125 us.)
namespace {
struct HostLane {
    int device = -1;
    cudaStream_t st = nullptr;
    char *pinned = nullptr; // LANE_BYTES, or null when it could not be had
};
constexpr size_t LANE_BYTES = size_t(2) << 20;
constexpr size_t LANES_KEPT = 4;
std::mutex g_lane_mu;
std::vector<HostLane> g_lanes;

void drop_lane(HostLane &l)
{
    if (l.st) cudaStreamDestroy(l.st);
    if (l.pinned) cudaFreeHost(l.pinned);
    l = HostLane{};
}

slcs_status take_lane(HostLane *l)
{
    int dev = 0;
    SLCS_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> g(g_lane_mu);
        for (size_t i = 0; i < g_lanes.size(); ++i)
            if (g_lanes[i].device == dev) {
                *l = g_lanes[i];
                g_lanes.erase(g_lanes.begin() + long(i));
                return SLCS_OK;
            }
    }
    l->device = dev;
    SLCS_CUDA(cudaStreamCreateWithFlags(&l->st, cudaStreamNonBlocking));
    if (cudaHostAlloc(reinterpret_cast<void **>(&l->pinned), LANE_BYTES, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        l->pinned = nullptr;
    }
    return SLCS_OK;
}

// With its stream synchronised; after a failed call a lane is dropped.
void give_lane(HostLane &l, bool good)
{
    if (good) {
        std::lock_guard<std::mutex> g(g_lane_mu);
        if (g_lanes.size() < LANES_KEPT) {
            g_lanes.push_back(l);
            return;
        }
    }
    drop_lane(l);
}

// One pair from host memory: symbols of `width` bytes (1, or 4 for Words that
// become bytes on the device).
slcs_status comb_host(const void *a, int32_t m, const void *b, int32_t n, size_t width, int32_t *h_out, int32_t *v_out,
                      const slcs_config *cfg)
{
    const bool words = width > 1;
    HostLane lane;
    slcs_status s = take_lane(&lane);
    if (s != SLCS_OK) {
        drop_lane(lane);
        return s;
    }
    cudaStream_t st = lane.st;
    (void)sm_count(); // per-device set-up (memory pool) before the first allocation
    // Device: [a | b | strands | alphabet | a and b as bytes | symbol workspace];
    // the lane's buffer holds a and b, then strands and alphabet, in the same layout.
    const size_t na = width * size_t(m), nb = width * size_t(n);
    const size_t o_b = align_up(na + 16, 256), in_bytes = o_b + nb;
    const size_t o_out = align_up(in_bytes + 16, 256), n_out = sizeof(int32_t) * (size_t(m) + n);
    const size_t o_alpha = o_out + n_out, out_bytes = n_out + (words ? sizeof(int32_t) : 0);
    const size_t o_ab = align_up(o_out + out_bytes + 16, 256);
    const size_t o_bb = o_ab + (words ? align_up(size_t(m) + 16, 256) : 0);
    const size_t o_ws = o_bb + (words ? align_up(size_t(n) + 16, 256) : 0);
    char *buf = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&buf), o_ws + (words ? symbols_workspace_bytes() : 0), st);
    if (e != cudaSuccess) {
        give_lane(lane, true);
        return cuda_fail(e, "cudaMallocAsync");
    }
    char *pin = o_out + out_bytes <= LANE_BYTES ? lane.pinned : nullptr;
    if (pin) {
        if (m) std::memcpy(pin, a, na);
        if (n) std::memcpy(pin + o_b, b, nb);
        if (m > 0 || n > 0) e = cudaMemcpyAsync(buf, pin, in_bytes, cudaMemcpyHostToDevice, st);
    } else {
        if (m) e = cudaMemcpyAsync(buf, a, na, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess && n) e = cudaMemcpyAsync(buf + o_b, b, nb, cudaMemcpyHostToDevice, st);
    }
    const uint8_t *da = reinterpret_cast<uint8_t *>(buf), *db = reinterpret_cast<uint8_t *>(buf + o_b);
    int32_t *dout = reinterpret_cast<int32_t *>(buf + o_out), *dalpha = reinterpret_cast<int32_t *>(buf + o_alpha);
    int32_t alphabet = 0;
    if (words && e == cudaSuccess) {
        uint8_t *ab = reinterpret_cast<uint8_t *>(buf + o_ab), *bb = reinterpret_cast<uint8_t *>(buf + o_bb);
        s = symbols_to_bytes(reinterpret_cast<const int32_t *>(da), m, reinterpret_cast<const int32_t *>(db), n, ab, bb,
                             dalpha, buf + o_ws, st);
        da = ab;
        db = bb;
        // The alphabet decides before a long comb; a short one it comes back with.
        if (s == SLCS_OK && !(pin && int64_t(m) * n < (int64_t(1) << 28))) {
            e = cudaMemcpyAsync(&alphabet, dalpha, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
    }
    if (e == cudaSuccess && s == SLCS_OK && alphabet >= 0) {
        s = slcs_comb_pair(da, m, db, n, dout, dout + m, cfg, st);
        if (s == SLCS_OK && pin) {
            if (out_bytes) e = cudaMemcpyAsync(pin + o_out, dout, out_bytes, cudaMemcpyDeviceToHost, st);
        } else if (s == SLCS_OK) {
            if (m) e = cudaMemcpyAsync(h_out, dout, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess && n)
                e = cudaMemcpyAsync(v_out, dout + m, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st);
        }
    }
    const cudaError_t f = cudaFreeAsync(buf, st);
    if (e == cudaSuccess) e = f;
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess && s == SLCS_OK && pin) {
        if (words) std::memcpy(&alphabet, pin + o_alpha, sizeof(alphabet));
        if (alphabet >= 0) {
            if (m) std::memcpy(h_out, pin + o_out, sizeof(int32_t) * m);
            if (n) std::memcpy(v_out, pin + o_out + sizeof(int32_t) * m, sizeof(int32_t) * n);
        }
    }
    give_lane(lane, e == cudaSuccess);
    if (s != SLCS_OK) return s;
    if (e != cudaSuccess) return cuda_fail(e, "symbol or strand copies");
    if (alphabet < 0) return fail(SLCS_ERR_RANGE, "more than 256 distinct symbols in a and b");
    int dev = 0;
    cudaGetDevice(&dev);
    return slcs_device_status(dev, 1);
}
} // namespace

slcs_status slcs_comb_pair_host(const uint8_t *a, int32_t m, const uint8_t *b, int32_t n, int32_t *h_out,
                                int32_t *v_out, const slcs_config *cfg)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if ((m > 0 && (!a || !h_out)) || (n > 0 && (!b || !v_out)))
        return fail(SLCS_ERR_INVALID, "null pointer for a non-empty side");
    return comb_host(a, m, b, n, sizeof(uint8_t), h_out, v_out, cfg);
}

slcs_status slcs_symbols_to_bytes(const int32_t *a, int32_t m, const int32_t *b, int32_t n, uint8_t *a_out,
                                  uint8_t *b_out, int32_t *alphabet_out, void *stream)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if ((m > 0 && (!a || !a_out)) || (n > 0 && (!b || !b_out)) || !alphabet_out)
        return fail(SLCS_ERR_INVALID, "null symbol or output pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    (void)sm_count(); // per-device set-up (memory pool) before the first allocation
    void *ws = nullptr;
    SLCS_CUDA(cudaMallocAsync(&ws, symbols_workspace_bytes(), st));
    const slcs_status s = symbols_to_bytes(a, m, b, n, a_out, b_out, alphabet_out, ws, st);
    SLCS_CUDA(cudaFreeAsync(ws, st));
    return s;
}

slcs_status slcs_comb_pair_words_host(const int32_t *a, int32_t m, const int32_t *b, int32_t n, int32_t *h_out,
                                      int32_t *v_out, const slcs_config *cfg)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if ((m > 0 && (!a || !h_out)) || (n > 0 && (!b || !v_out)))
        return fail(SLCS_ERR_INVALID, "null pointer for a non-empty side");
    if (int64_t(m) + n > INT32_MAX) return fail(SLCS_ERR_RANGE, "m+n exceeds int32 strand ids");
    return comb_host(a, m, b, n, sizeof(int32_t), h_out, v_out, cfg);
}

static slcs_status plan_create_impl(slcs_batch_plan **plan_out, const slcs_pair_desc *pairs, int32_t npairs,
                                    const slcs_config *cfg, bool chunk = false);
static void plan_add_chunks(slcs_batch_plan *P, const slcs_pair_desc *pairs, int32_t npairs, const slcs_config *cfg);

slcs_status slcs_batch_plan_create(slcs_batch_plan **plan_out, const slcs_pair_desc *pairs, int32_t npairs,
                                   const slcs_config *cfg)
{
    slcs_status s = plan_create_impl(plan_out, pairs, npairs, cfg);
    if (s == SLCS_OK) plan_add_chunks(*plan_out, pairs, npairs, cfg);
    return s;
}

// Chunks for host runs (an optimisation only: without them run_host copies
// everything in, combs, and copies everything out).  Made for batches of at
// least CHUNK_MIN_PAIRS pairs whose chunks' byte ranges do not overlap.
// 4 chunks: the 20,000 reads' int16 host run took 0.42 ms, with 2, 3 and 6
// chunks 0.44, 0.43 and 0.44 ms (one B200; the copies alone take 0.38 ms one
// after the other, and every chunk costs the host a dozen calls).
static constexpr int HOST_CHUNKS = 4;
static constexpr int32_t CHUNK_MIN_PAIRS = 8192;

static void plan_add_chunks(slcs_batch_plan *P, const slcs_pair_desc *pairs, int32_t npairs, const slcs_config *cfg)
{
    if (npairs < CHUNK_MIN_PAIRS) return;
    int64_t cells = 0;
    for (int32_t p = 0; p < npairs; ++p) cells += int64_t(pairs[p].m) * pairs[p].n;
    std::vector<slcs_batch_plan::Chunk> ch;
    int32_t p0 = 0;
    int64_t acc = 0;
    for (int c = 0; c < HOST_CHUNKS && p0 < npairs; ++c) {
        int32_t p1 = p0;
        const int64_t target = cells * (c + 1) / HOST_CHUNKS;
        while (p1 < npairs && (acc < target || p1 == p0)) {
            acc += int64_t(pairs[p1].m) * pairs[p1].n;
            ++p1;
        }
        if (c == HOST_CHUNKS - 1) {
            for (; p1 < npairs; ++p1) acc += int64_t(pairs[p1].m) * pairs[p1].n;
        }
        slcs_batch_plan::Chunk k;
        k.a_lo = k.b_lo = k.o_lo = INT64_MAX;
        for (int32_t p = p0; p < p1; ++p) {
            const slcs_pair_desc &d = pairs[p];
            k.a_lo = std::min(k.a_lo, d.a_offset);
            k.a_hi = std::max(k.a_hi, d.a_offset + d.m);
            k.b_lo = std::min(k.b_lo, d.b_offset);
            k.b_hi = std::max(k.b_hi, d.b_offset + d.n);
            k.o_lo = std::min(k.o_lo, d.out_offset);
            k.o_hi = std::max(k.o_hi, d.out_offset + d.m + d.n);
        }
        // Sub-plan over the chunk's pairs (offsets stay global).
        if (plan_create_impl(&k.plan, pairs + p0, p1 - p0, cfg, true) != SLCS_OK) {
            for (auto &x : ch) slcs_batch_plan_destroy(x.plan);
            if (k.plan) slcs_batch_plan_destroy(k.plan);
            cudaGetLastError(); // not the next launch's
            return;
        }
        ch.push_back(k);
        p0 = p1;
    }
    // Ranges must not overlap (reads of one chunk may not see another's copy
    // still in flight, writes must not race).
    auto disjoint = [&](int64_t slcs_batch_plan::Chunk::*lo, int64_t slcs_batch_plan::Chunk::*hi) {
        std::vector<std::pair<int64_t, int64_t>> r;
        for (auto &x : ch) r.push_back({x.*lo, x.*hi});
        std::sort(r.begin(), r.end());
        for (size_t i = 1; i < r.size(); ++i)
            if (r[i].first < r[i - 1].second) return false;
        return true;
    };
    bool ok = ch.size() > 1 && disjoint(&slcs_batch_plan::Chunk::a_lo, &slcs_batch_plan::Chunk::a_hi) &&
              disjoint(&slcs_batch_plan::Chunk::b_lo, &slcs_batch_plan::Chunk::b_hi) &&
              disjoint(&slcs_batch_plan::Chunk::o_lo, &slcs_batch_plan::Chunk::o_hi);
    for (auto &x : ch) {
        if (!ok) break;
        ok = cudaStreamCreateWithFlags(&x.stream, cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&x.done, cudaEventDisableTiming) == cudaSuccess;
    }
    if (ok) ok = cudaEventCreateWithFlags(&P->chunk_start, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        for (auto &x : ch) {
            slcs_batch_plan_destroy(x.plan);
            if (x.stream) cudaStreamDestroy(x.stream);
            if (x.done) cudaEventDestroy(x.done);
        }
        if (P->chunk_start) cudaEventDestroy(P->chunk_start);
        P->chunk_start = nullptr;
        return;
    }
    P->chunks = std::move(ch);
}

// Bundles in the order they were made, with what they have left: the first one
// with at least so much in a few steps (a tree of maxima).
struct FirstWith {
    size_t cap = 0;
    std::vector<int32_t> t;

    void set(int32_t i, int32_t left)
    {
        if (size_t(i) >= cap) {
            const size_t grown = std::max<size_t>(cap ? 2 * cap : 16, size_t(i) + 1);
            size_t c = 16;
            while (c < grown) c *= 2;
            std::vector<int32_t> x(2 * c, -1);
            std::copy(t.begin() + long(cap), t.end(), x.begin() + long(c));
            for (size_t k = c - 1; k > 0; --k) x[k] = std::max(x[2 * k], x[2 * k + 1]);
            t.swap(x);
            cap = c;
        }
        size_t k = cap + size_t(i);
        t[k] = left;
        while (k >>= 1) t[k] = std::max(t[2 * k], t[2 * k + 1]);
    }
    int32_t find(int32_t least) const // -1: none
    {
        if (cap == 0 || t[1] < least) return -1;
        size_t k = 1;
        while (k < cap) k = t[2 * k] >= least ? 2 * k : 2 * k + 1;
        return int32_t(k - cap);
    }
};

// Bundles of couples [k0, k1) side by side in a warp: longest couple first,
// each into the first bundle with lanes left whose length it comes near (within
// BUNDLE_SLACK), else into a new one; at most `blocks` blocks together.
// (100,000 pairs of 300 rows, whose couples fill no bundle, took 1.9 s with all
// bundles in one list, and take 0.05 s.)
static void make_bundles(const std::vector<CoupleDev> &couples, size_t k0, size_t k1, int tm, int32_t blocks,
                         std::vector<BundleLane> &out)
{
    constexpr double BUNDLE_SLACK = 0.6; // 0.85 left 5 % more steps on the 20,000 reads
    struct Open {
        int32_t index, room, steps, used;
    };
    std::vector<Open> made;
    FirstWith left[32]; // per lanes left, the blocks left
    auto lanes_of = [&](const CoupleDev &k) { return k.rows / tm; };
    auto steps_of = [&](const CoupleDev &k) { return k.nb + lanes_of(k) - 1; };
    std::vector<int32_t> order(k1 - k0);
    std::iota(order.begin(), order.end(), int32_t(k0));
    std::stable_sort(order.begin(), order.end(),
                     [&](int32_t x, int32_t y) { return steps_of(couples[x]) > steps_of(couples[y]); });
    size_t closed = 0; // bundles too long for this couple, and so for the rest
    for (int32_t i : order) {
        const CoupleDev &k = couples[size_t(i)];
        const int lanes = lanes_of(k), steps = steps_of(k);
        for (; closed < made.size() && double(made[closed].steps) * BUNDLE_SLACK > double(steps); ++closed)
            if (made[closed].room > 0) left[made[closed].room].set(int32_t(closed), -1);
        int32_t first = -1;
        for (int room = lanes; room < 32; ++room) {
            const int32_t f = left[room].find(k.nb);
            if (f >= 0 && (first < 0 || f < first)) first = f;
        }
        if (first < 0) {
            first = int32_t(made.size());
            made.push_back({int32_t(out.size() / 32), 32, steps, 0});
            out.insert(out.end(), 32, BundleLane{-1, 0, 1, 0, steps});
        } else {
            left[made[size_t(first)].room].set(first, -1);
        }
        Open &o = made[size_t(first)];
        BundleLane *b = &out[size_t(o.index) * 32 + size_t(32 - o.room)];
        for (int l = 0; l < lanes; ++l) b[l] = BundleLane{i, int16_t(l), int16_t(lanes), o.used, o.steps};
        o.room -= lanes;
        o.used += k.nb;
        if (o.room > 0) left[o.room].set(first, blocks - o.used);
    }
}

// Deal the bundles from the first on out to at most `most` lists, longest
// first to the least loaded one, and put them in the order of the lists;
// off: where each list starts among them, and their number.
static void deal_bundles(std::vector<BundleLane> &lanes, size_t first, int most, std::vector<int32_t> &off)
{
    const size_t count = lanes.size() / 32 - first;
    const size_t nlists = std::min(count, size_t(most));
    off.assign(1, 0);
    if (count == 0) return;
    constexpr int64_t BUNDLE_COST = 12; // filling and emptying a bundle, in steps
    std::vector<int32_t> order(count);
    std::iota(order.begin(), order.end(), 0);
    auto steps = [&](int32_t k) { return lanes[(first + size_t(k)) * 32].steps; };
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return steps(x) > steps(y); });
    using Load = std::pair<int64_t, int32_t>;
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
    for (size_t l = 0; l < nlists; ++l) heap.push({0, int32_t(l)});
    std::vector<std::vector<int32_t>> list(nlists);
    for (int32_t k : order) {
        Load top = heap.top();
        heap.pop();
        list[size_t(top.second)].push_back(k);
        top.first += steps(k) + BUNDLE_COST;
        heap.push(top);
    }
    std::vector<BundleLane> dealt;
    dealt.reserve(count * 32);
    for (const auto &l : list) {
        for (int32_t k : l) {
            const auto b = lanes.begin() + long((first + size_t(k)) * 32);
            dealt.insert(dealt.end(), b, b + 32);
        }
        off.push_back(int32_t(dealt.size() / 32));
    }
    std::copy(dealt.begin(), dealt.end(), lanes.begin() + long(first * 32));
}

static slcs_status plan_create_impl(slcs_batch_plan **plan_out, const slcs_pair_desc *pairs, int32_t npairs,
                                    const slcs_config *cfg, bool chunk)
{
    if (!plan_out) return fail(SLCS_ERR_INVALID, "plan is null");
    *plan_out = nullptr;
    slcs_status s = check_pairs(pairs, npairs);
    if (s != SLCS_OK) return s;
    auto *P = new (std::nothrow) slcs_batch_plan();
    if (!P) return fail(SLCS_ERR_ALLOC, "plan allocation");
    cudaGetDevice(&P->device);
    // Typical m: the median of the batch.
    std::vector<int32_t> ms;
    ms.reserve(npairs);
    int64_t cells = 0;
    for (int32_t p = 0; p < npairs; ++p) {
        ms.push_back(pairs[p].m);
        cells += int64_t(pairs[p].m) * pairs[p].n;
    }
    int32_t med = 0;
    if (!ms.empty()) {
        std::nth_element(ms.begin(), ms.begin() + ms.size() / 2, ms.end());
        med = ms[ms.size() / 2];
    }
    P->warps = pick_warps(cfg, pick_tile_m(cfg, med, cells));
    P->use_graph = cfg && cfg->use_graph;
    P->wait_ns = wait_limit_ns(cfg);
    P->npairs = npairs;
    const bool wavefront_only = cfg && cfg->algo == SLCS_ALGO_WAVEFRONT;
    if (wavefront_only) {
        P->tm = pick_tile_m(cfg, med, cells);
        if (!tile_m_supported(P->tm)) {
            delete P;
            return fail(SLCS_ERR_UNSUPPORTED, "tile_m must be one of 2, 4, 8, 12, 14, 16");
        }
    } else {
        // Stream mode: pairs of at most 512 rows stream through segments,
        // each pair in the smallest class whose segment holds all its rows;
        // taller pairs are the relay kernel's (P->tm only counts their stripes).
        // A configuration naming tile_m (and seg) asks for that one class.
        P->tm = BATCH_WF_TM;
        const int bits = cfg ? cfg->strand_bits : 0;
        if (bits != 0 && bits != 16 && bits != 32) {
            delete P;
            return fail(SLCS_ERR_UNSUPPORTED, "strand_bits must be 0, 16 or 32");
        }
        // Two pairs per register (4 columns per step) when some pair fits a
        // packed class; otherwise 8 columns per step by default.
        bool packable = false;
        for (int32_t p = 0; p < npairs && !packable; ++p)
            packable = pairs[p].m > 0 && pairs[p].m <= 256 && int64_t(pairs[p].m) + pairs[p].n <= PACKED16_MAX_IDS;
        P->tns = (cfg && cfg->tile_n) ? cfg->tile_n : (bits != 32 && packable ? 4 : 8);
        if (P->tns != 4 && P->tns != 8) {
            delete P;
            return fail(SLCS_ERR_UNSUPPORTED, "stream mode needs tile_n 4 or 8");
        }
        // Long packed pairs are staged in 8 bytes per row and column of a couple;
        // batches beyond 16 GiB of that comb 32-bit strands.
        int64_t ids = 0;
        for (int32_t p = 0; p < npairs; ++p) ids += int64_t(pairs[p].m) + pairs[p].n + 64;
        const bool pack = bits != 32 && P->tns == 4 && 8 * ids < (int64_t(16) << 30);
        // Packed pairs are combed in couples of as many lanes as their rows
        // need, 16 rows per lane; a configuration naming tile_m (and 16 lanes)
        // asks for couples of 16 lanes of that height.
        if (cfg && cfg->tile_m) {
            P->stm = cfg->tile_m;
            P->seg = cfg->seg ? cfg->seg : 16;
            if (pack && packed16_supported(P->stm, P->seg)) P->couple_tm = P->stm;
            P->classes.push_back({P->stm, P->seg});
        } else {
            P->stm = 16;
            P->seg = 16;
            if (pack) P->couple_tm = COUPLE_TM;
            for (int t : {4, 8, 12, 16}) P->classes.push_back({t, 16});
            P->classes.push_back({12, 32});
            P->classes.push_back({16, 32});
        }
        for (const auto &c : P->classes)
            if (!stream_variant_supported(c.tm, c.seg)) {
                delete P;
                return fail(SLCS_ERR_UNSUPPORTED, "stream mode needs tile_m in {4,8,12,16} and seg in {8,16,32}");
            }
        // 32-bit classes run at full occupancy (2 blocks per SM: 361 -> 420 us
        // on the 20,000 reads) with 15 % of a class's work in its pool.
        P->blocks_per_sm = (cfg && cfg->blocks_per_sm > 0) ? cfg->blocks_per_sm : 0;
        P->depth = P->blocks_per_sm;
        P->pool_pct = 15;
        if (cfg && cfg->pool_pct != 0) P->pool_pct = cfg->pool_pct < 0 ? 0 : std::min(cfg->pool_pct, 90);
    }
    for (int32_t p = 0; p < npairs; ++p) {
        if (pairs[p].m == 0 || pairs[p].n == 0) P->empty_pairs.push_back(pairs[p]);
        P->need_a = std::max<int64_t>(P->need_a, pairs[p].a_offset + pairs[p].m);
        P->need_b = std::max<int64_t>(P->need_b, pairs[p].b_offset + pairs[p].n);
        P->need_out = std::max<int64_t>(P->need_out, pairs[p].out_offset + pairs[p].m + pairs[p].n);
        P->max_ids = std::max<int64_t>(P->max_ids, int64_t(pairs[p].m) + pairs[p].n);
    }
    P->wide = wide_ids(P->max_ids, 0, wavefront_only ? cfg : nullptr);
    if (P->wide && !wavefront_only) { // the batch kernel has only the fast cell rule
        P->stm = 0;
        P->couple_tm = 0;
        P->classes.clear();
    }
    int32_t stream_rows = 0;
    for (const auto &c : P->classes) stream_rows = std::max(stream_rows, c.tm * c.seg);
    Schedule S = build_schedule(pairs, npairs, P->tm, stream_rows);
    P->ntasks = int32_t(S.tasks.size());
    // One-time device set-up now, so a graph capture in run() issues only
    // capturable work: the mapped status word and the occupancy queries.
    device_status_word();
    int full_grid = 0;
    {
        CombLaunch dummy{};
        dummy.ntasks = 1;
        dummy.wide = P->wide;
        slcs_status ps = P->stm > 0 ? launch_batch(BatchLaunch{dummy}, P->tns, PREPARE_ONLY, &full_grid)
                                    : launch_comb(dummy, P->tm, P->warps, PREPARE_ONLY, nullptr);
        if (ps == SLCS_OK && P->couple_tm > 0) ps = launch_couples(CouplesLaunch{}, P->couple_tm, 0, false, 1, PREPARE_ONLY);
        if (ps != SLCS_OK) {
            delete P;
            return ps;
        }
    }
    P->nstream = int32_t(S.stream_pairs.size());
    // The pairs too tall to stream: the relay shape, and whether a quarter of
    // the SMs holds all their groups.
    const int sms = sm_count();
    auto tall = [&](int32_t p) { return pairs[p].m > stream_rows; };
    const bool may_two = P->stm > 0 && !(cfg && cfg->strand_bits == 32);
    BatchRelay relay;
    if (P->stm > 0 && P->ntasks > 0) {
        relay = plan_batch_relay(pairs, npairs, may_two, sms, tall);
        if (relay.groups <= sms / 4) P->relay_sms = int32_t(relay.groups);
    }
    // Couples of the packed pairs and their bundles.
    std::vector<CoupleDev> couples;
    std::vector<BundleLane> bundle_lanes;
    std::vector<int32_t> list_off;
    int64_t stage_elems = COUPLE_HEAD;
    std::vector<int32_t> single_pairs; // streamed with 32-bit strands, largest first
    std::vector<char> in_couple(size_t(npairs), 0);
    {
        const int tm = P->couple_tm;
        const int fixed = cfg && cfg->tile_m ? 16 : 0; // lanes of a couple when the configuration says
        std::vector<std::pair<int, int32_t>> packed;   // (lanes, pair)
        for (int32_t p : S.stream_pairs) {
            const int lanes = tm > 0 ? (fixed ? fixed : (pairs[p].m + tm - 1) / tm) : 0;
            if (tm > 0 && pairs[p].m <= lanes * tm && lanes <= 32 && pairs[p].m + pairs[p].n <= PACKED16_MAX_IDS)
                packed.push_back({lanes, p}), in_couple[size_t(p)] = 1;
            else
                single_pairs.push_back(p);
        }
        P->npacked = int32_t(packed.size());
        // Pairs of as many lanes and about as many columns go together.
        std::sort(packed.begin(), packed.end(), [&](const std::pair<int, int32_t> &x, const std::pair<int, int32_t> &y) {
            if (x.first != y.first) return x.first > y.first;
            if (pairs[x.second].n != pairs[y.second].n) return pairs[x.second].n > pairs[y.second].n;
            return x.second < y.second;
        });
        for (size_t i = 0; i < packed.size(); ++i) {
            CoupleDev k{};
            std::memcpy(&k.a, &pairs[packed[i].second], sizeof(k.a));
            k.rows = tm * packed[i].first;
            k.nb = (k.a.n + 3) / 4; // the longer of the two
            if (i + 1 < packed.size() && packed[i + 1].first == packed[i].first)
                std::memcpy(&k.b, &pairs[packed[++i].second], sizeof(k.b));
            couples.push_back(k);
        }
        // The staged ones first: those that do not fit, and those so long for
        // their lanes that bundles of them would leave lanes idle (2,000
        // pairs of 300 x 3000: 262 us staged, 440 with a couple to a bundle).
        const auto mid = std::stable_partition(couples.begin(), couples.end(), [&](const CoupleDev &k) {
            return k.nb > BUNDLE_BLOCKS || int64_t(k.nb) * 24 > int64_t(BUNDLE_BLOCKS) * (k.rows / tm);
        });
        P->nstaged = int32_t(mid - couples.begin());
        P->ncouples = int32_t(couples.size());
        for (int32_t i = 0; i < P->nstaged; ++i) {
            CoupleDev &k = couples[size_t(i)];
            k.off = int32_t(stage_elems);
            stage_elems += int64_t(k.rows) / 2 + 2 * int64_t(k.nb);
        }
        make_bundles(couples, 0, size_t(P->nstaged), tm, INT32_MAX, bundle_lanes);
        P->nstaged_bundles = int32_t(bundle_lanes.size() / 32);
        make_bundles(couples, size_t(P->nstaged), couples.size(), tm, BUNDLE_BLOCKS, bundle_lanes);
        if (P->relay_sms > 0) {
            // Beside couples the relay kernel need not be fast but few: its
            // groups keep their SMs to themselves, and the couples take about
            // 0.22 us a step and sub-partition.  (20,000 reads, 7 of
            // them taller: 14 SMs for those 117 us, 4 SMs 106 us.)
            double steps = 0;
            for (size_t i = 0; i < bundle_lanes.size(); i += 32) steps += bundle_lanes[i].steps + 12.0;
            relay = plan_batch_relay(pairs, npairs, may_two, sms, tall, 0.7 * 0.22 * steps / (4.0 * sms));
            P->relay_sms = int32_t(relay.groups);
        }
        deal_bundles(bundle_lanes, P->nstaged_bundles, 4 * (sm_count() - P->relay_sms), list_off);
        P->nlists = int32_t(list_off.size()) - 1;
    }
    // Stream classes, warps and pair lists of the other pairs.  A pair costs
    // its column blocks plus a switch; each class gets warps in proportion to
    // its cost per warp (a warp runs 32/seg segments side by side), and within
    // a class the pairs go longest first to the least loaded segment.  The grid
    // is the persistent one (or blocks_per_sm per SM), fewer for small batches.
    std::vector<int32_t> seg_off, seg_list, pool_list;
    if (!single_pairs.empty()) {
        const int occ_blocks = std::max(1, full_grid / std::max(1, sm_count()));
        int grid = sm_count() * (P->blocks_per_sm > 0 ? std::min(P->blocks_per_sm, occ_blocks) : occ_blocks);
        const int nclass = int(P->classes.size());
        std::vector<std::vector<int32_t>> items(nclass);
        for (int32_t p : single_pairs) {
            int c = 0;
            while (c < nclass && pairs[p].m > P->classes[c].tm * P->classes[c].seg) ++c;
            if (c == nclass) { // cannot happen: stream_rows is the tallest class
                delete P;
                return fail(SLCS_ERR_INVALID, "internal: no stream class for a pair");
            }
            items[c].push_back(p);
        }
        // Cost of a pair: its column blocks plus a pair switch, in steps.
        auto cost = [&](int32_t p) { return int64_t((pairs[p].n + P->tns - 1) / P->tns) + 2; };
        // Per class: its steps in total, its longest pair, and how many warps
        // (of 32 / seg segments) can have work at all.
        std::vector<double> csteps(nclass, 0.0), clong(nclass, 0.0);
        std::vector<long> umax(nclass, 0);
        auto unit_segs = [&](int c) { return 32 / P->classes[c].seg; };
        long want = 0;
        for (int c = 0; c < nclass; ++c) {
            for (int32_t p : items[c]) {
                csteps[c] += double(cost(p));
                clong[c] = std::max(clong[c], double(cost(p)));
            }
            umax[c] = (long(items[c].size()) + unit_segs(c) - 1) / unit_segs(c);
            want += umax[c];
        }
        grid = int(std::max<long>(1, std::min<long>(grid, (want + BATCH_WARPS - 1) / BATCH_WARPS)));
        const long warps_total = long(grid) * BATCH_WARPS;
        // Warps per class so that the classes end together.  A class of u
        // warps ends about when each of its segments has combed its share of
        // the class's steps and the last one its longest pair, half of which
        // is still to go on average: end(u) = t * (S / (u * segments per
        // warp) + L / 2), t the class's time per step.  Each warp goes to the
        // class that would end last, while the warps last.
        std::vector<long> uc(nclass, 0);
        auto class_end = [&](int c, long u) {
            return class_step_time(P->classes[c], P->tns) * (csteps[c] / double(u * unit_segs(c)) + clong[c] / 2.0);
        };
        long used = 0;
        for (int c = 0; c < nclass; ++c)
            if (!items[c].empty()) ++used, uc[c] = 1;
        while (used < warps_total) {
            int worst = -1;
            double worst_end = -1.0;
            for (int c = 0; c < nclass; ++c) {
                if (uc[c] == 0 || uc[c] >= umax[c]) continue;
                const double e = class_end(c, uc[c]);
                if (e > worst_end) {
                    worst_end = e;
                    worst = c;
                }
            }
            if (worst < 0) break; // every class has a warp per 32 / seg pairs
            ++uc[worst];
            ++used;
        }
        P->grid = int(std::max<long>(grid, (used + BATCH_WARPS - 1) / BATCH_WARPS));
        std::vector<std::vector<int32_t>> slot_lists(size_t(used) * SEG_SLOTS);
        long wbase = 0;
        for (int c = 0; c < nclass; ++c) {
            if (uc[c] == 0) continue;
            const int spw = unit_segs(c), k = P->nclass++;
            const long nseg = uc[c] * spw;
            using Load = std::pair<int64_t, int64_t>;
            std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
            for (long sgi = 0; sgi < nseg; ++sgi) heap.push({0, sgi});
            std::stable_sort(items[c].begin(), items[c].end(),
                             [&](int32_t x, int32_t y) { return cost(x) > cost(y); });
            // Longest first to the least loaded segment until every segment
            // holds (100 - pool_pct) % of the class's average load; the rest,
            // the shortest pairs, form the class's pool, which segments claim
            // one pair at a time when their lists run out, so that the class
            // ends evenly whatever the real speed of its segments.
            const double cap = (100 - P->pool_pct) / 100.0 * csteps[c] / double(nseg);
            P->pool_off[k] = int32_t(pool_list.size());
            for (int32_t p : items[c]) {
                Load top = heap.top();
                if (P->pool_pct > 0 && double(top.first) >= cap) {
                    pool_list.push_back(p);
                    continue;
                }
                heap.pop();
                slot_lists[size_t((wbase + top.second / spw) * SEG_SLOTS + top.second % spw)].push_back(p);
                top.first += cost(p);
                heap.push(top);
            }
            wbase += uc[c];
            P->class_warp_end[k] = int32_t(wbase);
            P->class_code[k] = P->classes[c].tm * 100 + P->classes[c].seg;
        }
        for (int k = P->nclass; k <= MAX_CLASSES; ++k) P->pool_off[k] = int32_t(pool_list.size());
        P->nwarps = int32_t(used);
        seg_off.push_back(0);
        for (const auto &l : slot_lists) {
            seg_list.insert(seg_list.end(), l.begin(), l.end());
            seg_off.push_back(int32_t(seg_list.size()));
        }
    }
    // Relay items: the groups of every pair that does not stream (all pairs
    // when the relay kernel takes the whole plan), largest pair first.
    std::vector<int2> relay_items;
    std::vector<int64_t> row_off;
    // Without a configuration the relay kernel takes a whole batch where it is
    // predicted to end first: few pairs, or tall or wide ones, leave a warp of
    // couples a chain of its own.  Of couples, a step of a chain takes about 0.22
    // us and a step in all 0.22 us of a sub-partition; of streamed 32-bit pairs,
    // about three times that.  (20,000 reads: 115 us in couples, 361 by relay;
    // 4,000: 54 and 81; 1,000: 51 and 43; 64: 47 and 25; 64 pairs of 400 x 5000:
    // 390 in staged couples, 76 by relay.)
    if (P->stm > 0) {
        double chain = 0, steps = 0;
        for (size_t i = 0; i < bundle_lanes.size(); i += 32) {
            const bool staged = i / 32 < size_t(P->nstaged_bundles);
            chain = std::max(chain, (staged ? 0.3 : 0.22) * bundle_lanes[i].steps);
            steps += 0.22 * (bundle_lanes[i].steps + 12.0);
        }
        for (int32_t p : single_pairs) {
            chain = std::max(chain, 0.66 * (pairs[p].n / double(P->tns) + 32.0));
            steps += 0.33 * (pairs[p].n / double(P->tns) + 2.0);
        }
        double us = P->nstream > 0 ? (P->nstaged > 0 ? 25.0 : 10.0) + std::max(chain, steps / (4.0 * sms)) : 0.0;
        us = P->relay_sms > 0 ? std::max(us, relay.us) : us + relay.us;
        // (A chunk of a host run shares the GPU with the others: couples take less
        // of it.)
        const bool plain = chunk ? false : !cfg || (cfg->algo == SLCS_ALGO_AUTO && cfg->tile_m == 0 && cfg->tile_n == 0 &&
                                    cfg->warps == 0 && cfg->seg == 0 && cfg->blocks_per_sm == 0 &&
                                    cfg->strand_bits == 0 && cfg->pool_pct == 0);
        BatchRelay all;
        if (P->nstream > 0 && plain) all = plan_batch_relay(pairs, npairs, may_two, sms, [](int32_t) { return true; });
        if (P->nstream == 0 || (plain && all.us < us)) {
            P->relay_all = P->nstream + P->ntasks > 0;
            if (P->nstream > 0) relay = std::move(all);
        }
    }
    if (P->relay_all || (P->stm > 0 && P->ntasks > 0)) {
        P->relay = relay.shape;
        P->nduos = int32_t(relay.duos.size());
        RelayLaunch prepare{};
        prepare.two = P->nduos > 0;
        const slcs_status rs = launch_relay(prepare, P->relay, sm_count(), PREPARE_ONLY);
        if (rs != SLCS_OK) {
            delete P;
            return rs;
        }
        int64_t row_elems = 0;
        auto add = [&](int32_t i, int32_t m, int32_t n) { // pair or duo i
            const int32_t groups = relay_groups(m, P->relay);
            for (int32_t g = 0; g < groups; ++g) relay_items.push_back(make_int2(i, g));
            row_off[size_t(i)] = row_elems;
            row_elems += relay_row_elems(m, n, P->relay);
        };
        if (P->nduos > 0) { // sorted largest first
            row_off.assign(relay.duos.size(), 0);
            for (int32_t i = 0; i < P->nduos; ++i) {
                const int2 d = relay.duos[size_t(i)];
                const slcs_pair_desc &x = pairs[d.x], &y = pairs[d.y >= 0 ? d.y : d.x];
                add(i, std::max(x.m, y.m), std::max(x.n, y.n));
            }
        } else {
            row_off.assign(npairs, 0);
            for (int32_t p : S.order) {
                if (pairs[p].m == 0 || pairs[p].n == 0 || (!P->relay_all && pairs[p].m <= stream_rows)) continue;
                add(p, pairs[p].m, pairs[p].n);
            }
        }
        P->nrelay = int32_t(relay_items.size());
        P->relay_ws_bytes = 16 + sizeof(int2) * size_t(row_elems);
    }
    P->work_bytes = align_up(sizeof(int32_t) * (WORK_HEAD + (P->stm > 0 ? 0 : S.tasks.size())), 256);
    // One device block for the plan: what is uploaded first, then the work
    // areas (an allocation and a copy for each array took a third of the time
    // to make a plan).
    std::vector<char> up;
    size_t bytes = 0;
    auto place = [&](auto **ptr, size_t count) {
        const size_t at = align_up(bytes, 256);
        bytes = at + sizeof(**ptr) * count;
        *ptr = reinterpret_cast<std::remove_pointer_t<decltype(ptr)>>(at); // an offset until the block exists
        return at;
    };
    auto upload = [&](auto **ptr, const void *src, size_t count) {
        const size_t at = place(ptr, count);
        up.resize(bytes);
        if (count) std::memcpy(up.data() + at, src, sizeof(**ptr) * count);
    };
    static const uint32_t masked_block[4 * COUPLE_HEAD] = {0x01000100u, 0x01000100u, 0x01000100u, 0x01000100u,
                                                           0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu, 0x7FFF7FFFu};
    const bool stream = !P->relay_all && P->stm > 0;
    if (P->relay_all) P->nstaged = P->ncouples = P->nstaged_bundles = P->nlists = P->nwarps = 0;
    upload(&P->d_pairs, pairs, size_t(npairs));
    upload(&P->d_relay, relay_items.data(), relay_items.size());
    upload(&P->d_row_off, row_off.data(), row_off.size());
    upload(&P->d_duos, relay.duos.data(), size_t(P->nduos));
    upload(&P->d_seg_off, seg_off.data(), stream ? seg_off.size() : 0);
    upload(&P->d_seg_list, seg_list.data(), stream ? seg_list.size() : 0);
    upload(&P->d_pool_list, pool_list.data(), stream ? pool_list.size() : 0);
    std::vector<int32_t> others;
    if (P->ncouples > 0)
        for (int32_t p = 0; p < npairs; ++p)
            if (!in_couple[size_t(p)]) others.push_back(p);
    P->nothers = int32_t(others.size());
    upload(&P->d_others, others.data(), others.size());
    upload(&P->d_couples, couples.data(), size_t(P->ncouples));
    upload(&P->d_bundles, bundle_lanes.data(), P->ncouples > 0 ? bundle_lanes.size() : 0);
    upload(&P->d_list_off, list_off.data(), P->nlists > 0 ? list_off.size() : 0);
    upload(&P->d_tasks, S.tasks.data(), P->stm > 0 ? 0 : S.tasks.size());
    upload(&P->d_scr_off, S.scratch_off.data(), P->stm > 0 ? 0 : S.scratch_off.size());
    upload(&P->d_couple_stage, masked_block, P->nstaged > 0 ? COUPLE_HEAD : 0);
    if (P->nstaged > 0) bytes += sizeof(uint4) * size_t(stage_elems - COUPLE_HEAD); // the couples, after the block
    place(&P->d_scratch, P->stm > 0 ? 0 : size_t(S.scratch_elems));
    place(&P->d_work, P->work_bytes / sizeof(int32_t));
    place(&P->d_relay_ws, P->relay_ws_bytes);
    // From the plans' pool (a cudaMalloc beyond a megabyte maps memory, about
    // 300 us a plan).  The block and what is copied to it are there when the
    // stream has synchronised: runs may use streams that do not wait for it.
    P->pooled = dev_state().plan_pool != nullptr;
    cudaError_t e = P->pooled ? cudaMallocFromPoolAsync(reinterpret_cast<void **>(&P->d_block), std::max<size_t>(bytes, 256),
                                                        dev_state().plan_pool, nullptr)
                              : cudaMalloc(reinterpret_cast<void **>(&P->d_block), std::max<size_t>(bytes, 256));
    auto rebase = [&](auto *&ptr) {
        ptr = e == cudaSuccess ? reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(
                                     P->d_block + reinterpret_cast<uintptr_t>(ptr))
                               : nullptr;
    };
    rebase(P->d_pairs);
    rebase(P->d_relay);
    rebase(P->d_row_off);
    rebase(P->d_duos);
    rebase(P->d_seg_off);
    rebase(P->d_seg_list);
    rebase(P->d_pool_list);
    rebase(P->d_others);
    rebase(P->d_couples);
    rebase(P->d_bundles);
    rebase(P->d_list_off);
    rebase(P->d_tasks);
    rebase(P->d_scr_off);
    rebase(P->d_couple_stage);
    rebase(P->d_scratch);
    rebase(P->d_work);
    rebase(P->d_relay_ws);
    if (e == cudaSuccess && !up.empty())
        e = cudaMemcpyAsync(P->d_block, up.data(), up.size(), cudaMemcpyHostToDevice, nullptr);
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
    if (P->nrelay > 0 && !P->relay_all && P->relay_sms > 0 && P->nstream > 0) {
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&P->side, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&P->fork, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&P->join, cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        slcs_batch_plan_destroy(P);
        if (e == cudaErrorMemoryAllocation && !wavefront_only && !chunk) {
            // No room for staged couples or hand-down rows: wavefront plans need
            // the least.  (A chunk is only there to be faster.)
            cudaGetLastError();
            slcs_config least{};
            least.algo = SLCS_ALGO_WAVEFRONT;
            least.use_graph = cfg ? cfg->use_graph : 0;
            least.wait_ms = cfg ? cfg->wait_ms : 0;
            return plan_create_impl(plan_out, pairs, npairs, &least, chunk);
        }
        return cuda_fail(e, "batch plan upload");
    }
    *plan_out = P;
    return SLCS_OK;
}

slcs_status slcs_pair_plan_info_sms(int32_t m, int32_t n, const slcs_config *cfg, int32_t sms, slcs_pair_info *info)
{
    if (!info) return fail(SLCS_ERR_INVALID, "null info");
    if (m < 0 || n < 0 || sms < 1) return fail(SLCS_ERR_INVALID, "m and n must be >= 0 and sms >= 1");
    *info = slcs_pair_info{};
    if (m == 0 || n == 0) return SLCS_OK;
    PairPlan pp;
    const slcs_status s = plan_pair(m, n, cfg, sms, &pp);
    if (s != SLCS_OK) return s;
    const slcs_config &c = pp.c;
    info->algo = c.algo;
    info->tile_m = c.tile_m;
    info->warps = c.warps;
    info->strips = c.strips;
    info->bands = c.bands;
    info->braid_cutoff = c.algo == SLCS_ALGO_STRIPS ? c.braid_cutoff : 0;
    const int64_t stripes = stripes_of(m, c.tile_m);
    info->stripes = int32_t(stripes * (c.algo == SLCS_ALGO_STRIPS ? c.strips : 1));
    // Columns per step as the launch picks them for a b aligned to 8 bytes:
    // the longest chain is the tallest band's, the narrowest tile the
    // narrowest strip.
    int64_t chain = stripes, width = n;
    if (c.algo == SLCS_ALGO_STRIPS) {
        chain = 0;
        for (int32_t h : band_heights(m, c.bands, c.tile_m)) chain = std::max<int64_t>(chain, stripes_of(h, c.tile_m));
        width = INT64_MAX;
        for (int32_t w : strip_widths(n, c.strips)) width = std::min<int64_t>(width, w);
    }
    info->cols_per_step = pick_tw(c.tile_m, chain, width, nullptr);
    if (pp.relay.relay.tm > 0) {
        info->relay_tile_m = pp.relay.relay.tm;
        info->relay_cols = pp.relay.relay.tw;
        info->relay_warps = pp.relay.relay.warps;
        info->relay_strips = pp.relay.strips;
        info->relay_bands = pp.relay.bands;
    }
    return SLCS_OK;
}

slcs_status slcs_pair_plan_info(int32_t m, int32_t n, const slcs_config *cfg, slcs_pair_info *info)
{
    if (!info) return fail(SLCS_ERR_INVALID, "null info");
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if (m == 0 || n == 0) {
        *info = slcs_pair_info{};
        return SLCS_OK;
    }
    return slcs_pair_plan_info_sms(m, n, cfg, sm_count(), info);
}

slcs_status slcs_batch_plan_info(const slcs_batch_plan *P, slcs_plan_info *info)
{
    if (!P || !info) return fail(SLCS_ERR_INVALID, "null plan or info");
    std::memset(info, 0, sizeof(*info));
    info->stream_tile_m = P->stm;
    info->seg = P->stm > 0 ? P->seg : 0;
    info->stream_classes = P->nclass + (P->npacked > 0 ? 1 : 0);
    info->tile_n = P->stm > 0 ? P->tns : 4;
    info->grid = P->grid;
    info->wavefront_tile_m = P->tm;
    info->warps = P->warps;
    info->stream_pairs = P->nstream;
    info->wavefront_tasks = P->ntasks;
    info->packed_pairs = P->npacked;
    info->relay_groups = P->nrelay;
    info->relay_all = P->relay_all;
    info->relay_duos = P->nduos;
    return SLCS_OK;
}

int32_t slcs_batch_plan_launches(const slcs_batch_plan *P)
{
    if (!P) return 0;
    const bool rest = !P->relay_all && (P->stm > 0 ? P->nstream > 0 : P->ntasks > 0);
    const int32_t stream = P->stm > 0 ? (P->nwarps > 0 ? 1 : 0) + (P->nstaged > 0 ? 3 : 0) + (P->nlists > 0 ? 1 : 0) : 1;
    return (rest ? stream : 0) + (P->nrelay > 0 ? 1 : 0) +
           int32_t(P->empty_pairs.size());
}

slcs_status slcs_batch_plan_run(slcs_batch_plan *P, const uint8_t *a, const uint8_t *b, int32_t *out, void *stream)
{
    if (!P) return fail(SLCS_ERR_INVALID, "plan is null");
    if (P->npairs > 0 && (!out || (P->ntasks > 0 && (!a || !b))))
        return fail(SLCS_ERR_INVALID, "null blob or output pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!P->use_graph) return P->enqueue(a, b, out, nullptr, st);
    if (!P->gexec || P->g_a != a || P->g_b != b || P->g_out != out) {
        if (P->gexec) {
            cudaGraphExecDestroy(P->gexec);
            P->gexec = nullptr;
        }
        if (!P->cap_stream) SLCS_CUDA(cudaStreamCreateWithFlags(&P->cap_stream, cudaStreamNonBlocking));
        SLCS_CUDA(cudaStreamBeginCapture(P->cap_stream, cudaStreamCaptureModeThreadLocal));
        slcs_status s = P->enqueue(a, b, out, nullptr, P->cap_stream);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(P->cap_stream, &g);
        if (s != SLCS_OK) {
            if (g) cudaGraphDestroy(g);
            return s;
        }
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
        e = cudaGraphInstantiate(&P->gexec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
        P->g_a = a;
        P->g_b = b;
        P->g_out = out;
    }
    SLCS_CUDA(cudaGraphLaunch(P->gexec, st));
    return SLCS_OK;
}

slcs_status slcs_batch_plan_run_host(slcs_batch_plan *P, const uint8_t *a, int64_t a_len, const uint8_t *b,
                                     int64_t b_len, int32_t *out, int64_t out_len, void *stream)
{
    if (!P) return fail(SLCS_ERR_INVALID, "plan is null");
    if (a_len < P->need_a || b_len < P->need_b || out_len < P->need_out)
        return fail(SLCS_ERR_RANGE, "a host buffer is shorter than the plan's descriptors reach");
    if ((P->need_a && !a) || (P->need_b && !b) || (P->need_out && !out))
        return fail(SLCS_ERR_INVALID, "null host buffer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t ab = align_up(size_t(P->need_a) + 16, 256), bb = align_up(size_t(P->need_b) + 16, 256);
    const size_t need = ab + bb + sizeof(int32_t) * size_t(P->need_out) + 16;
    if (need > P->h_stage_bytes) {
        SLCS_CUDA(cudaStreamSynchronize(st));
        cudaFree(P->h_stage);
        P->h_stage = nullptr;
        P->h_stage_bytes = 0;
        SLCS_CUDA(cudaMalloc(reinterpret_cast<void **>(&P->h_stage), need));
        P->h_stage_bytes = need;
    }
    uint8_t *da = reinterpret_cast<uint8_t *>(P->h_stage);
    uint8_t *db = reinterpret_cast<uint8_t *>(P->h_stage + ab);
    int32_t *dout = reinterpret_cast<int32_t *>(P->h_stage + ab + bb);
    if (!P->chunks.empty()) {
        // Each chunk on its own stream: copy its ranges in, comb, copy its
        // strands out.  With pinned host buffers the copy engines move one
        // chunk while another combs.
        SLCS_CUDA(cudaEventRecord(P->chunk_start, st));
        for (auto &k : P->chunks) {
            SLCS_CUDA(cudaStreamWaitEvent(k.stream, P->chunk_start, 0));
            if (k.a_hi > k.a_lo)
                SLCS_CUDA(cudaMemcpyAsync(da + k.a_lo, a + k.a_lo, size_t(k.a_hi - k.a_lo), cudaMemcpyHostToDevice,
                                          k.stream));
            if (k.b_hi > k.b_lo)
                SLCS_CUDA(cudaMemcpyAsync(db + k.b_lo, b + k.b_lo, size_t(k.b_hi - k.b_lo), cudaMemcpyHostToDevice,
                                          k.stream));
            slcs_status s = slcs_batch_plan_run(k.plan, da, db, dout, k.stream);
            if (s != SLCS_OK) return s;
            if (k.o_hi > k.o_lo)
                SLCS_CUDA(cudaMemcpyAsync(out + k.o_lo, dout + k.o_lo, sizeof(int32_t) * size_t(k.o_hi - k.o_lo),
                                          cudaMemcpyDeviceToHost, k.stream));
            SLCS_CUDA(cudaEventRecord(k.done, k.stream));
            SLCS_CUDA(cudaStreamWaitEvent(st, k.done, 0));
        }
        SLCS_CUDA(cudaStreamSynchronize(st));
        return slcs_device_status(P->device, 1);
    }
    if (P->need_a) SLCS_CUDA(cudaMemcpyAsync(da, a, size_t(P->need_a), cudaMemcpyHostToDevice, st));
    if (P->need_b) SLCS_CUDA(cudaMemcpyAsync(db, b, size_t(P->need_b), cudaMemcpyHostToDevice, st));
    slcs_status s = slcs_batch_plan_run(P, da, db, dout, stream);
    if (s != SLCS_OK) return s;
    if (P->need_out)
        SLCS_CUDA(cudaMemcpyAsync(out, dout, sizeof(int32_t) * size_t(P->need_out), cudaMemcpyDeviceToHost, st));
    SLCS_CUDA(cudaStreamSynchronize(st));
    return slcs_device_status(P->device, 1);
}

// The strands of [lo, hi) narrowed to int16 (every id of the plan is below 2^15).
__global__ void narrow16_kernel(const int32_t *__restrict__ in, int16_t *__restrict__ out, int64_t lo, int64_t hi)
{
    for (int64_t i = lo + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < hi; i += int64_t(gridDim.x) * blockDim.x)
        out[i] = int16_t(in[i]);
}

static slcs_status narrow16(const int32_t *in, int16_t *out, int64_t lo, int64_t hi, cudaStream_t st)
{
    if (hi <= lo) return SLCS_OK;
    const int blocks = int(std::min<int64_t>((hi - lo + 255) / 256, int64_t(sm_count()) * 8));
    narrow16_kernel<<<blocks, 256, 0, st>>>(in, out, lo, hi);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

// The same for the strands of the listed pairs, one block each.
__global__ void narrow16_pairs_kernel(const PairDev *pairs, const int32_t *list, const int32_t *__restrict__ in,
                                      int16_t *__restrict__ out)
{
    const PairDev P = pairs[list[blockIdx.x]];
    for (int32_t i = threadIdx.x; i < P.m + P.n; i += blockDim.x) out[P.out_off + i] = int16_t(in[P.out_off + i]);
}

// A run of the plan whose strands end up as int16 in out16 (entries lo to hi):
// the couples write them so, the other pairs' are narrowed from out.
static slcs_status run16(slcs_batch_plan *P, const uint8_t *a, const uint8_t *b, int32_t *out, int16_t *out16,
                         int64_t lo, int64_t hi, cudaStream_t st)
{
    if (P->ncouples == 0) {
        const slcs_status s = slcs_batch_plan_run(P, a, b, out, st);
        return s == SLCS_OK ? narrow16(out, out16, lo, hi, st) : s;
    }
    const slcs_status s = P->enqueue(a, b, out, out16, st);
    if (s != SLCS_OK || P->nothers == 0) return s;
    narrow16_pairs_kernel<<<P->nothers, 256, 0, st>>>(P->d_pairs, P->d_others, out, out16);
    SLCS_CUDA(cudaGetLastError());
    return SLCS_OK;
}

slcs_status slcs_batch_plan_run_host16(slcs_batch_plan *P, const uint8_t *a, int64_t a_len, const uint8_t *b,
                                       int64_t b_len, int16_t *out, int64_t out_len, void *stream)
{
    if (!P) return fail(SLCS_ERR_INVALID, "plan is null");
    if (P->max_ids > 32767) return fail(SLCS_ERR_RANGE, "a pair of the plan has m + n > 32767: ids need int32");
    if (a_len < P->need_a || b_len < P->need_b || out_len < P->need_out)
        return fail(SLCS_ERR_RANGE, "a host buffer is shorter than the plan's descriptors reach");
    if ((P->need_a && !a) || (P->need_b && !b) || (P->need_out && !out))
        return fail(SLCS_ERR_INVALID, "null host buffer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t ab = align_up(size_t(P->need_a) + 16, 256), bb = align_up(size_t(P->need_b) + 16, 256);
    const size_t need = ab + bb + sizeof(int32_t) * size_t(P->need_out) + 16;
    if (need > P->h_stage_bytes || size_t(P->need_out) > P->out16_elems) {
        SLCS_CUDA(cudaStreamSynchronize(st));
        if (need > P->h_stage_bytes) {
            cudaFree(P->h_stage);
            P->h_stage = nullptr;
            P->h_stage_bytes = 0;
            SLCS_CUDA(cudaMalloc(reinterpret_cast<void **>(&P->h_stage), need));
            P->h_stage_bytes = need;
        }
        if (size_t(P->need_out) > P->out16_elems) {
            cudaFree(P->d_out16);
            P->d_out16 = nullptr;
            P->out16_elems = 0;
            SLCS_CUDA(cudaMalloc(reinterpret_cast<void **>(&P->d_out16), sizeof(int16_t) * size_t(P->need_out) + 16));
            P->out16_elems = size_t(P->need_out);
        }
    }
    uint8_t *da = reinterpret_cast<uint8_t *>(P->h_stage);
    uint8_t *db = reinterpret_cast<uint8_t *>(P->h_stage + ab);
    int32_t *dout = reinterpret_cast<int32_t *>(P->h_stage + ab + bb);
    int16_t *d16 = P->d_out16;
    if (!P->chunks.empty()) {
        // As slcs_batch_plan_run_host, chunk by chunk on their own streams,
        // with half the bytes to copy back.
        SLCS_CUDA(cudaEventRecord(P->chunk_start, st));
        for (auto &k : P->chunks) {
            SLCS_CUDA(cudaStreamWaitEvent(k.stream, P->chunk_start, 0));
            if (k.a_hi > k.a_lo)
                SLCS_CUDA(cudaMemcpyAsync(da + k.a_lo, a + k.a_lo, size_t(k.a_hi - k.a_lo), cudaMemcpyHostToDevice,
                                          k.stream));
            if (k.b_hi > k.b_lo)
                SLCS_CUDA(cudaMemcpyAsync(db + k.b_lo, b + k.b_lo, size_t(k.b_hi - k.b_lo), cudaMemcpyHostToDevice,
                                          k.stream));
            const slcs_status s = run16(k.plan, da, db, dout, d16, k.o_lo, k.o_hi, k.stream);
            if (s != SLCS_OK) return s;
            if (k.o_hi > k.o_lo)
                SLCS_CUDA(cudaMemcpyAsync(out + k.o_lo, d16 + k.o_lo, sizeof(int16_t) * size_t(k.o_hi - k.o_lo),
                                          cudaMemcpyDeviceToHost, k.stream));
            SLCS_CUDA(cudaEventRecord(k.done, k.stream));
            SLCS_CUDA(cudaStreamWaitEvent(st, k.done, 0));
        }
        SLCS_CUDA(cudaStreamSynchronize(st));
        return slcs_device_status(P->device, 1);
    }
    if (P->need_a) SLCS_CUDA(cudaMemcpyAsync(da, a, size_t(P->need_a), cudaMemcpyHostToDevice, st));
    if (P->need_b) SLCS_CUDA(cudaMemcpyAsync(db, b, size_t(P->need_b), cudaMemcpyHostToDevice, st));
    const slcs_status s = run16(P, da, db, dout, d16, 0, P->need_out, st);
    if (s != SLCS_OK) return s;
    if (P->need_out)
        SLCS_CUDA(cudaMemcpyAsync(out, d16, sizeof(int16_t) * size_t(P->need_out), cudaMemcpyDeviceToHost, st));
    SLCS_CUDA(cudaStreamSynchronize(st));
    return slcs_device_status(P->device, 1);
}

slcs_status slcs_batch_plan_destroy(slcs_batch_plan *P)
{
    if (!P) return SLCS_OK;
    cudaFree(P->d_out16);
    for (auto &k : P->chunks) {
        slcs_batch_plan_destroy(k.plan);
        if (k.stream) cudaStreamDestroy(k.stream);
        if (k.done) cudaEventDestroy(k.done);
    }
    if (P->chunk_start) cudaEventDestroy(P->chunk_start);
    if (P->gexec) cudaGraphExecDestroy(P->gexec);
    if (P->cap_stream) cudaStreamDestroy(P->cap_stream);
    if (P->side) cudaStreamDestroy(P->side);
    if (P->fork) cudaEventDestroy(P->fork);
    if (P->join) cudaEventDestroy(P->join);
    if (P->d_block) {
        int cur = 0;
        cudaGetDevice(&cur);
        if (cur != P->device) cudaSetDevice(P->device);
        cudaDeviceSynchronize(); // as cudaFree waits: the plan may still be running
        if (P->pooled) {
            cudaFreeAsync(P->d_block, nullptr);
            cudaStreamSynchronize(nullptr); // gives back what is past PLAN_POOL_KEPT
        } else {
            cudaFree(P->d_block);
        }
        if (cur != P->device) cudaSetDevice(cur);
    }
    cudaFree(P->h_stage);
    delete P;
    return SLCS_OK;
}

slcs_status slcs_comb_batch(const slcs_pair_desc *pairs, int32_t npairs, const uint8_t *a_blob,
                            const uint8_t *b_blob, int32_t *out, const slcs_config *cfg, void *stream)
{
    slcs_batch_plan *P = nullptr;
    slcs_config c{};
    if (cfg) c = *cfg;
    c.use_graph = 0;
    slcs_status s = slcs_batch_plan_create(&P, pairs, npairs, &c);
    if (s != SLCS_OK) return s;
    s = slcs_batch_plan_run(P, a_blob, b_blob, out, stream);
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    slcs_batch_plan_destroy(P);
    if (s != SLCS_OK) return s;
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
    return SLCS_OK;
}

slcs_status slcs_comb_batch_host(const slcs_pair_desc *pairs, int32_t npairs, const uint8_t *a_blob, int64_t a_len,
                                 const uint8_t *b_blob, int64_t b_len, int32_t *out, int64_t out_len,
                                 const slcs_config *cfg)
{
    slcs_status s = check_pairs(pairs, npairs);
    if (s != SLCS_OK) return s;
    for (int32_t p = 0; p < npairs; ++p) {
        const slcs_pair_desc &d = pairs[p];
        if (d.a_offset + d.m > a_len || d.b_offset + d.n > b_len || d.out_offset + d.m + d.n > out_len)
            return fail(SLCS_ERR_RANGE, "pair " + std::to_string(p) + " reaches past its blob");
    }
    slcs_batch_plan *P = nullptr;
    s = slcs_batch_plan_create(&P, pairs, npairs, cfg);
    if (s != SLCS_OK) return s;
    cudaStream_t st = nullptr;
    char *buf = nullptr;
    const size_t ab = align_up(size_t(a_len) + 16, 256), bb = align_up(size_t(b_len) + 16, 256);
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMallocAsync(reinterpret_cast<void **>(&buf), ab + bb + sizeof(int32_t) * size_t(out_len), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(buf, a_blob, size_t(a_len), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(buf + ab, b_blob, size_t(b_len), cudaMemcpyHostToDevice, st);
    int32_t *dout = reinterpret_cast<int32_t *>(buf + ab + bb);
    if (e == cudaSuccess) {
        s = slcs_batch_plan_run(P, reinterpret_cast<uint8_t *>(buf), reinterpret_cast<uint8_t *>(buf + ab), dout, st);
        if (s == SLCS_OK)
            e = cudaMemcpyAsync(out, dout, sizeof(int32_t) * size_t(out_len), cudaMemcpyDeviceToHost, st);
    }
    if (buf) cudaFreeAsync(buf, st);
    cudaError_t e2 = st ? cudaStreamSynchronize(st) : cudaSuccess;
    if (st) cudaStreamDestroy(st);
    slcs_batch_plan_destroy(P);
    if (s != SLCS_OK) return s;
    if (e != cudaSuccess) return cuda_fail(e, "batch host copies");
    if (e2 != cudaSuccess) return cuda_fail(e2, "cudaStreamSynchronize");
    int dev = 0;
    cudaGetDevice(&dev);
    return slcs_device_status(dev, 1);
}

slcs_status slcs_strands_to_permutation(const int32_t *h, int32_t m, const int32_t *v, int32_t n,
                                        int32_t *row_to_col, int32_t *col_to_row, void *stream)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if ((m > 0 && !h) || (n > 0 && !v)) return fail(SLCS_ERR_INVALID, "null strands");
    return launch_strands_to_perm(h, m, v, n, row_to_col, col_to_row, static_cast<cudaStream_t>(stream));
}

slcs_status slcs_substring_llcs(const int32_t *v_strands, int32_t m, int32_t n, const int32_t *begin,
                                const int32_t *end, int32_t nq, int32_t *llcs_out, void *stream)
{
    if (m < 0 || n < 0 || nq < 0) return fail(SLCS_ERR_INVALID, "m, n and nq must be >= 0");
    if (int64_t(m) + n > INT32_MAX) return fail(SLCS_ERR_RANGE, "m+n exceeds int32 strand ids");
    if (nq > 0 && (!begin || !end || !llcs_out || (n > 0 && !v_strands)))
        return fail(SLCS_ERR_INVALID, "null strands or query arrays");
    return launch_substring_llcs(v_strands, m, n, begin, end, nq, llcs_out, static_cast<cudaStream_t>(stream));
}

slcs_status slcs_permutation_to_strands(const int32_t *row_to_col, int32_t m, int32_t n, int32_t *h, int32_t *v,
                                        void *stream)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if (int64_t(m) + n > INT32_MAX) return fail(SLCS_ERR_RANGE, "m+n exceeds int32 strand ids");
    if ((m + n > 0 && !row_to_col) || (m > 0 && !h) || (n > 0 && !v))
        return fail(SLCS_ERR_INVALID, "null permutation or strands");
    return perm_to_strands(row_to_col, m, n, h, v, static_cast<cudaStream_t>(stream));
}

slcs_status slcs_strands_hash(const int32_t *h, int32_t m, const int32_t *v, int32_t n, int64_t *hash_out,
                              void *stream)
{
    if (m < 0 || n < 0) return fail(SLCS_ERR_INVALID, "m and n must be >= 0");
    if (int64_t(m) + n > INT32_MAX) return fail(SLCS_ERR_RANGE, "m+n exceeds int32 strand ids");
    if ((m > 0 && !h) || (n > 0 && !v) || !hash_out) return fail(SLCS_ERR_INVALID, "null strands or output");
    return launch_strands_hash(h, m, v, n, hash_out, static_cast<cudaStream_t>(stream));
}

slcs_status slcs_batch_plan_hash(const slcs_batch_plan *P, const int32_t *strands, int64_t *hashes_out,
                                 void *stream)
{
    if (!P) return fail(SLCS_ERR_INVALID, "plan is null");
    if (P->npairs > 0 && (!strands || !hashes_out)) return fail(SLCS_ERR_INVALID, "null strands or output");
    return launch_batch_hash(P->d_pairs, P->npairs, strands, hashes_out, static_cast<cudaStream_t>(stream));
}

// Restates PermutationMatrix::hash (src/permutation_matrix.hpp:192-203): the
// reference multiplies in signed 64-bit and its build wraps on overflow, so
// the wrap is reproduced in unsigned arithmetic; % truncates toward zero.
int64_t slcs_permutation_hash(const int32_t *col_to_row, int32_t size)
{
    const int64_t R = 4294967279LL, M = 4294967291LL;
    int64_t r = 0;
    for (int32_t i = 0; i < size; ++i) {
        const uint64_t t = uint64_t(R) * uint64_t(r) + uint64_t(int64_t(col_to_row[i]));
        r = int64_t(t) % M;
    }
    return r;
}

slcs_status slcs_braid_multiply(const int32_t *p_r2c, int32_t p_size, const int32_t *q_r2c, int32_t q_size,
                                int32_t k, int32_t row_glue, int32_t *out_r2c, const slcs_config *cfg, void *stream)
{
    if (p_size < 0 || q_size < 0 || k < 0 || k > p_size || k > q_size)
        return fail(SLCS_ERR_INVALID, "need 0 <= k <= min(p_size, q_size)");
    if ((p_size && !p_r2c) || (q_size && !q_r2c) || (p_size + q_size - k > 0 && !out_r2c))
        return fail(SLCS_ERR_INVALID, "null permutation pointer");
    if (p_size + q_size == 0) return SLCS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int cutoff = (cfg && cfg->braid_cutoff > 0) ? cfg->braid_cutoff : 0;
    (void)sm_count(); // per-device set-up (memory pool) before the first allocation
    size_t bytes = 0;
    braid_workspace_bytes(p_size, q_size, k, cutoff, &bytes);
    void *ws = nullptr;
    SLCS_CUDA(cudaMallocAsync(&ws, bytes, st));
    const BraidJob job{p_r2c, p_size, q_r2c, q_size, out_r2c};
    slcs_status s = launch_braids(&job, 1, k, row_glue != 0, cutoff, ws, bytes, st);
    SLCS_CUDA(cudaFreeAsync(ws, st));
    return s;
}

} // extern "C"
