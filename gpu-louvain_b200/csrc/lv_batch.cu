// lv_batch.cu -- many independent graphs, each run by one CTA or one
// thread-block cluster from start to finish (lv_batch_create / lv_batch_run).
//
// Every graph of a batch goes through the level loop of gpulouvain.cu:30-37
// with the rule of lv_run: sweeps of the seven degree-bucket sub-rounds
// (modularity_optimisation.cu:284-363) with exact gains, the sweep loop's stop
// rule, exact aggregation (community_aggregation.cu:248-347) and the final
// modularity.  A graph's partition, modularity, level and sweep counts are
// therefore what lv_create + lv_run (and the CPU oracle) give for that graph
// alone.
//
// Execution.  One CTA, or a thread-block cluster of up to 16 for a large
// graph, runs one graph from start to finish; graphs start in decreasing
// entry count.  A graph's state lives in slices of batch-wide arrays at the
// graph's own vertex and entry offsets, and the steps of the level loop are
// separated by CTA or cluster barriers instead of kernel launches and host
// round trips.  Vertex ids stay global at every level: the
// level-L vertices of a graph whose first vertex is v0 are v0 .. v0 + V_L - 1.
//
// Tables.  A vertex of degree <= DW (or a merged row of at most DW entries)
// is handled by a lane group or a warp with a table in shared memory; a longer
// row by a warp while it shows few communities, else (as larger merged rows) by
// the whole CTA, with the CTA's shared table when 2 * min(degree, V)
// slots fit, else with the graph's own global table of 2^ceil(log2(2 V0))
// slots.  Every table is empty between uses.
//
// Coherence.  Rows of aggregated levels, the fixed-point weights and the
// community state are written inside the launch, so they are read with
// ordinary (coherent) loads.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

// one kernel holds the whole level loop: near-tie comparisons stay out of line
#define LV_EXACT_CALL 1
#include "../../include/louvain_b200.h"
#include "lv_internal.h"

namespace lv {
namespace {

// 512 threads and 2 CTAs per SM (64 registers).  Smaller CTAs were measured
// for small graphs (8 CTAs of 128 threads per SM): 2048 planted graphs of 100
// to 1500 vertices took 7.7 ms against 5.8 ms, since eight graphs at different
// points of the level loop do not share the instruction cache.
constexpr int BT = 512;             // threads per CTA
constexpr int BW = BT / 32;         // warps per CTA
constexpr int WTAB = 256;           // slots of one warp's table
constexpr int DW = WTAB / 2;        // degree / merged-row bound served by a warp table
constexpr int CTAB = BW * WTAB;     // slots of the CTA table (the warp tables together)
constexpr int WIDE_CLAIMS = 160;    // distinct communities a warp accepts in a longer row
// Graphs with fewer entries evaluate every vertex: their few sweeps skip less
// than the limits cost to keep (ms with / without skipping: 8192 planted graphs
// of 60 to 160 vertices 12.0 / 11.4, 592 R-MAT-8 graphs 2.48 / 2.36, 592 planted
// graphs of 200 vertices 1.36 / 1.35, of 400 (about 5400 entries) 1.57 / 1.63).
constexpr int64_t SKIP_MIN_ENTRIES = 4608;
constexpr int FEW_WIDE = 2;         // longer rows per CTA that are not tried by a warp first
// Work split of a launch (plan_launch): a team's CTA takes TEAM_PART of the
// entries that one resident CTA would have if the batch were spread evenly
// over the GPU, BATCH_MIN_PART at least.  256 planted graphs of 100 to 50,000
// vertices took 27.0 / 25.9 / 24.8 / 25.4 / 34.3 ms with 0.3 / 0.5 / 0.7 / 1 /
// 2 (152 ms with one CTA per graph, the largest graph's time), 2048 of 100 to
// 1500 vertices 7.1 / 6.0 / 5.8 / 5.8 / 5.8 ms.  296 graphs of 300 vertices
// (3600 entries) took 1.78 ms split in two and 0.93 whole.  A lone graph of
// lv_run is split down to TEAM_MIN_PART entries per CTA.
constexpr double TEAM_PART = 0.7, BATCH_MIN_PART = 4096.0, TEAM_MIN_PART = 2048.0;
// Teams of many graphs of about one size do not all fit on the GPU and run in
// waves, which costs more than they save when the parts are small.  So the
// parts grow until the CTAs of the graphs that are not small (more than half
// the even share) fit, up to this many entries.  148 / 200 / 296 planted graphs
// of 2000 vertices took 2.79 / 3.24 / 3.30 ms without this, 1.69 / 2.21 / 2.42
// with it (1.87 / 2.21 / 2.43 with one CTA each), of 10,000 vertices 10.6 / 12.3 /
// 15.1 ms both ways (11.4 / 13.7 / 14.7); 128 of 1000 to 20,000 vertices 7.7 and
// 8.0 ms, 8.5 with a limit of 65,536.
constexpr double TEAM_FIT_PART = 49152.0;
// Iteration caps that keep a launch bounded; a graph that reaches one stops
// with LV_ERR_DEVICE (the rule itself has no cap: with min_gain <= 0 a sweep
// loop that keeps moving at zero gain would not end).
constexpr int SWEEP_CAP = 4096;
constexpr int LEVEL_CAP = 256;

// CTAs of the largest team (a thread-block cluster) that one graph runs on.
constexpr int TEAM_MAX = 16;

// Exchange area of a team in global memory (zero before the first launch,
// counters returned to zero after each use).
struct TeamScratch {
    u64 red[2][TEAM_MAX][6];   // per-CTA parts of a team reduction, double-buffered
    u64 drift;                 // drift of the level so far (GState::drift_of)
    int32_t cnt[16], cur[16];  // bucket sizes and cursors
    int32_t nbig;
};

struct BatchParams {
    // the caller's block-diagonal CSR (read-only during the launch); w is null
    // when the start rows carry fixed-point sums (s_w64, job only)
    const int32_t *rowptr, *rowend;
    const int32_t *col;
    const float *w;
    const u64 *s_w64;
    TeamResult *job;           // set: one graph of V, E (checked by the caller), results here
    int32_t job_V;
    int64_t job_E;
    double job_scale;
    int job_narrow;
    int32_t sweep_cap, level_cap;
    const int32_t *gptr;       // [G + 1] first vertex of each graph
    const int32_t *order;      // [G] graphs by decreasing entry count
    const int64_t *tbl_off;    // [G + 1] first slot of each graph's global table
    int32_t lo;                // the launch's first graph in order
    int32_t max_sweeps;
    double min_gain;
    // per vertex (V entries; mstart / roff: V + G, the slice of graph g starts at v0 + g)
    int32_t *comm, *newc, *size, *blist, *newid, *members, *o2c, *mstart, *roff;
    int32_t *rs[2], *re[2];    // aggregated levels: row v = [rs[v], re[v])
    u64 *k, *S;
    u64 *lim;                  // a vertex keeps its community while the level's drift is below lim
    // per entry (E entries): aggregated rows, ping-pong
    int32_t *colb[2];
    u64 *wb[2];
    int32_t *tkeys;            // global tables (-1 / 0 between uses)
    u64 *tvals;
    TeamScratch *scratch;      // one per graph that runs on a team, in order
    // results
    int32_t *out_comm;         // [V] community of each vertex, numbered within its graph
    double *q;
    int32_t *nc, *status, *levels;
    int64_t *sweeps, *edge_sweeps, *vertex_sweeps, *moves;
    u64 *t_start, *t_end;      // %globaltimer (ns) around each graph
};

// A graph's current level and totals (the same in every thread of the team).
struct GState {
    int32_t g, v0, V0, V;
    int64_t e0;     // first entry of the graph in the caller's CSR
    int64_t E;      // entries of the current level
    int64_t tbl;    // first slot of the graph's global table
    u64 T;
    double scale;
    int cur;        // -1: level 0 (the caller's CSR), else the buffer of the level's rows
    int dsh;        // drift is counted in units of 2^dsh
    float dunit;    // 2^-dsh
    bool narrow;    // level-0 weights fit 32 bits
    bool sym;       // every entry has its mirror entry (same weight)
    bool skip;      // vertices may be skipped: sym, and the graph is not too small
    // what one move of a vertex of weight k adds to the drift: an upper bound of 2 k
    __device__ __forceinline__ u64 drift_of(u64 k) const { return ((2 * k) >> dsh) + 1; }
};

struct Acc {
    int64_t sweeps, edge_sweeps, vertex_sweeps, moves;
    double q;
};

// A level's rows: [rs[v], re[v]) in col and in w32 (level 0, when its
// fixed-point weights fit 32 bits) or w64.  Level 0 reads the fixed-point
// weights that level_setup wrote, so that one code path serves every level
// (the kernel's code has to fit the instruction cache) and no sweep converts
// floats.
struct Rows {
    const int32_t *rs;
    const int32_t *re;
    const int32_t *col;
    const uint32_t *w32;
    const u64 *w64;
    __device__ __forceinline__ int32_t r0(int32_t v) const { return rs[v]; }
    __device__ __forceinline__ int32_t r1(int32_t v) const { return re[v]; }
    __device__ __forceinline__ int32_t c(int64_t e) const { return col[e]; }
    __device__ __forceinline__ u64 x(int64_t e) const { return w32 ? (u64)w32[e] : w64[e]; }
};

// Update-order bucket of a degree (modularity_optimisation.cuh:7-8).
__device__ __forceinline__ int bucket_of(int32_t d) {
    if (d <= 0) return -1;
    if (d <= 4) return 0;
    if (d <= 8) return 1;
    if (d <= 16) return 2;
    if (d <= 32) return 3;
    if (d <= 84) return 4;
    if (d <= 319) return 5;
    return 6;
}

__device__ __forceinline__ u64 globaltimer() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ int table_lg(int32_t bound) {
    const int lg = ceil_log2_i(2 * (int64_t)bound);
    return lg < 1 ? 1 : lg;
}

// ---- reductions and scan (every thread gets the result) ----
struct Totals5 {
    u64 a, b;      // wrapping sums
    u128 s2;       // exact sum
    u64 err;       // OR
};

// ---- which vertices need a decision ----
// A vertex v that was evaluated and stayed, with slack = T e_own - max(0, max_C
// G(C)) >= 0, stays as long as no neighbour changes community and Sigma_tot
// moves little: then every e_C is unchanged and G(C) = T e_C + k (S_own - k -
// S_C) grows by at most k times the total change of Sigma_tot, to which a move
// of a vertex of weight k' adds 2 k'.  The level's drift sums an upper bound
// of 2 k' over its moves, and v is skipped while drift < lim[v] =
// drift at evaluation + floor(slack / k) + 1 (in drift units).  A move sets
// lim to 0 (evaluate next time) for the mover and for its neighbours; a vertex
// that was alone in its community when evaluated is never skipped, since the
// singleton guard may have hidden candidates from its slack.  Decisions are
// therefore exactly those of evaluating every vertex; the batch of 256 planted
// graphs of 100 to 50,000 vertices takes 30.7 ms with skipping and 40.9 ms
// without.
__device__ __forceinline__ u64 skip_limit(const MoveCtx &m, const Best &b, u64 drift, float dunit) {
    constexpr u64 FAR = (u64)1 << 62;
    if (m.kv == 0) return FAR;
    // a lower bound of slack / k in drift units: gain_err bounds the estimate
    // gd, and 2^-20 covers the roundings of the remaining operations
    const double g = b.c == m.own ? 0.0 : fmax(0.0, b.gd + gain_err(m, b));
    const double slack = fmax(0.0, m.Td * (double)b.eo * (1.0 - 0x1p-48) - g);
    const float d = __fdividef((float)slack, (float)m.kvd) * dunit * (1.0f - 0x1p-20f);
    return d < 0x1p61f ? drift + (u64)d + 1 : FAR;
}

// calculateModularity (modularity_optimisation.cu:395-401) from exact totals.
__device__ __forceinline__ double modularity_from(const GState &gs, u64 e_own, u128 s2) {
    return q_from_parts_dev(gs.T, e_own, (u64)(s2 >> 64), (u64)s2);
}

// Group tables: the sum of a slot is kept in three 32-bit counters of 22-bit
// pieces, so that an add is two or three shared atomics without a returned
// value or a carry; exact for up to 1024 adds per slot (rows of at most DW
// entries) and weights up to 2^62 (T <= 2^62).
struct PieceSlots {
    int32_t *keys;
    uint32_t *lo, *mid, *hi;
    // adds w to key's sum; the slot when it was newly claimed, else -1
    __device__ __forceinline__ int32_t insert(int lg, int32_t key, u64 w, int *err) const {
        const uint32_t mask = (1u << lg) - 1u;
        uint32_t s = hash_slot(key, lg);
        int32_t claimed = -1;
        for (uint32_t p = 0;; ++p) {
            const int32_t k = ((volatile int32_t *)keys)[s];
            if (k == key) break;
            if (k < 0) {
                const int32_t prev = atomicCAS(keys + s, -1, key);
                if (prev < 0) claimed = (int32_t)s;
                if (prev < 0 || prev == key) break;
            }
            if (p == mask) {
                atomicOr(err, DEVERR_HASH_FULL);
                return -1;
            }
            s = (s + 1u) & mask;
        }
        atomicAdd(lo + s, (uint32_t)w & 0x3FFFFFu);
        const uint32_t b = (uint32_t)(w >> 22) & 0x3FFFFFu, c = (uint32_t)(w >> 44);
        if (b) atomicAdd(mid + s, b);
        if (c) atomicAdd(hi + s, c);
        return claimed;
    }
    // the sum of slot s, which is emptied
    __device__ __forceinline__ u64 take(int s) const {
        const u64 x = (u64)lo[s] + ((u64)mid[s] << 22) + ((u64)hi[s] << 44);
        keys[s] = -1;
        lo[s] = 0;
        mid[s] = 0;
        hi[s] = 0;
        return x;
    }
};
static_assert(DW <= 1024, "pieces of 22 bits in 32-bit counters");

// The level loop of one graph.
struct Loop {
struct BatchSmem {
    u64 vals[CTAB];            // 64-bit sums, or two counters of PieceSlots per slot
    uint32_t hi[CTAB];         // the third counter
    int32_t keys[CTAB];
    u64 red[BW][5];
    u64 tot[5];
    u64 drift;
    double bgd[BW];
    u64 be[BW], bS[BW], beo[BW];
    int32_t bc[BW];
    int32_t scan[BW];
    int32_t bcnt[16], boff[16], bcur[16];   // bucket b: [2b] degree <= DW, [2b + 1] larger
    int32_t err, nbig, cnt;
    uint8_t ord[BW][32];       // a warp's chunk: lanes holding vertices to decide, in order
    uint8_t occ[BW][DW];       // claimed slots of the warp's group tables
    // State that is the same in every thread.  In registers it was spilled in
    // the sub-rounds' loops, and the local memory of 1024 threads pushed the
    // graph's state out of L1 (stack frame 248 -> 120 bytes; 2048 planted graphs
    // of 100 to 1500 vertices 5.52 -> 5.07 ms, 592 of 1600 4.35 -> 4.09, 200 stars of
    // 500 vertices 0.89 -> 0.79).  gs, rows: every thread writes the same values
    // before it reads them; the others are thread 0's.
    GState gs;
    Rows rows;
    Acc acc;
    double q_before;           // modularity before the current sweep
    u64 e_own;                 // sum of e_{i->C(i)}
};

// The CTAs that run one graph together: this CTA alone (nc == 1), or every
// CTA of its cluster.  Steps of the level loop are separated by sync(): the
// cluster barrier orders the team's accesses to the graph's global arrays
// (release on arrival, acquire on the wait).  Every branch around a sync()
// depends only on values that all threads of the team agree on (the graph's
// sizes and reduced totals), so the team's CTAs pass the same barriers.
struct Team {
    int32_t rank, nc;
    int par;                   // which half of scratch->red the next reduction uses
    TeamScratch *scr;
    __device__ __forceinline__ void sync() const {
        if (nc == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::
                             : "memory");
        }
    }
    __device__ __forceinline__ int32_t tid() const { return rank * BT + (int32_t)threadIdx.x; }
    __device__ __forceinline__ int32_t threads() const { return nc * BT; }
    __device__ __forceinline__ int32_t warp() const { return rank * BW + (int32_t)(threadIdx.x >> 5); }
    __device__ __forceinline__ int32_t warps() const { return nc * BW; }
};

// Sums over the CTA (warp 0 combines the warps' parts); contains barriers.
static __device__ __forceinline__ Totals5 block_totals(Totals5 x, BatchSmem &sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    x.a = warp_sum_u64(x.a);
    x.b = warp_sum_u64(x.b);
    x.s2 = warp_sum_u128(x.s2);
    x.err = __reduce_or_sync(FULL, (unsigned)x.err);
    __syncthreads();
    if (lane == 0) {
        sm.red[warp][0] = x.a;
        sm.red[warp][1] = x.b;
        sm.red[warp][2] = (u64)(x.s2 >> 64);
        sm.red[warp][3] = (u64)x.s2;
        sm.red[warp][4] = x.err;
    }
    __syncthreads();
    if (warp == 0) {
        Totals5 y{};
        if (lane < BW) {
            y.a = sm.red[lane][0];
            y.b = sm.red[lane][1];
            y.s2 = ((u128)sm.red[lane][2] << 64) | (u128)sm.red[lane][3];
            y.err = sm.red[lane][4];
        }
        y.a = warp_sum_u64(y.a);
        y.b = warp_sum_u64(y.b);
        y.s2 = warp_sum_u128(y.s2);
        y.err = __reduce_or_sync(FULL, (unsigned)y.err);
        if (lane == 0) {
            sm.tot[0] = y.a;
            sm.tot[1] = y.b;
            sm.tot[2] = (u64)(y.s2 >> 64);
            sm.tot[3] = (u64)y.s2;
            sm.tot[4] = y.err;
        }
    }
    __syncthreads();
    Totals5 t;
    t.a = sm.tot[0];
    t.b = sm.tot[1];
    t.s2 = ((u128)sm.tot[2] << 64) | (u128)sm.tot[3];
    t.err = sm.tot[4];
    return t;
}

// Sums over the team.  Each CTA writes its part to the scratch area and reads
// all parts after the barrier; the next reduction uses the other half, and
// the one after that is separated from this one's reads by a barrier.
static __device__ __forceinline__ Totals5 team_totals(Totals5 x, Team &t, BatchSmem &sm) {
    x = block_totals(x, sm);
    if (t.nc == 1) return x;
    u64(*red)[6] = t.scr->red[t.par];
    t.par ^= 1;
    if (threadIdx.x == 0) {
        red[t.rank][0] = x.a;
        red[t.rank][1] = x.b;
        red[t.rank][2] = (u64)(x.s2 >> 64);
        red[t.rank][3] = (u64)x.s2;
        red[t.rank][4] = x.err;
    }
    t.sync();
    const int lane = threadIdx.x & 31;
    Totals5 y{};
    if (lane < t.nc) {
        y.a = __ldcg(&red[lane][0]);
        y.b = __ldcg(&red[lane][1]);
        y.s2 = ((u128)__ldcg(&red[lane][2]) << 64) | (u128)__ldcg(&red[lane][3]);
        y.err = __ldcg(&red[lane][4]);
    }
    y.a = warp_sum_u64(y.a);
    y.b = warp_sum_u64(y.b);
    y.s2 = warp_sum_u128(y.s2);
    y.err = __reduce_or_sync(FULL, (unsigned)y.err);
    return y;
}

static __device__ __forceinline__ u64 block_sum_u64(u64 x, BatchSmem &sm) {
    Totals5 t{};
    t.a = x;
    return block_totals(t, sm).a;
}

static __device__ __forceinline__ int block_max_i32(int x, BatchSmem &sm) {
    for (int off = 16; off > 0; off >>= 1) x = max(x, __shfl_xor_sync(FULL, x, off));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sm.scan[threadIdx.x >> 5] = x;
    __syncthreads();
    int t = sm.scan[0];
    for (int i = 1; i < BW; ++i) t = max(t, sm.scan[i]);
    return t;
}

// Exclusive scan of get(0 .. n-1); put(i, prefix, value) for each i; returns
// the total.  Each index is read and written by the same thread, and each CTA
// of a team scans its own range after the ranges' totals were exchanged.
template <class Get, class Put>
static __device__ int32_t team_scan(int32_t n, Get get, Put put, Team &t, BatchSmem &sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t lo = 0, hi = n, carry = 0, all = -1;
    if (t.nc > 1) {
        const int32_t part = (n + t.nc - 1) / t.nc;
        lo = min(n, t.rank * part);
        hi = min(n, lo + part);
        u64 s = 0;
        for (int32_t i = lo + threadIdx.x; i < hi; i += BT) s += (u64)get(i);
        s = block_sum_u64(s, sm);
        u64(*red)[6] = t.scr->red[t.par];
        t.par ^= 1;
        if (threadIdx.x == 0) red[t.rank][0] = s;
        t.sync();
        all = 0;
        for (int r = 0; r < t.nc; ++r) {
            const int32_t x = (int32_t)__ldcg(&red[r][0]);
            carry += r < t.rank ? x : 0;
            all += x;
        }
    }
    for (int32_t base = lo; base < hi; base += BT) {
        const int32_t i = base + threadIdx.x;
        const int32_t x = i < hi ? get(i) : 0;
        int32_t inc = x;
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t y = __shfl_up_sync(FULL, inc, off);
            if (lane >= off) inc += y;
        }
        __syncthreads();
        if (lane == 31) sm.scan[warp] = inc;
        __syncthreads();
        int32_t pre = 0, tot = 0;
        for (int j = 0; j < BW; ++j) {
            const int32_t y = sm.scan[j];
            pre += j < warp ? y : 0;
            tot += y;
        }
        if (i < hi) put(i, carry + pre + inc - x, x);
        carry += tot;
    }
    t.sync();
    return t.nc > 1 ? all : carry;
}

// List entries per chunk when nw warps share n of them: at most 32, the same
// number of chunks for every warp, as nearly as multiples of g allow.
static __device__ __forceinline__ int32_t chunk_of(int32_t n, int32_t nw, int32_t g) {
    const int32_t rounds = max(1, (n + nw * 32 - 1) / (nw * 32));
    return min(32, ((n + nw * rounds - 1) / (nw * rounds) + g - 1) / g * g);
}

// ---- move phase ----
// Vertices of one bucket with degree <= 2^(lg-1): a warp takes chunks of the
// list (32 vertices, or fewer when the list is short for the team's warps),
// loads the headers of the vertices that need a decision (one per lane) and
// decides them with W lanes each (32/W at a time) and a table of 2^lg slots
// per group inside the warp's table.  U entries per lane are in flight at a
// time (U column loads, then U community gathers).
template <int W, int U>
static __device__ void decide_groups(const Rows &L, const BatchParams &P, const GState &gs, const Team &t,
                              const int32_t *list, int32_t n, int lg, u64 drift, BatchSmem &sm) {
    constexpr int GPW = 32 / W;
    constexpr int GTAB = WTAB / GPW;   // slots of one group's table, of which 2^lg are used
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane / W, gl = lane % W;
    const unsigned gmask = W == 32 ? FULL : (((1u << (W & 31)) - 1u) << (grp * W));
    PieceSlots tb;
    tb.keys = sm.keys + warp * WTAB + grp * GTAB;
    tb.lo = reinterpret_cast<uint32_t *>(sm.vals + warp * WTAB) + grp * GTAB;
    tb.mid = tb.lo + WTAB;
    tb.hi = sm.hi + warp * WTAB + grp * GTAB;
    uint8_t *occ = sm.occ[warp] + grp * (DW / GPW);
    uint8_t *ord = sm.ord[warp];
    const int32_t nw = t.warps();
    const int32_t cs = chunk_of(n, nw, GPW);
    for (int32_t c0 = t.warp() * cs; c0 < n; c0 += nw * cs) {
        const int32_t idx = c0 + lane;
        int32_t lv = -1, lr0 = 0, lr1 = 0, lown = -1;
        u64 lkv = 0, lsown = 0;
        bool need = false, lsingle = false;
        if (lane < cs && idx < n) {
            lv = list[idx];
            need = !gs.skip || drift >= P.lim[lv];
        }
        const unsigned mask = __ballot_sync(FULL, need);
        if (!mask) continue;
        if (need) {
            lr0 = L.r0(lv);
            lr1 = L.r1(lv);
            lown = P.comm[lv];
            lkv = P.k[lv];
            lsown = P.S[lown];
            lsingle = P.size[lown] == 1;
            ord[__popc(mask & ((1u << lane) - 1u))] = (uint8_t)lane;
        }
        __syncwarp();
        const int cnt = __popc(mask);
        for (int q0 = 0; q0 < cnt; q0 += GPW) {
            const bool have = q0 + grp < cnt;
            const int src = have ? ord[q0 + grp] : 0;
            int32_t v = __shfl_sync(FULL, lv, src), own = __shfl_sync(FULL, lown, src);
            int32_t r0 = __shfl_sync(FULL, lr0, src), r1 = __shfl_sync(FULL, lr1, src);
            const u64 kv = __shfl_sync(FULL, lkv, src), sown = __shfl_sync(FULL, lsown, src);
            const bool single = __shfl_sync(FULL, (int)lsingle, src) != 0;
            if (!have) {
                v = -1;
                own = -1;
                r0 = r1 = 0;
            }
            u64 eo = 0;
            int nocc = 0;
            // every lane of the warp takes the same number of steps
            const int steps = (int)__reduce_max_sync(FULL, (unsigned)((r1 - r0 + U * W - 1) / (U * W)));
            for (int st = 0; st < steps; ++st) {
                const int32_t base = r0 + gl + st * U * W;
                int32_t jj[U];
                u64 xx[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int32_t e = base + u * W;
                    jj[u] = -1;
                    xx[u] = 0;
                    if (e < r1) {
                        jj[u] = L.c(e);
                        xx[u] = L.x(e);
                    }
                }
                int32_t cc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) cc[u] = (jj[u] >= 0 && jj[u] != v) ? P.comm[jj[u]] : -1;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    int32_t claimed = -1;
                    if (cc[u] >= 0) {
                        if (cc[u] == own) eo += xx[u];
                        else claimed = tb.insert(lg, cc[u], xx[u], &sm.err);
                    }
                    // the group's claimed slots are listed, so that only they are evaluated and emptied
                    const unsigned bal = __ballot_sync(FULL, claimed >= 0) & gmask;
                    if (claimed >= 0) occ[nocc + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)claimed;
                    nocc += __popc(bal);
                }
            }
            __syncwarp();
            const MoveCtx m = move_ctx(own, single, gs.T, kv, sown);
            Best b = best_init(own);
            b.eo = eo;
            for (int i = gl; i < nocc; i += W) {
                const int s = occ[i];
                const int32_t c = tb.keys[s];
                const u64 Sc = P.S[c];
                const int32_t szc = guard_needs_size(m, c) ? P.size[c] : 0;
                eval_loaded(c, tb.take(s), Sc, szc, m, b);
            }
            __syncwarp();
            group_reduce_best(m, b, W);
            if (v >= 0 && gl == 0) {
                u64 d;
                const int32_t nc = move_decision(m, b, &d);
                P.newc[v] = nc;
                if (gs.skip) P.lim[v] = (nc == own && !single) ? skip_limit(m, b, drift, gs.dunit) : 0;
            }
        }
        __syncwarp();
    }
}

// One vertex of degree > DW by the whole CTA.
static __device__ void decide_cta(const Rows &L, const BatchParams &P, const GState &gs, int32_t v, u64 drift,
                           BatchSmem &sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t r0 = L.r0(v), r1 = L.r1(v);
    const int32_t own = P.comm[v];
    const u64 kv = P.k[v], sown = P.S[own];
    const bool single = P.size[own] == 1;
    const int lg = table_lg(min(r1 - r0, gs.V));
    int32_t *keys = sm.keys;
    u64 *vals = sm.vals;
    if ((1 << lg) > CTAB) {
        keys = P.tkeys + gs.tbl;
        vals = P.tvals + gs.tbl;
    }
    u64 eo = 0;
    for (int32_t e = r0 + threadIdx.x; e < r1; e += BT) {
        const int32_t j = L.c(e);
        if (j == v) continue;
        const u64 x = L.x(e);
        const int32_t c = P.comm[j];
        if (c == own) eo += x;
        else table_insert<0>(keys, vals, lg, c, x, &sm.err);
    }
    __syncthreads();
    const MoveCtx m = move_ctx(own, single, gs.T, kv, sown);
    Best b = best_init(own);
    b.eo = eo;
    for (int32_t s = threadIdx.x; s < (1 << lg); s += BT) {
        const int32_t c = keys[s];
        if (c < 0) continue;
        const u64 ec = vals[s];
        keys[s] = -1;
        vals[s] = 0;
        eval_loaded(c, ec, P.S[c], guard_needs_size(m, c) ? P.size[c] : 0, m, b);
    }
    group_reduce_best(m, b, 32);
    if (lane == 0) {
        sm.bgd[warp] = b.gd;
        sm.be[warp] = b.e;
        sm.bS[warp] = b.S;
        sm.bc[warp] = b.c;
        sm.beo[warp] = b.eo;
    }
    __syncthreads();
    if (warp == 0) {
        Best x = best_init(own);
        if (lane < BW) {
            x.gd = sm.bgd[lane];
            x.e = sm.be[lane];
            x.S = sm.bS[lane];
            x.c = sm.bc[lane];
            x.eo = sm.beo[lane];
        }
        group_reduce_best(m, x, 32);
        if (lane == 0) {
            u64 d;
            const int32_t nc = move_decision(m, x, &d);
            P.newc[v] = nc;
            if (gs.skip) P.lim[v] = (nc == own && !single) ? skip_limit(m, x, drift, gs.dunit) : 0;
        }
    }
    __syncthreads();
}

// The vertices of degree > DW of a bucket: a warp each, with the warp's table
// while the row shows at most WIDE_CLAIMS distinct communities (most rows of
// an aggregated level after its first sweeps), else a whole CTA afterwards
// (the vertices are listed in members, free during sweeps).  A vertex whose
// table needs the graph's one global table is left to the first CTA.  When a
// CTA has no more than FEW_WIDE of them, they go to whole CTAs at once: a warp
// alone reads a long row slowly and its attempt is often in vain (512 R-MAT-10
// graphs 8.73 ms, with 2 / 4 rows 8.16 / 8.39; 200 stars of 500 vertices 1.00 ->
// 0.94; 2048 planted graphs of 100 to 1500 vertices 5.59 both ways).
static __device__ void decide_wide(const Rows &L, const BatchParams &P, const GState &gs, const Team &t,
                            const int32_t *list, int32_t n, u64 drift, BatchSmem &sm) {
    constexpr int U = 2;
    constexpr int LG = ilog2_c(WTAB);
    static_assert(WIDE_CLAIMS + 32 * U < WTAB, "a step's claims fit the warp's table");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *keys = sm.keys + warp * WTAB;
    u64 *vals = sm.vals + warp * WTAB;
    int32_t *ovf = P.members + gs.v0;
    int32_t *novf = t.nc == 1 ? &sm.nbig : &t.scr->nbig;   // zero here (level_setup, sweep)
    __syncwarp();
    for (int32_t i = t.warp(); i < n; i += t.warps()) {
        const int32_t v = list[i];
        if (gs.skip && drift < P.lim[v]) continue;
        if (n <= FEW_WIDE * t.nc) {
            if (lane == 0) ovf[atomicAdd(novf, 1)] = v;
            continue;
        }
        const int32_t r0 = L.r0(v), r1 = L.r1(v);
        const int32_t own = P.comm[v];
        const u64 kv = P.k[v], sown = P.S[own];
        const bool single = P.size[own] == 1;
        u64 eo = 0;
        int32_t claims = 0;
        bool over = false;
        for (int32_t b0 = r0; b0 < r1 && !over; b0 += 32 * U) {
            int32_t jj[U];
            u64 xx[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int32_t e = b0 + lane + 32 * u;
                jj[u] = -1;
                xx[u] = 0;
                if (e < r1) {
                    jj[u] = L.c(e);
                    xx[u] = L.x(e);
                }
            }
            int32_t cc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) cc[u] = (jj[u] >= 0 && jj[u] != v) ? P.comm[jj[u]] : -1;
            unsigned mine = 0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (cc[u] < 0) continue;
                if (cc[u] == own) eo += xx[u];
                else mine += table_insert_claim<0>(keys, vals, LG, cc[u], xx[u], &sm.err) >= 0 ? 1u : 0u;
            }
            claims += (int32_t)__reduce_add_sync(FULL, mine);
            over = claims > WIDE_CLAIMS;
        }
        __syncwarp();
        if (over) {
            for (int s = lane; s < WTAB; s += 32) {
                keys[s] = -1;
                vals[s] = 0;
            }
            if (lane == 0) ovf[atomicAdd(novf, 1)] = v;
            __syncwarp();
            continue;
        }
        const MoveCtx m = move_ctx(own, single, gs.T, kv, sown);
        Best b = best_init(own);
        b.eo = eo;
        for (int s = lane; s < WTAB; s += 32) {
            const int32_t c = keys[s];
            if (c < 0) continue;
            const u64 ec = vals[s];
            keys[s] = -1;
            vals[s] = 0;
            eval_loaded(c, ec, P.S[c], guard_needs_size(m, c) ? P.size[c] : 0, m, b);
        }
        __syncwarp();
        group_reduce_best(m, b, 32);
        if (lane == 0) {
            u64 d;
            const int32_t nc = move_decision(m, b, &d);
            P.newc[v] = nc;
            if (gs.skip) P.lim[v] = (nc == own && !single) ? skip_limit(m, b, drift, gs.dunit) : 0;
        }
    }
    t.sync();
    const int32_t no = *(volatile int32_t *)novf;
    for (int pass = 0; pass < (t.nc > 1 ? 2 : 1); ++pass) {
        if (pass == 1 && t.rank != 0) break;
        for (int32_t i = pass ? 0 : t.rank; i < no; i += pass ? 1 : t.nc) {
            const int32_t v = ovf[i];
            if (t.nc > 1) {
                const bool global = (1 << table_lg(min(L.r1(v) - L.r0(v), gs.V))) > CTAB;
                if (global != (pass == 1)) continue;
            }
            decide_cta(L, P, gs, v, drift, sm);
        }
    }
}

// Exact change of sum_i e_{i->C(i)} when one sub-round's decisions commit.
// For a mover v (o -> n) and a neighbour x != v the pair's term changes by
// w ([n == C'(x)] - [o == C(x)]): counted twice from v's row when x stays
// (the entry in x's row is not visited), once from each row when x moves
// too.  Between sub-rounds newc == comm, so newc[x] != comm[x] marks a mover
// of this sub-round.  The neighbours need a new evaluation (lim = 0).  A warp
// takes chunks of the list as in decide_groups and spreads the movers of a
// chunk over lane groups of 8; wrapping uint64 sum.
static __device__ __forceinline__ u64 commit_delta(const Rows &L, const BatchParams &P, const GState &gs,
                                            const Team &t, const int32_t *list, int32_t n, BatchSmem &sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane >> 3, gl = lane & 7;
    uint8_t *ord = sm.ord[warp];
    const int32_t nw = t.warps();
    const int32_t cs = chunk_of(n, nw, 4);
    u64 d = 0;
    for (int32_t c0 = t.warp() * cs; c0 < n; c0 += nw * cs) {
        int32_t lv = -1, ln = 0, lo = 0;
        if (lane < cs && c0 + lane < n) {
            lv = list[c0 + lane];
            ln = P.newc[lv];
            lo = P.comm[lv];
        }
        const bool mover = ln != lo;
        const unsigned mask = __ballot_sync(FULL, mover);
        if (!mask) continue;
        int32_t lr0 = 0, lr1 = 0;
        if (mover) {
            lr0 = L.r0(lv);
            lr1 = L.r1(lv);
            ord[__popc(mask & ((1u << lane) - 1u))] = (uint8_t)lane;
        }
        __syncwarp();
        const int cnt = __popc(mask);
        for (int q0 = 0; q0 < cnt; q0 += 4) {
            const int src = q0 + grp < cnt ? ord[q0 + grp] : -1;
            const int at = src < 0 ? 0 : src;
            const int32_t v = __shfl_sync(FULL, lv, at), nv = __shfl_sync(FULL, ln, at), ov = __shfl_sync(FULL, lo, at);
            const int32_t r0 = __shfl_sync(FULL, lr0, at);
            const int32_t r1s = __shfl_sync(FULL, lr1, at), r1 = src < 0 ? 0 : r1s;
            for (int32_t e = r0 + gl; e < r1; e += 8) {
                const int32_t x = L.c(e);
                if (x == v) continue;
                const u64 w = L.x(e);
                const int32_t cx = P.comm[x], nx = P.newc[x];
                if (gs.skip) P.lim[x] = 0;
                if (nx != cx) {
                    if (nv == nx) d += w;
                    if (ov == cx) d -= w;
                } else {
                    if (nv == cx) d += 2 * w;
                    if (ov == cx) d -= 2 * w;
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    return d;
}

// updateVertexCommunity (modularity_optimisation.cu:237-249) for one
// sub-round's vertices, with exact Sigma_tot and size updates; *drift gets
// the thread's share of the drift.
static __device__ __forceinline__ int32_t commit_list(const BatchParams &P, const GState &gs, const Team &t,
                                               const int32_t *list, int32_t n, u64 *drift) {
    int32_t moved = 0;
    u64 dd = 0;
    for (int32_t i = t.tid(); i < n; i += t.threads()) {
        const int32_t v = list[i];
        const int32_t nc = P.newc[v], oc = P.comm[v];
        if (nc == oc) continue;
        P.comm[v] = nc;
        atomicSub(P.size + oc, 1);
        atomicAdd(P.size + nc, 1);
        const u64 kv = P.k[v];
        atomicAdd(P.S + oc, (u64)0 - kv);
        atomicAdd(P.S + nc, kv);
        dd += gs.drift_of(kv);
        ++moved;
    }
    *drift = dd;
    return moved;
}

// One sweep: the seven sub-rounds, each deciding against the state committed
// before it.  Returns this thread's moves; *de receives its share of the exact
// change of sum_i e_{i->C(i)}.
static __device__ u64 sweep(const Rows &L, const BatchParams &P, const GState &gs, Team &t, BatchSmem &sm, u64 *de) {
    u64 moved = 0, d = 0;
    const int32_t *bl = P.blist + gs.v0;
    volatile u64 *drift_at = t.nc == 1 ? &sm.drift : &t.scr->drift;
    for (int b = 0; b < NBUCKETS; ++b) {
        const int32_t o = sm.boff[2 * b], ns = sm.bcnt[2 * b], nb = sm.bcnt[2 * b + 1];
        if (ns + nb == 0) continue;
        const u64 drift = *drift_at;
        // one code path for the short buckets and one for the longer rows: the
        // kernel's code would not fit the instruction cache with one per bucket
        if (b < 3) decide_groups<4, 4>(L, P, gs, t, bl + o, ns, 3 + b, drift, sm);
        else if (b == 3) decide_groups<8, 4>(L, P, gs, t, bl + o, ns, 6, drift, sm);
        else if (ns) decide_groups<32, 4>(L, P, gs, t, bl + o, ns, 8, drift, sm);
        if (nb) decide_wide(L, P, gs, t, bl + o + ns, nb, drift, sm);
        t.sync();
        if (nb && t.tid() == 0) *(t.nc == 1 ? &sm.nbig : &t.scr->nbig) = 0;   // used again after the barriers below
        d += commit_delta(L, P, gs, t, bl + o, ns + nb, sm);
        t.sync();
        u64 dd = 0;
        const int32_t mv = commit_list(P, gs, t, bl + o, ns + nb, &dd);
        moved += (u64)mv;
        if (gs.skip && __any_sync(FULL, mv != 0)) {
            dd = warp_sum_u64(dd);
            if ((threadIdx.x & 31) == 0) atomicAdd((u64 *)drift_at, dd);
        }
        t.sync();
    }
    *de = d;
    return moved;
}

// This thread's share of sum_i e_{i->C(i)} over whole rows, self-loops included
// (calculateToOwnCommunity, modularity_optimisation.cu:365-393).
static __device__ u64 own_weight(const Rows &L, const BatchParams &P, const GState &gs, const Team &t) {
    const int lane = threadIdx.x & 31;
    u64 eo = 0;
    for (int32_t i0 = t.warp() * 4; i0 < gs.V; i0 += t.warps() * 4) {
        const int32_t i = i0 + (lane >> 3);
        if (i >= gs.V) continue;
        const int32_t v = gs.v0 + i;
        const int32_t cv = P.comm[v];
        const int32_t r1 = L.r1(v);
        for (int32_t e = L.r0(v) + (lane & 7); e < r1; e += 8)
            if (P.comm[L.c(e)] == cv) eo += L.x(e);
    }
    return eo;
}

// This thread's share of sum_C Sigma_tot^2.
static __device__ __forceinline__ u128 s2_part(const BatchParams &P, const GState &gs, const Team &t) {
    u128 s2 = 0;
    for (int32_t i = t.tid(); i < gs.V; i += t.threads()) {
        const u64 s = P.S[gs.v0 + i];
        s2 += (u128)s * (u128)s;
    }
    return s2;
}

// Level set-up: k_i (level 0; aggregation writes it for later levels),
// singleton communities, Sigma_tot = k, and the bucket lists.
static __device__ void level_setup(const Rows &L, const BatchParams &P, GState &gs, Team &t, BatchSmem &sm) {
    const int lane = threadIdx.x & 31;
    const int32_t v0 = gs.v0, V = gs.V;
    if (gs.cur < 0) {
        Totals5 tt{};
        for (int32_t i0 = t.warp() * 4; i0 < V; i0 += t.warps() * 4) {
            const int32_t i = i0 + (lane >> 3);
            u64 s = 0;
            if (i < V) {
                const int32_t r1 = L.r1(v0 + i);
                for (int32_t e = L.r0(v0 + i) + (lane & 7); e < r1; e += 8) {
                    const u64 x = P.w ? wfix(P.w, e, gs.scale) : L.w64[e];
                    if (gs.narrow) const_cast<uint32_t *>(L.w32)[e] = (uint32_t)x;
                    else if (P.w) const_cast<u64 *>(L.w64)[e] = x;
                    const int32_t j = L.c(e);
                    s += x;
                    tt.b += sym_share(v0 + i, j, x);
                }
            }
            for (int off = 4; off > 0; off >>= 1) s += __shfl_xor_sync(FULL, s, off);
            if (i < V && (lane & 7) == 0) {
                P.k[v0 + i] = s;
                tt.a += s;
            }
        }
        tt = team_totals(tt, t, sm);
        gs.T = tt.a;
        gs.sym = tt.b == 0;
        gs.skip = gs.sym && gs.E >= SKIP_MIN_ENTRIES;
        // T in at most 2^40 drift units: the drift of a level stays far below 2^62
        gs.dsh = max(0, 64 - __clzll((long long)gs.T) - 40);
        gs.dunit = ldexpf(1.0f, -gs.dsh);
    }
    if (threadIdx.x < 16) sm.bcnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        sm.drift = 0;
        sm.nbig = 0;
        if (t.nc > 1 && t.rank == 0) {
            t.scr->drift = 0;
            t.scr->nbig = 0;
        }
    }
    __syncthreads();
    // k of an aggregated level, and the rows, were written before the last barrier
    for (int32_t i = t.tid(); i < V; i += t.threads()) {
        const int32_t v = v0 + i;
        P.comm[v] = v;
        P.newc[v] = v;
        P.size[v] = 1;
        P.S[v] = P.k[v];
        P.lim[v] = 0;
        const int32_t d = L.r1(v) - L.r0(v);
        const int b = bucket_of(d);
        if (b >= 0) atomicAdd(&sm.bcnt[2 * b + (d > DW ? 1 : 0)], 1);
    }
    __syncthreads();
    int32_t mine = 0;
    if (t.nc > 1) {
        if (threadIdx.x < 16) {
            mine = sm.bcnt[threadIdx.x];
            if (mine) atomicAdd(&t.scr->cnt[threadIdx.x], mine);
        }
        t.sync();
        if (threadIdx.x < 16) sm.bcnt[threadIdx.x] = __ldcg(&t.scr->cnt[threadIdx.x]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int32_t o = 0;
        for (int j = 0; j < 2 * NBUCKETS; ++j) {
            sm.boff[j] = o;
            sm.bcur[j] = o;
            o += sm.bcnt[j];
        }
    }
    __syncthreads();
    if (t.nc > 1) {
        // this CTA's part of each bucket's range
        if (threadIdx.x < 2 * NBUCKETS && mine) sm.bcur[threadIdx.x] += atomicAdd(&t.scr->cur[threadIdx.x], mine);
        __syncthreads();
    }
    for (int32_t i = t.tid(); i < V; i += t.threads()) {
        const int32_t d = L.r1(v0 + i) - L.r0(v0 + i);
        const int b = bucket_of(d);
        if (b >= 0) P.blist[v0 + atomicAdd(&sm.bcur[2 * b + (d > DW ? 1 : 0)], 1)] = v0 + i;
    }
    t.sync();
    if (t.nc > 1 && t.rank == 0 && threadIdx.x < 16) {
        t.scr->cnt[threadIdx.x] = 0;   // read again only after this level's barriers
        t.scr->cur[threadIdx.x] = 0;
    }
}

// optimiseModularity (modularity_optimisation.cu:284-363): sweeps while the
// sweep's gain >= min_gain (the first always runs), stopping after a sweep
// without moves; changed = some sweep gained (> 0).  Then
// originalToCommunity <- C(originalToCommunity) (:251-257, :361).
static __device__ int optimise_level(const Rows &L, const BatchParams &P, const GState &gs, Team &t, BatchSmem &sm,
                              int *status) {
    Totals5 tt{};
    tt.a = own_weight(L, P, gs, t);
    tt.s2 = s2_part(P, gs, t);
    tt = team_totals(tt, t, sm);
    u64 &e_own = sm.e_own;
    double &q_before = sm.q_before;
    if (threadIdx.x == 0) {
        e_own = tt.a;
        q_before = modularity_from(gs, tt.a, tt.s2);
    }
    __syncthreads();
    double gain = P.min_gain;
    int changed = 0, sw = 0;
    while (gain >= P.min_gain) {
        if (P.max_sweeps > 0 && sw >= P.max_sweeps) break;
        if (sw >= P.sweep_cap) {
            *status = LV_ERR_DEVICE;
            break;
        }
        tt = Totals5{};
        tt.b = sweep(L, P, gs, t, sm, &tt.a);
        tt.s2 = s2_part(P, gs, t);
        tt.err = (u64)(unsigned)sm.err;
        tt = team_totals(tt, t, sm);
        const int64_t moves = (int64_t)tt.b;
        ++sw;
        if (threadIdx.x == 0) sm.acc.moves += moves;
        if (tt.err) {
            *status = LV_ERR_DEVICE;
            break;
        }
        const u64 e_now = e_own + tt.a;
        const double q_after = modularity_from(gs, e_now, tt.s2);
        gain = __dsub_rn(q_after, q_before);
        if (gain > 0) changed = 1;
        __syncthreads();
        if (threadIdx.x == 0) {
            e_own = e_now;
            q_before = q_after;
        }
        if (moves == 0) break;
    }
    if (threadIdx.x == 0) {
        Acc &acc = sm.acc;
        acc.sweeps += sw;
        acc.edge_sweeps += (int64_t)sw * gs.E;
        acc.vertex_sweeps += (int64_t)sw * gs.V;
        acc.q = q_before;
    }
    for (int32_t u = t.tid(); u < gs.V0; u += t.threads()) {
        const int32_t x = P.o2c[gs.v0 + u];
        P.o2c[gs.v0 + u] = P.comm[x];
    }
    t.sync();
    return changed;
}

// aggregateCommunities (community_aggregation.cu:248-347): nonempty
// communities renumbered in ascending old id; each new vertex's row is the sum
// of its members' rows keyed by the neighbours' new ids (intra-community
// entries become one self-loop); new k = row sum; originalToCommunity <-
// newID (:222-228).  Rows are written at the offset of their bound (the sum of
// the members' degrees) inside the graph's entry range and stay there.
// Returns whether a device check failed.
static __device__ bool aggregate(const Rows &L, const BatchParams &P, GState &gs, Team &t, BatchSmem &sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = gs.cur < 0 ? 0 : 1 - gs.cur;
    const int32_t v0 = gs.v0, V = gs.V;
    const int32_t tid = t.tid(), tn = t.threads();
    int32_t *nbig_at = t.nc == 1 ? &sm.nbig : &t.scr->nbig;
    int32_t *ms = P.mstart + v0 + gs.g;
    int32_t *ro = P.roff + v0 + gs.g;
    int32_t *nid = P.newid;
    const int32_t nv = team_scan(
        V, [&](int32_t i) { return P.size[v0 + i] > 0 ? 1 : 0; },
        [&](int32_t i, int32_t pre, int32_t x) { nid[v0 + i] = x ? pre : -1; }, t, sm);
    for (int32_t i = tid; i <= nv; i += tn) {
        ms[i] = 0;
        ro[i] = 0;
    }
    t.sync();
    for (int32_t i = tid; i < V; i += tn) {
        const int32_t v = v0 + i;
        const int32_t c = nid[P.comm[v]];
        atomicAdd(ms + c, 1);
        atomicAdd(ro + c, L.r1(v) - L.r0(v));
    }
    t.sync();
    team_scan(nv + 1, [&](int32_t i) { return ms[i]; },
              [&](int32_t i, int32_t pre, int32_t) {
                  ms[i] = pre;
                  if (i < nv) P.newc[v0 + i] = pre;
              }, t, sm);
    team_scan(nv + 1, [&](int32_t i) { return ro[i]; }, [&](int32_t i, int32_t pre, int32_t) { ro[i] = pre; }, t,
              sm);
    if (tid == 0) *nbig_at = 0;
    for (int32_t i = tid; i < V; i += tn) {
        const int32_t v = v0 + i;
        const int32_t pos = atomicAdd(P.newc + v0 + nid[P.comm[v]], 1);
        P.members[v0 + pos] = v;
    }
    t.sync();

    int32_t *ocol = P.colb[nb];
    u64 *ow = P.wb[nb];
    int32_t *ors = P.rs[nb], *ore = P.re[nb];
    u64 enew = 0;
    // merged rows of bound <= DW: one warp each, table in the warp's slots
    for (int32_t c = t.warp(); c < nv; c += t.warps()) {
        const int32_t bound = ro[c + 1] - ro[c];
        if (bound > DW) {
            if (lane == 0) P.blist[v0 + atomicAdd(nbig_at, 1)] = c;
            continue;
        }
        const int lg = table_lg(min(bound, nv));
        int32_t *keys = sm.keys + warp * WTAB;
        u64 *vals = sm.vals + warp * WTAB;
        u64 self = 0;   // weight inside the community (its self-loop), summed in registers
        bool any = false;
        for (int32_t j = ms[c]; j < ms[c + 1]; ++j) {
            const int32_t m = P.members[v0 + j];
            const int32_t r1 = L.r1(m);
            for (int32_t e = L.r0(m) + lane; e < r1; e += 32) {
                const int32_t key = nid[P.comm[L.c(e)]];
                if (key == c) {
                    self += L.x(e);
                    any = true;
                } else {
                    table_insert<1>(keys, vals, lg, key, L.x(e), &sm.err);
                }
            }
        }
        if (any) table_insert<1>(keys, vals, lg, c, self, &sm.err);
        __syncwarp();
        const int64_t base = gs.e0 + ro[c];
        int32_t cnt = 0;
        u64 ks = 0;
        for (int s0 = 0; s0 < (1 << lg); s0 += 32) {
            const int s = s0 + lane;
            const int32_t key = s < (1 << lg) ? keys[s] : -1;
            const unsigned bal = __ballot_sync(FULL, key >= 0);
            if (key >= 0) {
                const int32_t pos = cnt + __popc(bal & ((1u << lane) - 1u));
                const u64 x = vals[s];
                if (pos < bound) {
                    ocol[base + pos] = v0 + key;
                    ow[base + pos] = x;
                } else {
                    atomicOr(&sm.err, DEVERR_BAD_STATE);
                }
                ks += x;
                keys[s] = -1;
                vals[s] = 0;
            }
            cnt += __popc(bal);
        }
        __syncwarp();
        ks = warp_sum_u64(ks);
        if (lane == 0) {
            ors[v0 + c] = (int32_t)base;
            ore[v0 + c] = (int32_t)(base + cnt);
            P.k[v0 + c] = ks;
            enew += (u64)cnt;
        }
    }
    t.sync();
    // larger merged rows: a whole CTA each (the first CTA for those that need
    // the graph's one global table)
    const int32_t nbig = *(volatile int32_t *)nbig_at;
    for (int pass = 0; pass < (t.nc > 1 ? 2 : 1); ++pass) {
        if (pass == 1 && t.rank != 0) break;
        for (int32_t b = pass ? 0 : t.rank; b < nbig; b += pass ? 1 : t.nc) {
            const int32_t c = P.blist[v0 + b];
            const int32_t bound = ro[c + 1] - ro[c];
            const int lg = table_lg(min(bound, nv));
            if (t.nc > 1 && ((1 << lg) > CTAB) != (pass == 1)) continue;
            int32_t *keys = sm.keys;
            u64 *vals = sm.vals;
            if ((1 << lg) > CTAB) {
                keys = P.tkeys + gs.tbl;
                vals = P.tvals + gs.tbl;
            }
            u64 self = 0;
            bool any = false;
            for (int32_t j = ms[c] + warp; j < ms[c + 1]; j += BW) {
                const int32_t m = P.members[v0 + j];
                const int32_t r1 = L.r1(m);
                for (int32_t e = L.r0(m) + lane; e < r1; e += 32) {
                    const int32_t key = nid[P.comm[L.c(e)]];
                    if (key == c) {
                        self += L.x(e);
                        any = true;
                    } else {
                        table_insert<1>(keys, vals, lg, key, L.x(e), &sm.err);
                    }
                }
            }
            if (any) table_insert<1>(keys, vals, lg, c, self, &sm.err);
            if (threadIdx.x == 0) sm.cnt = 0;
            __syncthreads();
            const int64_t base = gs.e0 + ro[c];
            u64 ks = 0;
            for (int32_t s0 = 0; s0 < (1 << lg); s0 += BT) {
                const int32_t s = s0 + threadIdx.x;
                const int32_t key = s < (1 << lg) ? keys[s] : -1;
                const unsigned bal = __ballot_sync(FULL, key >= 0);
                int32_t wbase = 0;
                if (lane == 0 && bal) wbase = atomicAdd(&sm.cnt, __popc(bal));
                wbase = __shfl_sync(FULL, wbase, 0);
                if (key >= 0) {
                    const int32_t pos = wbase + __popc(bal & ((1u << lane) - 1u));
                    const u64 x = vals[s];
                    if (pos < bound) {
                        ocol[base + pos] = v0 + key;
                        ow[base + pos] = x;
                    } else {
                        atomicOr(&sm.err, DEVERR_BAD_STATE);
                    }
                    ks += x;
                    keys[s] = -1;
                    vals[s] = 0;
                }
            }
            const u64 ktot = block_sum_u64(ks, sm);
            if (threadIdx.x == 0) {
                const int32_t cnt = sm.cnt;
                ors[v0 + c] = (int32_t)base;
                ore[v0 + c] = (int32_t)(base + cnt);
                P.k[v0 + c] = ktot;
                enew += (u64)cnt;
            }
            __syncthreads();
        }
    }
    for (int32_t u = tid; u < gs.V0; u += tn) {
        const int32_t x = P.o2c[v0 + u];
        P.o2c[v0 + u] = v0 + nid[x];
    }
    __syncthreads();
    Totals5 tt{};
    tt.a = enew;
    tt.err = (u64)(unsigned)sm.err;
    tt = team_totals(tt, t, sm);
    gs.V = nv;
    gs.E = (int64_t)tt.a;
    gs.cur = nb;
    return tt.err != 0;
}

// Range check and fixed-point scale of a batch's graph (orc_choose_scale):
// returns its status.
static __device__ int graph_scale(const BatchParams &P, GState &gs, Team &t, BatchSmem &sm) {
    int need = 0, top = 0, bad = 0;
    for (int64_t e = gs.e0 + t.tid(); e < gs.e0 + gs.E; e += t.threads()) {
        const int32_t j = __ldg(P.col + e);
        if (j < gs.v0 || j >= gs.v0 + gs.V0) bad = 1;
        int n, tp, b;
        weight_bits_dev(__ldg(P.w + e), n, tp, b);
        need = max(need, n);
        top = max(top, tp);
        bad |= b;
    }
    need = block_max_i32(need, sm);
    top = block_max_i32(top, sm);
    bad = block_max_i32(bad, sm);
    if (t.nc > 1) {
        u64(*red)[6] = t.scr->red[t.par];
        t.par ^= 1;
        if (threadIdx.x == 0) {
            red[t.rank][0] = (u64)need;
            red[t.rank][1] = (u64)top;
            red[t.rank][2] = (u64)bad;
        }
        t.sync();
        for (int r = 0; r < t.nc; ++r) {
            need = max(need, (int)__ldcg(&red[r][0]));
            top = max(top, (int)__ldcg(&red[r][1]));
            bad = max(bad, (int)__ldcg(&red[r][2]));
        }
    }
    if (bad) return LV_ERR_INVALID;
    const int tp = top ? top - 1024 : 0;
    const int cap = 61 - tp - ceil_log2_i(gs.E > 0 ? gs.E : 1);
    const int sc = need < cap ? need : cap;
    if (sc < 0) return LV_ERR_TOO_LARGE;
    gs.scale = ldexp(1.0, sc);
    gs.narrow = !top || tp + 1 + sc <= 31;   // every weight is at most 2^(tp + 1 + sc)
    return LV_OK;
}

// The whole level loop of one graph (gpulouvain.cu:30-37).
static __device__ void run_graph(const BatchParams &P, int32_t g, Team &t, BatchSmem &sm) {
    GState &gs = sm.gs;
    gs.g = g;
    gs.v0 = P.job ? 0 : P.gptr[g];
    gs.V0 = P.job ? P.job_V : P.gptr[g + 1] - gs.v0;
    gs.V = gs.V0;
    gs.e0 = P.job ? 0 : __ldg(P.rowptr + gs.v0);
    gs.E = P.job ? P.job_E : (int64_t)__ldg(P.rowptr + gs.v0 + gs.V0) - gs.e0;
    gs.tbl = P.job ? 0 : P.tbl_off[g];
    gs.T = 0;
    gs.scale = P.job_scale;
    gs.cur = -1;
    gs.dsh = 0;
    gs.dunit = 1.0f;
    gs.narrow = P.job_narrow != 0;
    gs.sym = false;
    gs.skip = false;
    if (threadIdx.x == 0) sm.err = 0;
    for (int s = threadIdx.x; s < CTAB; s += BT) {
        sm.keys[s] = -1;
        sm.vals[s] = 0;
        sm.hi[s] = 0;
    }
    Acc &acc = sm.acc;
    if (threadIdx.x == 0) acc = Acc{};
    int status = LV_OK;
    int32_t levels = 0;
    if (P.job) {
        // the scratch area and the graph's table are this launch's own
        if (t.tid() == 0) {
            t.scr->nbig = 0;
            for (int i = 0; i < 16; ++i) t.scr->cnt[i] = t.scr->cur[i] = 0;
        }
        const int32_t n = 1 << ceil_log2_i(2 * (int64_t)gs.V0);
        for (int32_t s = t.tid(); s < n; s += t.threads()) {
            P.tkeys[s] = -1;
            P.tvals[s] = 0;
        }
        t.sync();
    } else {
        if (t.tid() == 0) P.t_start[g] = globaltimer();
        status = graph_scale(P, gs, t, sm);
    }
    if (status == LV_OK) {
        for (int32_t u = t.tid(); u < gs.V0; u += t.threads()) P.o2c[gs.v0 + u] = gs.v0 + u;
        for (;;) {
            Rows &L = sm.rows;
            __syncthreads();
            if (gs.cur < 0) {
                // level 0's fixed-point weights use the graph's part of the second
                // weight buffer, which the first aggregation does not write
                L.rs = P.rowptr;
                L.re = P.rowend;
                L.col = P.col;
                L.w64 = P.w ? P.wb[1] : P.s_w64;
                L.w32 = gs.narrow ? reinterpret_cast<const uint32_t *>(P.wb[1] + gs.e0) - gs.e0 : nullptr;
            } else {
                L.rs = P.rs[gs.cur];
                L.re = P.re[gs.cur];
                L.col = P.colb[gs.cur];
                L.w64 = P.wb[gs.cur];
                L.w32 = nullptr;
            }
            level_setup(L, P, gs, t, sm);
            const int changed = optimise_level(L, P, gs, t, sm, &status);
            ++levels;
            if (!changed || status != LV_OK) break;
            if (aggregate(L, P, gs, t, sm) || levels >= P.level_cap) {
                status = LV_ERR_DEVICE;
                break;
            }
        }
    }
    if (P.job) {
        if (t.tid() == 0) {
            P.job->q = acc.q;
            P.job->status = status;
            P.job->V = gs.V;
            P.job->levels = levels;
            P.job->cur = gs.cur;
            P.job->E = gs.E;
            P.job->sweeps = acc.sweeps;
            P.job->edge_sweeps = acc.edge_sweeps;
            P.job->vertex_sweeps = acc.vertex_sweeps;
            P.job->moves = acc.moves;
        }
        return;
    }
    if (status != LV_OK) {
        // leave the graph's global table empty for the next run
        const int64_t n = P.tbl_off[g + 1] - gs.tbl;
        for (int64_t s = t.tid(); s < n; s += t.threads()) {
            P.tkeys[gs.tbl + s] = -1;
            P.tvals[gs.tbl + s] = 0;
        }
    }
    for (int32_t u = t.tid(); u < gs.V0; u += t.threads())
        P.out_comm[gs.v0 + u] = status == LV_OK ? P.o2c[gs.v0 + u] - gs.v0 : -1;
    if (t.tid() == 0) {
        P.q[g] = acc.q;
        P.nc[g] = status == LV_OK ? gs.V : 0;
        P.status[g] = status;
        P.levels[g] = levels;
        P.sweeps[g] = acc.sweeps;
        P.edge_sweeps[g] = acc.edge_sweeps;
        P.vertex_sweeps[g] = acc.vertex_sweeps;
        P.moves[g] = acc.moves;
        P.t_end[g] = globaltimer();
    }
    t.sync();
}

};

__device__ __forceinline__ int32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int32_t)r;
}
__device__ __forceinline__ int32_t cluster_ctas() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return (int32_t)r;
}

// Cluster i of a launch runs graph order[lo + i].
__global__ void __launch_bounds__(BT, 1024 / BT) batch_kernel(const __grid_constant__ BatchParams P) {
    extern __shared__ __align__(16) unsigned char batch_smem[];
    Loop::BatchSmem &sm = *reinterpret_cast<Loop::BatchSmem *>(batch_smem);
    Loop::Team t;
    t.nc = cluster_ctas();
    t.rank = t.nc > 1 ? cluster_rank() : 0;
    t.par = 0;
    const int32_t i = P.lo + (int32_t)blockIdx.x / t.nc;
    t.scr = P.scratch + i;
    Loop::run_graph(P, P.job ? 0 : P.order[i], t, sm);
}

// first entry of each graph: out[g] = rowptr[gptr[g]]
__global__ void graph_entries_kernel(const int32_t *rowptr, const int32_t *gptr, int32_t G,
                                     int32_t *out) {
    for (int32_t g = blockIdx.x * 256 + threadIdx.x; g <= G; g += gridDim.x * 256)
        out[g] = rowptr[gptr[g]];
}

__global__ void fill_tables_kernel(int32_t *keys, u64 *vals, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        keys[i] = -1;
        vals[i] = 0;
    }
}

void launch_config(cudaStream_t s, int ctas, int cluster, cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(BT);
    cfg.dynamicSmemBytes = sizeof(Loop::BatchSmem);
    cfg.stream = s;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)cluster;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
}

// Dynamic shared memory and cluster attributes of batch_kernel (once per
// device and process); the widest cluster the device takes.
int widest_team(int device) {
    static std::mutex mu;
    static int widest[64] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (device >= 0 && device < 64 && widest[device]) return widest[device];
    if (cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(Loop::BatchSmem)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    int cl = TEAM_MAX;
    for (; cl > 1; cl /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        launch_config(0, cl, cl, cfg, at);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, batch_kernel, &cfg) == cudaSuccess && n > 0) break;
    }
    cudaGetLastError();
    if (device >= 0 && device < 64) widest[device] = cl;
    return cl;
}

}  // namespace
}  // namespace lv

using namespace lv;

namespace {
// Layout of a team run's arena for V vertices and E entries.
struct TeamArena {
    size_t at = 0;
    template <typename T>
    T *take(unsigned char *base, size_t n) {
        at = (at + 255) / 256 * 256;
        T *p = reinterpret_cast<T *>(base + at);
        at += n * sizeof(T);
        return p;
    }
    BatchParams lay(unsigned char *base, int32_t V, int64_t E) {
        BatchParams P{};
        at = 0;
        const size_t v = (size_t)V + 1, e = (size_t)E + 1;
        P.job = take<TeamResult>(base, 1);
        P.scratch = take<TeamScratch>(base, 1);
        P.o2c = take<int32_t>(base, v);
        P.blist = take<int32_t>(base, v);
        P.newid = take<int32_t>(base, v);
        P.members = take<int32_t>(base, v);
        P.mstart = take<int32_t>(base, v);
        P.roff = take<int32_t>(base, v);
        P.lim = take<u64>(base, v);
        for (int i = 0; i < 2; ++i) {
            P.rs[i] = take<int32_t>(base, v);
            P.re[i] = take<int32_t>(base, v);
            P.colb[i] = take<int32_t>(base, e);
            P.wb[i] = take<u64>(base, e);
        }
        const size_t slots = (size_t)1 << ceil_log2_i(2 * (int64_t)V);
        P.tkeys = take<int32_t>(base, slots);
        P.tvals = take<u64>(base, slots);
        return P;
    }
};
}  // namespace

size_t lv::team_arena_bytes(int32_t V, int64_t E) {
    TeamArena a;
    a.lay(nullptr, V, E);
    return a.at;
}

int lv::team_run(const TeamJob &j, void *arena, int device, cudaStream_t s, TeamRows *rows) {
    TeamArena a;
    BatchParams P = a.lay((unsigned char *)arena, j.V, j.E);
    P.rowptr = j.rs;
    P.rowend = j.re;
    P.col = j.col;
    P.w = j.w;
    P.s_w64 = j.w64;
    P.job_V = j.V;
    P.job_E = j.E;
    P.job_scale = j.scale;
    P.job_narrow = j.w && j.narrow;
    P.sweep_cap = TEAM_RUN_SWEEP_CAP;
    P.level_cap = 1 << 20;
    P.max_sweeps = j.max_sweeps;
    P.min_gain = j.min_gain;
    P.comm = j.comm;
    P.newc = j.newc;
    P.size = j.size;
    P.k = j.k;
    P.S = j.S;
    const int widest = widest_team(device);
    if (!widest) return 0;
    int nc = 1;
    while (nc < widest && (double)j.E > TEAM_MIN_PART * nc) nc *= 2;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    launch_config(s, nc, nc, cfg, at);
    if (cudaLaunchKernelEx(&cfg, batch_kernel, P) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    note_launches(1);
    rows->result = P.job;
    rows->o2c = P.o2c;
    for (int i = 0; i < 2; ++i) {
        rows->rs[i] = P.rs[i];
        rows->re[i] = P.re[i];
        rows->col[i] = P.colb[i];
        rows->w64[i] = P.wb[i];
    }
    return 1;
}

struct lv_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    lv_opts opts{};
    std::string err;
    int32_t G = 0, V = 0;
    int64_t E = 0;
    std::vector<int32_t> gptr_h;
    std::vector<int64_t> entries_h;   // [G] entries per graph
    const int32_t *rowptr = nullptr, *col = nullptr;
    const float *w = nullptr;
    BatchParams P{};
    int64_t tbl_total = 0;
    MemSet mem;
    struct Tier { int nc; int32_t lo, hi; };   // CTAs per graph, graphs order[lo .. hi)
    std::vector<Tier> tiers;
    std::vector<cudaStream_t> side;            // streams of the launches after the first
    std::vector<cudaEvent_t> side_ev;
    bool ran = false;
    bool tables_dirty = false;
    float last_ms = 0;
    int64_t last_edge_sweeps = 0, last_vertex_sweeps = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace {

int bfail(lv_batch *b, int code, const std::string &msg) {
    if (b) b->err = msg;
    return code;
}

template <typename T>
int balloc(lv_batch *b, T **p, size_t n) {
    void *q = nullptr;
    const cudaError_t e = b->mem.alloc(&q, sizeof(T) * n, b->stream);
    *p = (T *)q;
    if (e != cudaSuccess) return bfail(b, LV_ERR_NOMEM, "device allocation failed");
    return LV_OK;
}

#define LVB_TRY(expr)           \
    do {                        \
        int rc__ = (expr);      \
        if (rc__) return rc__;  \
    } while (0)

#define LVB_CUDA(b, call)                                                                      \
    do {                                                                                       \
        cudaError_t e__ = (call);                                                              \
        if (e__ != cudaSuccess) {                                                              \
            cudaGetLastError();                                                                \
            return bfail((b), LV_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__)); \
        }                                                                                      \
    } while (0)

int batch_sync(lv_batch *b) {
    LVB_CUDA(b, cudaStreamSynchronize(b->stream));
    LVB_CUDA(b, cudaGetLastError());
    return LV_OK;
}

int batch_begin(const int32_t *graph_ptr, int32_t G, int32_t V, int64_t E, const lv_opts *opts,
                lv_batch **out, lv_batch **bp) {
    if (!out) return LV_ERR_INVALID;
    *out = nullptr;
    if (G < 0 || V < 0 || E < 0 || (G > 0 && !graph_ptr)) return LV_ERR_INVALID;
    if (E > 0x7fffffffLL || (int64_t)V + G >= 0x7fffffffLL) return LV_ERR_TOO_LARGE;
    if (G > 0 && (graph_ptr[0] != 0 || graph_ptr[G] != V)) return LV_ERR_INVALID;
    for (int32_t g = 0; g < G; ++g) {
        if (graph_ptr[g + 1] < graph_ptr[g]) return LV_ERR_INVALID;
        if (graph_ptr[g + 1] - graph_ptr[g] > LV_BATCH_MAX_GRAPH_VERTICES) return LV_ERR_TOO_LARGE;
    }
    if (G == 0 && V != 0) return LV_ERR_INVALID;
    lv_batch *b = new lv_batch();
    lv_default_opts(&b->opts);
    if (opts) {
        size_t n = opts->struct_size && opts->struct_size < sizeof(lv_opts) ? opts->struct_size : sizeof(lv_opts);
        std::memcpy(&b->opts, opts, n);
        b->opts.struct_size = sizeof(lv_opts);
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        delete b;
        return LV_ERR_NO_DEVICE;
    }
    if (b->opts.device < 0 || b->opts.device >= ndev) {
        delete b;
        return LV_ERR_INVALID;
    }
    b->device = b->opts.device;
    cudaSetDevice(b->device);
    b->mem.dev = b->device;
    if (stream_take(b->device, &b->stream) != cudaSuccess) {
        cudaGetLastError();
        delete b;
        return LV_ERR_CUDA;
    }
    cudaEventCreate(&b->ev0);
    cudaEventCreate(&b->ev1);
    b->G = G;
    b->V = V;
    b->E = E;
    b->gptr_h.assign(graph_ptr, graph_ptr + (G > 0 ? G + 1 : 0));
    *bp = b;
    return LV_OK;
}

// Launches by graph size (the order is by decreasing entries): the larger the
// graph, the more CTAs run it, one per part of its entries, rounded up to a
// power of two and at most 16 (the largest cluster).
int plan_launch(lv_batch *b, const std::vector<int32_t> &order) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    const int widest = widest_team(b->device);
    if (!widest) return bfail(b, LV_ERR_CUDA, "batch kernel attributes");
    int64_t total = 0;
    for (int64_t e : b->entries_h) total += e;
    const int resident = 2 * (sms > 0 ? sms : 148);
    const double share = (double)total / resident;
    double part = std::max(BATCH_MIN_PART, TEAM_PART * share);
    auto team_of = [&](int32_t i) {
        const double e = (double)b->entries_h[order[i]];
        int nc = 1;
        while (nc < widest && e > part * nc) nc *= 2;
        return nc;
    };
    for (; part < TEAM_FIT_PART; part *= 1.2) {
        int64_t ctas = 0;
        for (int32_t i = 0; i < b->G && (double)b->entries_h[order[i]] > 0.5 * share; ++i) ctas += team_of(i);
        if (ctas <= resident) break;
    }
    b->tiers.clear();
    for (int32_t i = 0; i < b->G; ++i) {
        const int nc = team_of(i);
        if (b->tiers.empty() || b->tiers.back().nc != nc) b->tiers.push_back({nc, i, i});
        b->tiers.back().hi = i + 1;
    }
    return LV_OK;
}

int batch_finish(lv_batch *b) {
    const int32_t G = b->G, V = b->V;
    const int64_t E = b->E;
    BatchParams &P = b->P;
    // whole-CSR checks: offsets, column ids, weights
    int32_t *chk = nullptr;
    LVB_TRY(balloc(b, &chk, 8 + (size_t)G + 1));
    LVB_CUDA(b, cudaMemsetAsync(chk, 0, sizeof(int32_t) * 8, b->stream));
    launch_csr_scan(b->rowptr, b->col, b->w, V, E, chk, chk + 4, nullptr, 0, b->stream);
    int32_t *gptr_d = nullptr;
    LVB_TRY(balloc(b, &gptr_d, (size_t)G + 1));
    if (G > 0) {
        LVB_CUDA(b, cudaMemcpyAsync(gptr_d, b->gptr_h.data(), sizeof(int32_t) * ((size_t)G + 1),
                                    cudaMemcpyHostToDevice, b->stream));
    }
    std::vector<int32_t> hchk(8 + (size_t)G + 1, 0);
    LVB_CUDA(b, cudaMemcpyAsync(hchk.data(), chk, sizeof(int32_t) * 8, cudaMemcpyDeviceToHost, b->stream));
    LVB_TRY(batch_sync(b));
    if (hchk[0]) return bfail(b, LV_ERR_INVALID, "malformed CSR (offsets or column ids)");
    if (hchk[6]) return bfail(b, LV_ERR_WEIGHT, "negative, NaN or infinite edge weight");
    // entries per graph, processing order (decreasing entries), table layout
    if (G > 0) {
        graph_entries_kernel<<<(G + 256) / 256, 256, 0, b->stream>>>(b->rowptr, gptr_d, G, chk + 8);
        note_launches(1);
        LVB_CUDA(b, cudaMemcpyAsync(hchk.data() + 8, chk + 8, sizeof(int32_t) * ((size_t)G + 1),
                                    cudaMemcpyDeviceToHost, b->stream));
        LVB_TRY(batch_sync(b));
    }
    b->entries_h.assign(G, 0);
    for (int32_t g = 0; g < G; ++g) b->entries_h[g] = (int64_t)hchk[8 + g + 1] - hchk[8 + g];
    std::vector<int32_t> order(G);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int32_t a, int32_t c) { return b->entries_h[a] > b->entries_h[c]; });
    std::vector<int64_t> toff((size_t)G + 1, 0);
    for (int32_t g = 0; g < G; ++g) {
        const int32_t vg = b->gptr_h[g + 1] - b->gptr_h[g];
        toff[g + 1] = toff[g] + ((int64_t)1 << ceil_log2_i(2 * (int64_t)(vg > 0 ? vg : 1)));
    }
    b->tbl_total = toff[G];
    int32_t *order_d = nullptr;
    int64_t *toff_d = nullptr;
    LVB_TRY(balloc(b, &order_d, (size_t)G));
    LVB_TRY(balloc(b, &toff_d, (size_t)G + 1));
    if (G > 0) {
        LVB_CUDA(b, cudaMemcpyAsync(order_d, order.data(), sizeof(int32_t) * G, cudaMemcpyHostToDevice, b->stream));
        LVB_CUDA(b, cudaMemcpyAsync(toff_d, toff.data(), sizeof(int64_t) * ((size_t)G + 1),
                                    cudaMemcpyHostToDevice, b->stream));
    }
    const size_t nv = (size_t)V + 1, nvg = (size_t)V + G + 1, ne = (size_t)E + 1;
    P.rowptr = b->rowptr;
    P.rowend = b->rowptr + 1;
    P.sweep_cap = SWEEP_CAP;
    P.level_cap = LEVEL_CAP;
    P.job_scale = 1.0;
    P.col = b->col;
    P.w = b->w;
    P.gptr = gptr_d;
    P.order = order_d;
    P.tbl_off = toff_d;
    P.max_sweeps = b->opts.max_sweeps;
    LVB_TRY(balloc(b, &P.comm, nv));
    LVB_TRY(balloc(b, &P.newc, nv));
    LVB_TRY(balloc(b, &P.size, nv));
    LVB_TRY(balloc(b, &P.blist, nv));
    LVB_TRY(balloc(b, &P.newid, nv));
    LVB_TRY(balloc(b, &P.members, nv));
    LVB_TRY(balloc(b, &P.o2c, nv));
    LVB_TRY(balloc(b, &P.mstart, nvg));
    LVB_TRY(balloc(b, &P.roff, nvg));
    for (int i = 0; i < 2; ++i) {
        LVB_TRY(balloc(b, &P.rs[i], nv));
        LVB_TRY(balloc(b, &P.re[i], nv));
        LVB_TRY(balloc(b, &P.colb[i], ne));
        LVB_TRY(balloc(b, &P.wb[i], ne));
    }
    LVB_TRY(balloc(b, &P.k, nv));
    LVB_TRY(balloc(b, &P.S, nv));
    LVB_TRY(balloc(b, &P.lim, nv));
    LVB_TRY(balloc(b, &P.tkeys, (size_t)b->tbl_total));
    LVB_TRY(balloc(b, &P.tvals, (size_t)b->tbl_total));
    LVB_TRY(balloc(b, &P.out_comm, nv));
    LVB_TRY(balloc(b, &P.q, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.nc, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.status, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.levels, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.sweeps, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.edge_sweeps, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.vertex_sweeps, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.moves, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.t_start, (size_t)G + 1));
    LVB_TRY(balloc(b, &P.t_end, (size_t)G + 1));
    if (b->tbl_total > 0) {
        fill_tables_kernel<<<148 * 8, 256, 0, b->stream>>>(P.tkeys, P.tvals, b->tbl_total);
        note_launches(1);
    }
    LVB_TRY(plan_launch(b, order));
    size_t teams = 0;
    for (const auto &t : b->tiers)
        if (t.nc > 1) teams = (size_t)t.hi;   // the team launches come first in order
    LVB_TRY(balloc(b, &P.scratch, teams + 1));
    LVB_CUDA(b, cudaMemsetAsync(P.scratch, 0, sizeof(TeamScratch) * (teams + 1), b->stream));
    for (size_t i = 1; i < b->tiers.size(); ++i) {
        cudaStream_t s = nullptr;
        cudaEvent_t ev = nullptr;
        LVB_CUDA(b, stream_take(b->device, &s));
        b->side.push_back(s);
        LVB_CUDA(b, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        b->side_ev.push_back(ev);
    }
    return batch_sync(b);
}

}  // namespace

extern "C" {

int lv_batch_destroy(lv_batch *b) {
    if (!b) return LV_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    for (cudaStream_t s : b->side) stream_give(b->device, s);
    b->mem.give_all(b->stream);   // the streams have drained
    for (cudaEvent_t e : b->side_ev) cudaEventDestroy(e);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    stream_give(b->device, b->stream);
    delete b;
    return LV_OK;
}

int lv_batch_create(const int32_t *rowptr, const int32_t *col, const float *w, int32_t V, int64_t E,
                    const int32_t *graph_ptr, int32_t num_graphs, const lv_opts *opts, lv_batch **out) {
    if (!rowptr || (E > 0 && (!col || !w))) return LV_ERR_INVALID;
    lv_batch *b = nullptr;
    int rc = batch_begin(graph_ptr, num_graphs, V, E, opts, out, &b);
    if (rc) return rc;
    int32_t *rp = nullptr, *cl = nullptr;
    float *wt = nullptr;
    rc = balloc(b, &rp, (size_t)V + 1);
    if (!rc) rc = balloc(b, &cl, (size_t)E);
    if (!rc) rc = balloc(b, &wt, (size_t)E);
    b->rowptr = rp;
    b->col = cl;
    b->w = wt;
    if (!rc && cudaMemcpyAsync((void *)b->rowptr, rowptr, sizeof(int32_t) * ((size_t)V + 1),
                               cudaMemcpyHostToDevice, b->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc && E > 0 && cudaMemcpyAsync((void *)b->col, col, sizeof(int32_t) * (size_t)E,
                                        cudaMemcpyHostToDevice, b->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc && E > 0 && cudaMemcpyAsync((void *)b->w, w, sizeof(float) * (size_t)E,
                                        cudaMemcpyHostToDevice, b->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc) rc = batch_finish(b);
    if (rc) {
        lv_batch_destroy(b);
        return rc;
    }
    *out = b;
    return LV_OK;
}

int lv_batch_create_device(const int32_t *d_rowptr, const int32_t *d_col, const float *d_w, int32_t V,
                           int64_t E, const int32_t *graph_ptr, int32_t num_graphs, const lv_opts *opts,
                           lv_batch **out) {
    if (!d_rowptr || (E > 0 && (!d_col || !d_w))) return LV_ERR_INVALID;
    lv_batch *b = nullptr;
    int rc = batch_begin(graph_ptr, num_graphs, V, E, opts, out, &b);
    if (rc) return rc;
    b->rowptr = d_rowptr;
    b->col = d_col;
    b->w = d_w;
    rc = batch_finish(b);
    if (rc) {
        lv_batch_destroy(b);
        return rc;
    }
    *out = b;
    return LV_OK;
}

const char *lv_batch_last_error(const lv_batch *b) { return b ? b->err.c_str() : "null batch"; }

int lv_batch_run(lv_batch *b, float min_gain) {
    if (!b) return LV_ERR_INVALID;
    cudaSetDevice(b->device);
    b->err.clear();
    if (b->tables_dirty && b->tbl_total > 0) {
        fill_tables_kernel<<<148 * 8, 256, 0, b->stream>>>(b->P.tkeys, b->P.tvals, b->tbl_total);
        note_launches(1);
        b->tables_dirty = false;
    }
    b->P.min_gain = (double)min_gain;
    cudaEventRecord(b->ev0, b->stream);
    // the launches run side by side: the smaller graphs fill what the larger leave
    for (size_t i = 0; i < b->tiers.size(); ++i) {
        const lv_batch::Tier &t = b->tiers[i];
        const cudaStream_t s = i ? b->side[i - 1] : b->stream;
        if (i) LVB_CUDA(b, cudaStreamWaitEvent(s, b->ev0, 0));
        BatchParams P = b->P;
        P.lo = t.lo;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        launch_config(s, (t.hi - t.lo) * t.nc, t.nc, cfg, at);
        LVB_CUDA(b, cudaLaunchKernelEx(&cfg, batch_kernel, P));
        note_launches(1);
        if (i) LVB_CUDA(b, cudaEventRecord(b->side_ev[i - 1], s));
    }
    for (cudaEvent_t e : b->side_ev) LVB_CUDA(b, cudaStreamWaitEvent(b->stream, e, 0));
    cudaEventRecord(b->ev1, b->stream);
    LVB_TRY(batch_sync(b));
    cudaEventElapsedTime(&b->last_ms, b->ev0, b->ev1);
    b->ran = true;
    // per-graph status and edge-sweeps
    std::vector<int32_t> st(b->G);
    std::vector<int64_t> es(b->G), vs(b->G);
    if (b->G > 0) {
        LVB_CUDA(b, cudaMemcpyAsync(st.data(), b->P.status, sizeof(int32_t) * b->G, cudaMemcpyDeviceToHost, b->stream));
        LVB_CUDA(b, cudaMemcpyAsync(es.data(), b->P.edge_sweeps, sizeof(int64_t) * b->G, cudaMemcpyDeviceToHost,
                                    b->stream));
        LVB_CUDA(b, cudaMemcpyAsync(vs.data(), b->P.vertex_sweeps, sizeof(int64_t) * b->G,
                                    cudaMemcpyDeviceToHost, b->stream));
        LVB_TRY(batch_sync(b));
    }
    int64_t tot = 0, vtot = 0;
    int32_t failed = 0, first = -1;
    for (int32_t g = 0; g < b->G; ++g) {
        tot += es[g];
        vtot += vs[g];
        if (st[g] != LV_OK) {
            if (first < 0) first = g;
            ++failed;
        }
    }
    b->last_edge_sweeps = tot;
    b->last_vertex_sweeps = vtot;
    if (failed) {
        b->tables_dirty = true;
        return bfail(b, LV_ERR_DEVICE,
                     std::to_string(failed) + " graph(s) failed (first: graph " + std::to_string(first) + ", " +
                         lv_status_string(st[first]) + "); see the per-graph status");
    }
    return LV_OK;
}

int lv_batch_get_results(lv_batch *b, int32_t *communities, double *modularity, int32_t *num_communities,
                         int32_t *status) {
    if (!b) return LV_ERR_INVALID;
    if (!b->ran) return bfail(b, LV_ERR_INVALID, "lv_batch_run has not run");
    cudaSetDevice(b->device);
    if (communities && b->V > 0)
        LVB_CUDA(b, cudaMemcpyAsync(communities, b->P.out_comm, sizeof(int32_t) * b->V, cudaMemcpyDeviceToHost,
                                    b->stream));
    if (b->G > 0) {
        if (modularity)
            LVB_CUDA(b, cudaMemcpyAsync(modularity, b->P.q, sizeof(double) * b->G, cudaMemcpyDeviceToHost, b->stream));
        if (num_communities)
            LVB_CUDA(b, cudaMemcpyAsync(num_communities, b->P.nc, sizeof(int32_t) * b->G, cudaMemcpyDeviceToHost,
                                        b->stream));
        if (status)
            LVB_CUDA(b, cudaMemcpyAsync(status, b->P.status, sizeof(int32_t) * b->G, cudaMemcpyDeviceToHost,
                                        b->stream));
    }
    return batch_sync(b);
}

int lv_batch_get_graph_stats(lv_batch *b, int32_t *levels, int64_t *sweeps, int64_t *edge_sweeps,
                             double *latency_ms) {
    if (!b) return LV_ERR_INVALID;
    if (!b->ran) return bfail(b, LV_ERR_INVALID, "lv_batch_run has not run");
    cudaSetDevice(b->device);
    const size_t G = (size_t)b->G;
    if (G == 0) return LV_OK;
    if (levels)
        LVB_CUDA(b, cudaMemcpyAsync(levels, b->P.levels, sizeof(int32_t) * G, cudaMemcpyDeviceToHost, b->stream));
    if (sweeps)
        LVB_CUDA(b, cudaMemcpyAsync(sweeps, b->P.sweeps, sizeof(int64_t) * G, cudaMemcpyDeviceToHost, b->stream));
    if (edge_sweeps)
        LVB_CUDA(b, cudaMemcpyAsync(edge_sweeps, b->P.edge_sweeps, sizeof(int64_t) * G, cudaMemcpyDeviceToHost,
                                    b->stream));
    std::vector<u64> t0, t1;
    if (latency_ms) {
        t0.resize(G);
        t1.resize(G);
        LVB_CUDA(b, cudaMemcpyAsync(t0.data(), b->P.t_start, sizeof(u64) * G, cudaMemcpyDeviceToHost, b->stream));
        LVB_CUDA(b, cudaMemcpyAsync(t1.data(), b->P.t_end, sizeof(u64) * G, cudaMemcpyDeviceToHost, b->stream));
    }
    LVB_TRY(batch_sync(b));
    if (latency_ms)
        for (size_t g = 0; g < G; ++g) latency_ms[g] = (double)(t1[g] - t0[g]) * 1e-6;
    return LV_OK;
}

int lv_batch_get_stats(lv_batch *b, double *device_ms, int64_t *edge_sweeps, int64_t *vertex_sweeps,
                       int32_t *ctas) {
    if (!b) return LV_ERR_INVALID;
    if (device_ms) *device_ms = b->last_ms;
    if (edge_sweeps) *edge_sweeps = b->last_edge_sweeps;
    if (vertex_sweeps) *vertex_sweeps = b->last_vertex_sweeps;
    if (ctas) {
        *ctas = 0;
        for (const auto &t : b->tiers) *ctas += (t.hi - t.lo) * t.nc;
    }
    return LV_OK;
}

}  // extern "C"
