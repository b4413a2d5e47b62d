// lv_engine.cu -- the engine handle, the level loop and the C ABI.
//
// Host orchestration of one Louvain run on one GPU (replaces main()'s level
// loop, gpulouvain.cu:30-37, optimiseModularity,
// modularity_optimisation.cu:284-363, and aggregateCommunities,
// community_aggregation.cu:248-347).  All state lives in device memory; the
// host waits for one word per sweep (whether another follows; in host-loop mode
// it reads the sweep's modularity parts, move count and error word) and reads a
// few counts per level.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <string>
#include <vector>

#include "../../include/louvain_b200.h"
#include "lv_internal.h"

namespace lv {
void init_agg_attributes();
void agg_prepare(const int32_t *rowptr, const int32_t *rowend, const int32_t *comm,
                 const int32_t *size, int32_t V, AggBuffers &ab, int32_t *mslot, int32_t *degm,
                 int32_t *P, cudaStream_t s);
void agg_classify(const int32_t *size, int32_t V, AggBuffers &ab, const int32_t *P,
                  const int32_t *offsets, cudaStream_t s);
template <typename WT>
void agg_permute(int cls, const GraphView<WT> &g, const AggBuffers &ab, const int32_t *mslot,
                 const int32_t *P, const int32_t *list, int32_t n, int32_t *vkey, u64 *vw, int sms,
                 cudaStream_t s);
void agg_new_vertices(const int32_t *size, const u64 *S, int32_t V, const AggBuffers &ab,
                      const int32_t *P, u64 *knew, cudaStream_t s);
void agg_merge_class(int acls, const AggBuffers &ab, const int32_t *P, const int32_t *list,
                     int32_t n, int32_t *vkey, u64 *vw, uint32_t *vw32, int *err, int *hiflag,
                     int sms, cudaStream_t s, bool narrow);
void agg_merge_global(const HubGlobal &hg, const AggBuffers &ab, const int32_t *P, int32_t *vkey,
                      u64 *vw, uint32_t *vw32, int *err, int *hiflag, cudaStream_t s,
                      bool narrow);
void agg_row_bounds(const AggBuffers &ab, int32_t Vn, int32_t *start, int32_t *end, cudaStream_t s);
void launch_gather_degrees(const int32_t *rowptr, const int32_t *rowend, const int32_t *list,
                           int32_t n, int32_t *out, cudaStream_t s);
void launch_gather_cdeg(const int32_t *mstart, const int32_t *P, const int32_t *list, int32_t n,
                        int32_t *out, cudaStream_t s);
}  // namespace lv

using namespace lv;

// Table sweeps (lv_nct.cuh), see where they are used below; settable so that
// small graphs can be run through them.
#ifndef LV_NCT_MIN_ENTRIES
#define LV_NCT_MIN_ENTRIES (1 << 21)
#endif
#ifndef LV_NCT_SWITCH
#define LV_NCT_SWITCH 0.1
#endif
#ifndef LV_NCT_MAX_SLOTS
#define LV_NCT_MAX_SLOTS 0.3
#endif

namespace {

constexpr int NAC = 5;   // aggregation merge classes (lv_agg.cu)
// cls_scratch layout: class counts, class cursors, then V0 int32 of scratch.
constexpr int SCRATCH_OFF = CLASS_COUNT_WORDS + NCLS + 8;

struct Totals {
    u64 e_own;   // full pass: sum_i e_{i->C(i)}
    u64 s2[2];   // hi, lo of sum_C Sigma_tot^2
    u64 moves;
    u64 dE;      // exact change of e_own over the sweep (wrapping)
    int err;
    int pad;
};

// Counters of one sweep, cleared together with the totals by one memset: the
// sub-rounds' mover counts, and a set of fallback-queue counters (count, next
// per queue, then the warp cursor) for each launch of the wide kernels.
constexpr int FB_SETS = 4;
constexpr int FB_CTR = 2 * (NFBQ + 1) + 2;
struct SweepBlock {
    u64 movers[NBUCKETS];
    int32_t nctq[2][2];   // the table build queue's count, next (buckets 5 and 6)
    int32_t fb[FB_SETS][FB_CTR];
    Totals tot;
};

struct Pending {
    int kind;   // 0..NCLS-1 class, 100 move phase, 101 modularity, 102 aggregate, 103 setup
    cudaEvent_t a, b;
    double bytes;    // algorithmic: 12 per edge + 20 per vertex
    double sbytes;   // as stored: 8 + weight width per edge + 20 per vertex
    int64_t verts, edges;
};

struct HubLayout {
    HubGlobal view;
    void *dev = nullptr;   // packed index arrays
    size_t dev_bytes = 0;
    std::vector<int32_t> ids;
};

}  // namespace

struct lv_handle {
    int device = 0;
    cudaStream_t stream = nullptr;
    lv_opts opts{};
    std::string err;
    DeviceInfo di;

    int32_t V0 = 0;
    int64_t E0 = 0;
    bool owns_input = false;
    int32_t *in_rowptr = nullptr, *in_col = nullptr;
    float *in_w = nullptr;
    int scale = 0;
    double scale_d = 1.0;
    u64 T = 0;
    int exact = 1;
    bool w0_narrow = false;   // level-0 fixed-point weights are all below 2^32
    int32_t giant_degree = HG_MIN_DEG;   // work-mapping knobs (lv_opts.giant_degree, warp_limit)

    int level = 0;
    int32_t V = 0;
    int64_t E = 0;
    // current level: row v = cur_col/cur_w[cur_rowptr[v] .. cur_rowend[v])
    int32_t *cur_rowptr = nullptr, *cur_rowend = nullptr, *cur_col = nullptr;
    u64 *cur_w = nullptr;   // nullptr at level 0 (float input weights)
    // 32-bit copy of cur_w: the move kernels read it, the modularity pass and
    // the aggregation read cur_w.  nullptr when the level holds a sum of 2^32 or
    // more outside the self-loops: it is swept with the 64-bit kernels on the
    // uint64 sums.  Both other ways were slower (move phase of an R-MAT-24 run
    // 241 ms): the 32-bit copy with those rows in the large queue 262 ms (the
    // piece tables' two atomics per add serialise where many lanes add to one
    // community), the 32-bit copy with 64-bit tables and the escaped sums read
    // from the uint64 ones 256 ms (the escape test per entry costs more than the
    // 4 bytes that it saves).
    uint32_t *cur_w32 = nullptr;

    // aggregated levels, ping-pong: rows stay where the merge wrote them
    int32_t *lvl_start[2] = {nullptr, nullptr};
    int32_t *lvl_end[2] = {nullptr, nullptr};
    int32_t *lvl_col[2] = {nullptr, nullptr};
    u64 *lvl_w[2] = {nullptr, nullptr};
    uint32_t *lvl_w32[2] = {nullptr, nullptr};
    int cur_buf = -1;

    int32_t *comm = nullptr, *newc = nullptr, *size = nullptr, *orig2comm = nullptr;
    int32_t *mv_list = nullptr;    // movers of a sub-round (StateView::mv_list)
    uint32_t mv_round = 0;         // sub-rounds launched so far
    u64 *k = nullptr, *S = nullptr;
    int32_t *list = nullptr;
    int32_t *cls_scratch = nullptr;   // class counts, cursors, then V0 entries of scratch
    int32_t *sort_buf = nullptr;      // 3 V0 int32: keys, keys and values of the degree sort
    void *sort_temp = nullptr;
    size_t sort_temp_bytes = 0;
    int32_t cls_off[NCLS + 1] = {0};
    int64_t cls_edges[NCLS] = {0};

    HubLayout hub_move, hub_agg;
    GSlot *tbl_buf = nullptr;
    size_t tbl_slots = 0;
    int32_t *occ_buf = nullptr;    // occupied-slot lists of the global tables
    size_t occ_cap = 0;
    int32_t *nocc_buf = nullptr;   // per-hub list lengths, zero between uses
    size_t nocc_cap = 0;
    int32_t *stage_key = nullptr;  // staging area of the hub path (entries = occ_cap)
    u64 *stage_val = nullptr;
    int32_t *stage2_key = nullptr; // the staged pairs regrouped by key partition (occ_cap)
    u64 *stage2_val = nullptr;
    int32_t *poff_buf = nullptr;   // partition offsets of the regrouped pairs
    size_t poff_cap = 0;
    u64 *eown_buf = nullptr;       // per hub, zero between uses (nocc_cap entries)
    int32_t *ovf_buf = nullptr;    // overflow list (nocc_cap entries) then its count
    bool in_loop = false;          // sweeps of run_sweeps are being launched (timers off)
    MemSet mem;                    // every device buffer of the handle
    void *loop_d = nullptr;        // device state of the sweep loop
    NctView nct;                   // neighbour-community tables (late sweeps)
    u64 nct_alloc = 0;             // slots allocated in the pool
    int64_t table_limit = 0;       // test hook: most slots of the pool (0: the default)
    int64_t table_sweeps = 0, table_slots = 0, table_without = 0;   // lv_get_table_stats
    int32_t table_full = 0, table_stale = 0;

    // level_setup not run yet for the current level: the state arrays are
    // unset (SETUP_ALL) or a team run set them and only the class lists are
    // missing (SETUP_LISTS)
    int setup_due = 0;
    bool singletons = false;   // the level's communities are its vertices
    bool move_ready = false;   // buffers of the move phase allocated
    void *team_arena = nullptr;
    size_t team_bytes = 0;

    bool agg_ready = false;
    AggBuffers ab{};
    int32_t *mslot = nullptr, *degm = nullptr, *P = nullptr;

    FallbackSet fb;

    SweepBlock *blk_d = nullptr;   // sweep counters and totals
    Totals *tot_d = nullptr;       // = &blk_d->tot
    Totals *tot_h = nullptr;
    int32_t *small_h = nullptr;   // pinned scratch for counts
    volatile int32_t *flag_h = nullptr;

    lv_stats st{};
    lv_class_stats cst{};
    long long launch_base = 0;
    // sum_i e_{i->C(i)} of the current state, maintained exactly across sweeps
    u64 e_own_cur = 0;
    bool e_own_valid = false;
    std::vector<cudaEvent_t> ev_free;
    std::vector<Pending> pend;

    // learned active set and move traces
    bool active_ready = false;      // every buffer below allocated
    float *feat = nullptr;          // [2 V0] features recorded by the move kernels
    uint8_t *moved = nullptr;       // [V0] moved in the previous sweep
    int32_t *nmoved = nullptr;      // [V0] row entries whose vertex moved in the previous sweep
    uint8_t *pred = nullptr;        // [V0] proposed by the predictor
    uint8_t *fresh = nullptr;       // [V0] evaluated in an active sweep since the last full sweep
    int32_t *comm_prev = nullptr;   // [V0] communities before the sweep
    int32_t *alist = nullptr;       // [V0] proposed vertices, at their class's offset
    int32_t *acnt = nullptr;        // [NCLS] proposed vertices per class
    u64 *actr = nullptr;            // [4] movers, proposed movers, trace rows
    uint16_t *model = nullptr;      // [LV_ACTIVE_MODEL_SIZE] bf16 parameters
    bool has_model = false;
    float logit_thr = 0.0f;
    float *tr_x = nullptr;          // trace rows: features, vertex, label
    int32_t *tr_v = nullptr;
    uint8_t *tr_y = nullptr;
    int64_t tr_cap = 0, tr_rows = 0;
    uint64_t tr_sweep = 0;
    int64_t act_evaluated = 0, act_full = 0, act_active = 0;
    double act_recall = -1.0;
    int32_t act_fell_back = 0;
};

namespace {

int fail(lv_handle *h, int code, const std::string &msg) {
    if (h) h->err = msg;
    return code;
}

#define LV_CUDA(h, call)                                                                   \
    do {                                                                                   \
        cudaError_t e__ = (call);                                                          \
        if (e__ != cudaSuccess)                                                            \
            return fail((h), e__ == cudaErrorMemoryAllocation ? LV_ERR_NOMEM : LV_ERR_CUDA, \
                        std::string(#call) + ": " + cudaGetErrorString(e__));             \
    } while (0)

#define LV_TRY(expr)            \
    do {                        \
        int rc__ = (expr);      \
        if (rc__) return rc__;  \
    } while (0)

template <typename T>
int dalloc(lv_handle *h, T **p, size_t n) {
    void *q = nullptr;
    const cudaError_t e = h->mem.alloc(&q, n * sizeof(T), h->stream);
    *p = (T *)q;
    if (e != cudaSuccess) return fail(h, LV_ERR_NOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
    return LV_OK;
}

// dalloc of a buffer that a run can do without: false when it cannot be had.
template <typename T>
bool dalloc_optional(lv_handle *h, T **p, size_t n) {
    void *q = nullptr;
    const bool ok = h->mem.alloc(&q, n * sizeof(T), h->stream) == cudaSuccess;
    *p = (T *)q;
    return ok;
}

// Stream-ordered free (after the handle's queued work).
template <typename T>
void dfree(lv_handle *h, T *&p) {
    if (p) h->mem.free((void *)p, h->stream);
    p = nullptr;
}

cudaEvent_t ev_get(lv_handle *h) {
    if (!h->ev_free.empty()) {
        cudaEvent_t e = h->ev_free.back();
        h->ev_free.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

// Begin / end a timed region on the handle's stream.
struct Timer {
    lv_handle *h;
    int kind;
    cudaEvent_t a = nullptr;
    double bytes = 0, sbytes = 0;
    int64_t verts = 0, edges = 0;
    Timer(lv_handle *hh, int k) : h(hh), kind(k) {
        if (h->in_loop) return;   // the sweep loop is one timed region
        a = ev_get(h);
        cudaEventRecord(a, h->stream);
    }
    void stop() {
        if (!a) return;
        cudaEvent_t b = ev_get(h);
        cudaEventRecord(b, h->stream);
        h->pend.push_back(Pending{kind, a, b, bytes, sbytes, verts, edges});
    }
};

void resolve_events(lv_handle *h) {
    for (const Pending &p : h->pend) {
        float ms = 0;
        cudaEventElapsedTime(&ms, p.a, p.b);
        if (p.kind < NCLS) {
            h->cst.launches[p.kind] += 1;
            h->cst.ms[p.kind] += ms;
            h->cst.bytes[p.kind] += p.bytes;
            h->cst.stored_bytes[p.kind] += p.sbytes;
            h->cst.vertices[p.kind] += p.verts;
            h->cst.edges[p.kind] += p.edges;
        } else if (p.kind == 100) {
            h->st.move_ms += ms;
        } else if (p.kind == 101) {
            h->st.modularity_ms += ms;
        } else if (p.kind == 102) {
            h->st.aggregate_ms += ms;
        } else if (p.kind == 103) {
            h->st.setup_ms += ms;
        }
        h->ev_free.push_back(p.a);
        h->ev_free.push_back(p.b);
    }
    h->pend.clear();
}

int sync(lv_handle *h) {
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return fail(h, LV_ERR_CUDA, std::string("stream: ") + cudaGetErrorString(e));
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(h, LV_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    resolve_events(h);
    return LV_OK;
}

int check_device_error(lv_handle *h, int errword) {
    if (errword == 0) return LV_OK;
    std::string m = "device check failed:";
    if (errword & DEVERR_HASH_FULL) m += " hash table full";
    if (errword & DEVERR_BAD_STATE) m += " invalid community id";
    if (errword & DEVERR_FALLBACK_FULL) m += " fallback list full";
    return fail(h, LV_ERR_DEVICE, m);
}

template <typename WT>
GraphView<WT> view_of(lv_handle *h);
template <>
GraphView<float> view_of<float>(lv_handle *h) {
    return GraphView<float>{h->cur_rowptr, h->cur_rowend, h->cur_col, h->in_w, h->scale_d, nullptr, h->E0};
}
template <>
GraphView<u64> view_of<u64>(lv_handle *h) {
    return GraphView<u64>{h->cur_rowptr, h->cur_rowend, h->cur_col, h->cur_w, h->scale_d, nullptr, h->E0};
}
template <>
GraphView<uint32_t> view_of<uint32_t>(lv_handle *h) {
    return GraphView<uint32_t>{h->cur_rowptr, h->cur_rowend, h->cur_col, h->cur_w32, h->scale_d, h->cur_w,
                               h->E0};
}

// Calls F<WT>(args...) with the weight type the move phase reads at the
// current level: float32 input at level 0, the 32-bit copy of the sums when
// every sum other than the self-loops is below 2^32 (the move kernels skip
// self-loops), the uint64 sums otherwise.
#define LV_BY_WEIGHT(h, F, ...)                                  \
    do {                                                         \
        if ((h)->cur_w32) F<uint32_t>(__VA_ARGS__);              \
        else if ((h)->cur_w) F<u64>(__VA_ARGS__);                \
        else F<float>(__VA_ARGS__);                              \
    } while (0)

// Every weight the move phase reads is below 2^32: the 32-bit view of an
// aggregated level, or level 0 when its fixed-point weights fit 32 bits
// (the move kernels then keep their table sums in 16-bit-piece counters).
// opts.wide_weights keeps 64-bit sums everywhere.
template <typename WT>
bool narrow_weights(const lv_handle *h) {
    if (h->opts.wide_weights) return false;
    if (std::is_same<WT, uint32_t>::value) return true;
    if (std::is_same<WT, float>::value) return h->w0_narrow;
    return false;
}

StateView state_of(lv_handle *h) {
    return StateView{h->comm, h->newc, h->size, h->k, h->S, h->T, &h->tot_d->err, h->feat,
                     h->blk_d->movers, h->mv_list, h->V0, 0, nullptr, nullptr,
                     (LV_DEDUP == 2 || (LV_DEDUP == 1 && h->level > 0)) ? 1 : 0};
}

// Numbers a sub-round.  When the numbers run out, the old ones are forgotten.
void next_round(lv_handle *h, StateView &st) {
    if (++h->mv_round == 0) {
        cudaMemsetAsync(h->mv_list + 3 * (size_t)h->V0, 0, sizeof(int32_t) * (size_t)h->V0, h->stream);
        h->mv_round = 1;
    }
    st.mv_round = h->mv_round;
}

// ---------------------------------------------------------------------------
// global hash-table layouts (hub vertices in the move phase, very large
// communities in aggregation)
// ---------------------------------------------------------------------------
// Pinned host scratch (the totals block and the class counts a handle reads
// back) comes from a process-wide free list: page-locking memory is a slow
// driver call, and a handle created per run should not pay it.
struct PinnedBlock {
    Totals tot;
    int32_t small[128];
    volatile int32_t flag[2];   // written by sweep_end_kernel: go on, sweep number
};
std::mutex g_pinned_mu;
std::vector<PinnedBlock *> g_pinned_free;

int pinned_take(lv_handle *h) {
    PinnedBlock *b = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        if (!g_pinned_free.empty()) {
            b = g_pinned_free.back();
            g_pinned_free.pop_back();
        }
    }
    if (!b) LV_CUDA(h, cudaMallocHost((void **)&b, sizeof(PinnedBlock)));
    h->tot_h = &b->tot;
    h->small_h = b->small;
    h->flag_h = b->flag;
    return LV_OK;
}

void pinned_give(lv_handle *h) {
    if (!h->tot_h) return;
    PinnedBlock *b = reinterpret_cast<PinnedBlock *>(h->tot_h);
    std::lock_guard<std::mutex> lock(g_pinned_mu);
    g_pinned_free.push_back(b);
    h->tot_h = nullptr;
    h->small_h = nullptr;
}

int ensure_tables(lv_handle *h, size_t slots) {
    if (slots <= h->tbl_slots) return LV_OK;
    size_t want = slots + slots / 4;
    dfree(h, h->tbl_buf);
    h->tbl_slots = 0;
    LV_TRY(dalloc(h, &h->tbl_buf, want));
    LV_CUDA(h, cudaMemsetAsync(h->tbl_buf, 0, want * sizeof(GSlot), h->stream));
    h->tbl_slots = want;
    return LV_OK;
}

// The staging buffers for n entries of giants.
constexpr size_t STAGING_BYTES = 28;   // per entry
int alloc_staging(lv_handle *h, size_t n) {
    dfree(h, h->occ_buf);
    dfree(h, h->stage_key);
    dfree(h, h->stage_val);
    dfree(h, h->stage2_key);
    dfree(h, h->stage2_val);
    h->occ_cap = 0;
    LV_TRY(dalloc(h, &h->occ_buf, n));
    LV_TRY(dalloc(h, &h->stage_key, n));
    LV_TRY(dalloc(h, &h->stage_val, n));
    LV_TRY(dalloc(h, &h->stage2_key, n));
    LV_TRY(dalloc(h, &h->stage2_val, n));
    h->occ_cap = n;
    return LV_OK;
}

int ensure_occ(lv_handle *h, size_t entries, size_t hubs) {
    if (entries > h->occ_cap) {
        // never more entries than the level 0 has.  A run that outgrows its
        // first buffers mostly goes on to about that many, so it takes them at
        // once where that is a small part of the device's memory: fewer
        // outgrown buffers for the next run to ask for again
        const size_t all = (size_t)h->E0, want = std::max(entries, std::min(entries + entries / 4 + 1, all));
        const size_t more = std::min(4 * entries, all);
        const bool grown = h->occ_cap > 0 && more > want && more * STAGING_BYTES <= mem_total(h->device) / 8 &&
                           alloc_staging(h, more) == LV_OK;
        if (!grown) LV_TRY(alloc_staging(h, want));
    }
    if (hubs > h->nocc_cap) {
        dfree(h, h->nocc_buf);
        dfree(h, h->eown_buf);
        dfree(h, h->ovf_buf);
        h->nocc_cap = 0;
        size_t want = hubs + hubs / 4 + 1;
        LV_TRY(dalloc(h, &h->nocc_buf, want));
        LV_TRY(dalloc(h, &h->eown_buf, want));
        LV_TRY(dalloc(h, &h->ovf_buf, want + 1));   // overflow list + its count
        LV_CUDA(h, cudaMemsetAsync(h->nocc_buf, 0, want * sizeof(int32_t), h->stream));
        LV_CUDA(h, cudaMemsetAsync(h->eown_buf, 0, want * sizeof(u64), h->stream));
        LV_CUDA(h, cudaMemsetAsync(h->ovf_buf, 0, (want + 1) * sizeof(int32_t), h->stream));
        h->nocc_cap = want;
    }
    return LV_OK;
}

// ids: hub vertices / communities; deg: their degree bound; cap_limit caps
// the distinct-key count (newV for aggregation, unlimited for moves).
int build_layout(lv_handle *h, HubLayout &L, const std::vector<int32_t> &ids,
                 const std::vector<int32_t> &deg, int64_t cap_limit, bool occ_lists, int echunk,
                 bool tables) {
    const int32_t n = (int32_t)ids.size();
    std::vector<int64_t> off(n), occ_off(n);
    int64_t occ_total = 0;
    std::vector<int32_t> lg(n), ech_hub, ech_e0, sch_hub, sch_s0, hub_s0(n + 1), hub_cap(n), pbase(n + 1, 0);
    int64_t total = 0;
    for (int32_t i = 0; i < n; ++i) {
        int64_t distinct = deg[i];
        if (cap_limit > 0 && distinct > cap_limit) distinct = cap_limit;
        int l = ceil_log2_i(2 * distinct);
        if (l < 3) l = 3;
        lg[i] = l;
        off[i] = total;
        total += int64_t(1) << l;
        for (int32_t e0 = 0; e0 < deg[i]; e0 += echunk) {
            ech_hub.push_back(i);
            ech_e0.push_back(e0);
        }
        // evaluation chunks: over the occupied list (room for deg entries)
        // when occ_lists is set, else over the contiguous table
        hub_s0[i] = (int32_t)sch_hub.size();
        occ_off[i] = occ_total;
        occ_total += deg[i];
        hub_cap[i] = deg[i];
        pbase[i + 1] = pbase[i] + (deg[i] + FB_KEYS - 1) / FB_KEYS + 2;
        const int64_t span = occ_lists ? (int64_t)deg[i] : (int64_t(1) << l);
        for (int64_t s0 = 0; s0 < span; s0 += HG_SLOT_CHUNK) {
            sch_hub.push_back(i);
            sch_s0.push_back((int32_t)s0);
        }
        if (span == 0) {
            sch_hub.push_back(i);
            sch_s0.push_back(0);
        }
    }
    hub_s0[n] = (int32_t)sch_hub.size();
    if (tables) LV_TRY(ensure_tables(h, (size_t)total));
    LV_TRY(ensure_occ(h, (size_t)occ_total, (size_t)n));
    const size_t ne = ech_hub.size(), ns = sch_hub.size();
    // packed: ids | lg | ech_hub | ech_e0 | sch_hub | sch_s0 | hub_s0 | res_c | (8-aligned) off |
    // res_g | res_e | res_b | occ_off
    size_t i32_count = (size_t)n + n + ne + ne + ns + ns + (n + 1) + ns + n + (n + 1);
    size_t i32_bytes = ((i32_count * 4 + 15) / 16) * 16;
    size_t bytes = i32_bytes + (size_t)n * 8 + ns * 16 + ns * 8 + ns * 8 + (size_t)n * 8 + 64;
    if (bytes > L.dev_bytes) {
        unsigned char *old_dev = (unsigned char *)L.dev;
        dfree(h, old_dev);
        L.dev = nullptr;
        L.dev_bytes = 0;
        unsigned char *nd = nullptr;
        LV_TRY(dalloc(h, &nd, bytes));
        L.dev = nd;
        L.dev_bytes = bytes;
    }
    std::vector<unsigned char> host(bytes, 0);
    int32_t *p32 = (int32_t *)host.data();
    size_t at = 0;
    auto put = [&](const int32_t *src, size_t cnt) {
        size_t start = at;
        if (cnt) std::memcpy(p32 + at, src, cnt * 4);
        at += cnt;
        return start;
    };
    size_t o_ids = put(ids.data(), n), o_lg = put(lg.data(), n);
    size_t o_eh = put(ech_hub.data(), ne), o_e0 = put(ech_e0.data(), ne);
    size_t o_sh = put(sch_hub.data(), ns), o_s0 = put(sch_s0.data(), ns);
    size_t o_hs = put(hub_s0.data(), n + 1);
    size_t o_rc = at;
    at += ns;
    size_t o_cap = put(hub_cap.data(), n), o_pb = put(pbase.data(), n + 1);
    unsigned char *base8 = host.data() + i32_bytes;
    if (n) std::memcpy(base8, off.data(), (size_t)n * 8);
    if (n) std::memcpy(base8 + (size_t)n * 8 + ns * 32, occ_off.data(), (size_t)n * 8);
    LV_CUDA(h, cudaMemcpyAsync(L.dev, host.data(), bytes, cudaMemcpyHostToDevice, h->stream));
    // the host vector must outlive the async copy
    LV_CUDA(h, cudaStreamSynchronize(h->stream));
    int32_t *d32 = (int32_t *)L.dev;
    unsigned char *d8 = (unsigned char *)L.dev + i32_bytes;
    HubGlobal &v = L.view;
    v.nhubs = n;
    v.n_echunks = (int32_t)ne;
    v.n_schunks = (int32_t)ns;
    v.hubs = d32 + o_ids;
    v.tbl_lg = d32 + o_lg;
    v.echunk_hub = d32 + o_eh;
    v.echunk_e0 = d32 + o_e0;
    v.schunk_hub = d32 + o_sh;
    v.schunk_s0 = d32 + o_s0;
    v.hub_schunk0 = d32 + o_hs;
    v.res_c = d32 + o_rc;
    v.hub_cap = d32 + o_cap;
    v.pbase = d32 + o_pb;
    v.tbl_off = (const int64_t *)d8;
    v.res_g = (u64 *)(d8 + (size_t)n * 8);
    v.res_e = (u64 *)(d8 + (size_t)n * 8 + ns * 16);
    v.res_b = (u64 *)(d8 + (size_t)n * 8 + ns * 24);
    v.occ_off = (const int64_t *)(d8 + (size_t)n * 8 + ns * 32);
    v.occ = h->occ_buf;
    v.nocc = h->nocc_buf;
    v.stage_key = h->stage_key;
    v.stage_val = h->stage_val;
    v.stage2_key = h->stage2_key;
    v.stage2_val = h->stage2_val;
    if ((size_t)pbase[n] > h->poff_cap) {
        dfree(h, h->poff_buf);
        h->poff_cap = 0;
        LV_TRY(dalloc(h, &h->poff_buf, (size_t)pbase[n] + 1));
        h->poff_cap = (size_t)pbase[n];
    }
    v.poff = h->poff_buf;
    v.eown = h->eown_buf;
    v.ovf_list = h->ovf_buf;
    v.ovf_count = h->ovf_buf + h->nocc_cap;
    v.slots = h->tbl_buf;
    L.ids = ids;
    return LV_OK;
}

// ---------------------------------------------------------------------------
// level set-up: degree classes, k_i (level 0), singleton state, hub layout
// ---------------------------------------------------------------------------
template <typename WT>
int compute_k(lv_handle *h) {
    GraphView<WT> g = view_of<WT>(h);
    LV_CUDA(h, cudaMemsetAsync(h->k, 0, sizeof(u64) * (size_t)h->V, h->stream));
    for (int c = 0; c < NCLS; ++c)
        launch_row_reduce<WT>(c, 0, g, h->comm, h->k, nullptr, h->list + h->cls_off[c],
                              h->cls_off[c + 1] - h->cls_off[c], h->di, h->stream);
    return LV_OK;
}

enum { SETUP_ALL = 1, SETUP_LISTS = 2 };
bool team_fits(const lv_handle *h);

int ensure_move(lv_handle *h);

int level_setup(lv_handle *h, bool lists_only = false) {
    LV_TRY(ensure_move(h));
    Timer t(h, 103);
    int32_t *counts = h->cls_scratch, *cursors = h->cls_scratch + CLASS_COUNT_WORDS;
    launch_class_count(h->cur_rowptr, h->cur_rowend, h->V, h->giant_degree, counts, h->stream);
    LV_CUDA(h, cudaMemcpyAsync(h->small_h, counts, sizeof(int32_t) * CLASS_COUNT_WORDS,
                               cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    h->cls_off[0] = 0;
    const u64 *esum = reinterpret_cast<const u64 *>(h->small_h + NCLS + (NCLS & 1));
    for (int c = 0; c < NCLS; ++c) {
        h->cls_off[c + 1] = h->cls_off[c] + h->small_h[c];
        h->cls_edges[c] = (int64_t)esum[c];
    }
    launch_class_scatter(h->cur_rowptr, h->cur_rowend, h->V, h->giant_degree, h->fb.warp_limit, h->cls_off,
                         cursors, h->list, h->fb.hint,
                         h->stream);
    // the warp kernels' vertices by decreasing degree within each update
    // bucket (bucket 6's warp part spans classes H1 and H2)
    {
        const int32_t V0 = h->V0;
        int32_t *kb = h->sort_buf, *ka = h->sort_buf + V0, *va = h->sort_buf + 2 * (size_t)V0;
        const int32_t seg[3][3] = {{CLS_B4, CLS_B5, 84}, {CLS_B5, CLS_H1, 319}, {CLS_H1, CLS_HG, h->giant_degree}};
        for (const auto &sg : seg) {
            const int32_t lo = h->cls_off[sg[0]], n = h->cls_off[sg[1]] - lo;
            sort_by_degree_desc(h->cur_rowptr, h->cur_rowend, h->list + lo, n, sg[2], kb, ka, va, h->sort_temp,
                                h->sort_temp_bytes, h->stream);
        }
    }
    if (!lists_only) {
        if (h->level == 0) LV_TRY(compute_k<float>(h));
        launch_level_init(h->comm, h->newc, h->size, h->k, h->S, h->V, h->stream);
        h->singletons = true;
    }
    // giants (degree > giant_degree): staging areas and global tables
    const int32_t nh = h->cls_off[CLS_HG + 1] - h->cls_off[CLS_HG];
    std::vector<int32_t> ids(nh), deg(nh);
    if (nh > 0) {
        int32_t *dd = h->cls_scratch + SCRATCH_OFF;   // room reserved at create: V0 entries
        launch_gather_degrees(h->cur_rowptr, h->cur_rowend, h->list + h->cls_off[CLS_HG], nh, dd,
                              h->stream);
        LV_CUDA(h, cudaMemcpyAsync(ids.data(), h->list + h->cls_off[CLS_HG], sizeof(int32_t) * nh,
                                   cudaMemcpyDeviceToHost, h->stream));
        LV_CUDA(h, cudaMemcpyAsync(deg.data(), dd, sizeof(int32_t) * nh, cudaMemcpyDeviceToHost,
                                   h->stream));
        LV_TRY(sync(h));
    }
    LV_TRY(build_layout(h, h->hub_move, ids, deg, 0, false, STAGE_CHUNK, false));
    t.stop();
    if (h->opts.trace) {
        std::fprintf(stderr, "[lv] level %d: V=%d E=%lld classes:", h->level, h->V, (long long)h->E);
        for (int c = 0; c < NCLS; ++c)
            std::fprintf(stderr, " %d/%lld", h->cls_off[c + 1] - h->cls_off[c], (long long)h->cls_edges[c]);
        std::fprintf(stderr, "\n");
    }
    return LV_OK;
}

// Runs the level set-up that was left out so far (every entry point that
// reads the level's state or lists calls this first).
int ensure_setup(lv_handle *h) {
    const int due = h->setup_due;
    if (!due) return LV_OK;
    h->setup_due = 0;
    const int rc = level_setup(h, due == SETUP_LISTS);
    if (rc) h->setup_due = due;
    return rc;
}

// ---------------------------------------------------------------------------
// sweep and modularity
// ---------------------------------------------------------------------------
// Profile slots of the move phase: 0..3 the group kernels of buckets 0..3,
// 4, 5, 6 the warp + fallback kernels of buckets 4, 5 and 6.
// The fallback queues on counter set i of the sweep.
FallbackSet queues_on(const lv_handle *h, int i) {
    FallbackSet fs = h->fb;
    int32_t *c = h->blk_d->fb[i];
    for (int q = 0; q <= NFBQ; ++q) {
        fs.q[q].count = c + 2 * q;
        fs.q[q].next = fs.q[q].count + 1;
    }
    fs.warp_next = c + 2 * (NFBQ + 1);
    return fs;
}

template <typename WT>
void enqueue_sweep(lv_handle *h) {
    GraphView<WT> g = view_of<WT>(h);
    StateView st = state_of(h);
    const double wbytes = sizeof(WT) == 4 ? 4.0 : 8.0;
    u64 *dE = &h->tot_d->dE;
    Timer tm(h, 100);
    int64_t sweep_verts = 0;
    for (int b = 0; b < NBUCKETS; ++b) {
        const int c0 = b, c1 = (b < 6) ? b + 1 : NCLS;
        const int32_t lo = h->cls_off[c0], hi = h->cls_off[c1];
        if (hi == lo) continue;
        const int32_t hg0 = (b == 6) ? h->cls_off[CLS_HG] : hi;   // bucket 6: giants after
        const FallbackSet fs = queues_on(h, b >= 4 ? b - 4 : 3);
        st.mv_cnt = h->blk_d->movers + b;
        next_round(h, st);
        int64_t edges = 0;
        for (int c = c0; c < c1; ++c)
            if (c != CLS_HG) edges += h->cls_edges[c];
        Timer *tc = nullptr;
        if (h->opts.profile) {
            tc = new Timer(h, b);
            tc->verts = hg0 - lo;
            tc->edges = edges;
            tc->bytes = 12.0 * (double)edges + 20.0 * (double)(hg0 - lo);
            tc->sbytes = (8.0 + wbytes) * (double)edges + 20.0 * (double)(hg0 - lo);
        }
        if (b < 4)
            launch_move_class<WT>(b, g, st, h->list + lo, hi - lo, dE, h->stream, narrow_weights<WT>(h));
        else if (hg0 > lo)
            launch_move_wide<WT>(g, st, h->list + lo, hg0 - lo, fs, h->di, dE, h->stream,
                                 b == 6 ? h->giant_degree : (b == 4 ? 84 : 319), narrow_weights<WT>(h),
                                 hi > hg0);
        if (tc) {
            tc->stop();
            delete tc;
            tc = nullptr;
        }
        if (hi > hg0) {
            if (h->opts.profile) {
                tc = new Timer(h, 7);
                tc->verts = hi - hg0;
                tc->edges = h->cls_edges[CLS_HG];
                tc->bytes = 12.0 * (double)tc->edges + 20.0 * (double)tc->verts;
                tc->sbytes = (8.0 + wbytes) * (double)tc->edges + 20.0 * (double)tc->verts;
            }
            launch_move_giants<WT>(g, st, h->hub_move.view, fs, h->di, dE, h->stream, narrow_weights<WT>(h));
            if (tc) {
                tc->stop();
                delete tc;
            }
        }
        if (b >= 4) launch_collect_movers<WT>(g, st, h->list + lo, hi - lo, h->stream);
        launch_movers<WT>(g, st, hi - lo, h->di, dE, &h->tot_d->moves, h->stream);
        sweep_verts += hi - lo;
    }
    tm.bytes = 12.0 * (double)h->E + 20.0 * (double)sweep_verts;
    tm.sbytes = (8.0 + wbytes) * (double)h->E + 20.0 * (double)sweep_verts;
    tm.stop();
    h->st.move_bytes += tm.bytes;
}

// A sweep whose vertices of degree > 32 are decided from their tables.
template <typename WT>
void enqueue_sweep_tables(lv_handle *h) {
    GraphView<WT> g = view_of<WT>(h);
    StateView st = state_of(h);
    st.tlg = h->nct.lg;
    st.tnever = h->nct.cursor + 1;
    u64 *dE = &h->tot_d->dE;
    for (int b = 0; b < NBUCKETS; ++b) {
        const int32_t lo = h->cls_off[b], hi = b < 6 ? h->cls_off[b + 1] : h->cls_off[NCLS];
        if (hi == lo) continue;
        const FallbackSet fs = queues_on(h, b >= 4 ? b - 4 : 3);
        st.mv_cnt = h->blk_d->movers + b;
        next_round(h, st);
        if (b < 4) {
            launch_move_class<WT>(b, g, st, h->list + lo, hi - lo, dE, h->stream, narrow_weights<WT>(h));
        } else {
            // rows of bucket 4 never hold more communities than a warp builds
            NctView t = h->nct;
            t.qctr = h->blk_d->nctq[b == 6];
            launch_nct<WT>(g, st, h->list + lo, hi - lo, t, fs, h->giant_degree, b > 4, h->di, dE, h->stream);
            if (b == 6) {
                if (hi > h->cls_off[CLS_HG])
                    launch_move_giants<WT>(g, st, h->hub_move.view, fs, h->di, dE, h->stream, narrow_weights<WT>(h));
                else
                    launch_large<WT>(g, st, fs, h->di, dE, h->stream);
            }
            launch_collect_movers<WT>(g, st, h->list + lo, hi - lo, h->stream);
        }
        launch_movers<WT>(g, st, hi - lo, h->di, dE, &h->tot_d->moves, h->stream, &h->nct);
    }
}

template <typename WT>
void enqueue_modularity(lv_handle *h) {
    GraphView<WT> g = view_of<WT>(h);
    Timer tm(h, 101);
    for (int c = 0; c < NCLS; ++c)
        launch_row_reduce<WT>(c, 1, g, h->comm, nullptr, &h->tot_d->e_own, h->list + h->cls_off[c],
                              h->cls_off[c + 1] - h->cls_off[c], h->di, h->stream);
    launch_s2(h->S, h->V, h->tot_d->s2, h->stream);
    tm.stop();
}

double q_from_totals(u64 T, const Totals &t) {
    // Same FP64 formula as the oracle: e_own/T - sum(S^2)/T^2, i.e.
    // toOwn/(2M) - sum(S^2)/(4M^2) of calculateModularity.
    const u128 s2 = ((u128)t.s2[0] << 64) | (u128)t.s2[1];
    const double td = (double)T;
    const double a = (double)t.e_own / td;
    const double b = (double)s2 / (td * td);
    return a - b;
}

// Clears the sweep counters and the totals, keeping the device error word.
int reset_totals(lv_handle *h) {
    LV_CUDA(h, cudaMemsetAsync(h->blk_d, 0, offsetof(SweepBlock, tot) + offsetof(Totals, err), h->stream));
    return LV_OK;
}

int read_totals(lv_handle *h) {
    LV_CUDA(h, cudaMemcpyAsync(h->tot_h, h->tot_d, sizeof(Totals), cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    return check_device_error(h, h->tot_h->err);
}

int modularity(lv_handle *h, double *q) {
    LV_TRY(reset_totals(h));
    if (h->cur_w) enqueue_modularity<u64>(h); else enqueue_modularity<float>(h);
    LV_TRY(read_totals(h));
    h->e_own_cur = h->tot_h->e_own;
    h->e_own_valid = true;
    *q = q_from_totals(h->T, *h->tot_h);
    return LV_OK;
}

// One sweep followed by the modularity of the resulting state.  The edge
// pass of calculateModularity is replaced by the exact update of
// sum_i e_{i->C(i)} accumulated by the move and mover kernels; only the
// sum of Sigma_tot^2 is recomputed (a pass over V).
int sweep_and_q(lv_handle *h, int64_t *moves, double *q) {
    h->singletons = false;
    if (!h->e_own_valid) {
        double q0;
        LV_TRY(modularity(h, &q0));
    }
    LV_TRY(reset_totals(h));
    clear_move_state(h->fb, h->hub_move.view, h->stream);
    LV_BY_WEIGHT(h, enqueue_sweep, h);
    {
        Timer tm(h, 101);
        launch_s2(h->S, h->V, h->tot_d->s2, h->stream);
        tm.stop();
    }
    LV_TRY(read_totals(h));
    h->e_own_cur += h->tot_h->dE;
    Totals t = *h->tot_h;
    t.e_own = h->e_own_cur;
    *moves = (int64_t)t.moves;
    const double q_inc = q_from_totals(h->T, t);
    if (h->opts.verify) {
        double q_full = 0;
        LV_TRY(modularity(h, &q_full));
        if (h->e_own_cur != t.e_own || q_full != q_inc)
            return fail(h, LV_ERR_DEVICE, "incremental modularity differs from the full pass");
    }
    if (q) *q = q_inc;
    if (h->opts.trace) {
        // per-class device time of this sweep (profile mode) and move phase
        std::fprintf(stderr, "[lv]   sweep: moves=%lld q=%.9f move_ms_total=%.3f", (long long)t.moves,
                     q_inc, h->st.move_ms);
        if (h->opts.profile) {
            std::fprintf(stderr, " class_ms_total:");
            for (int c = 0; c < NCLS; ++c) std::fprintf(stderr, " %.2f", h->cst.ms[c]);
        }
        std::fprintf(stderr, "\n");
    }
    h->st.sweeps += 1;
    h->st.edge_sweeps += h->E;
    h->st.moves += *moves;
    return LV_OK;
}

// ---------------------------------------------------------------------------
// device-side sweep control
// ---------------------------------------------------------------------------
// A level's sweeps (totals reset, the seven sub-rounds with corrections and
// commits, the sum of Sigma_tot^2) end with sweep_end_kernel, which updates
// sum_i e_{i->C(i)} by the sweep's exact change, forms Q with the host's FP64
// operations (each correctly rounded, so the value is the same bit for bit),
// decides exactly as the host loop does whether another sweep follows (the
// sweep gained at least min_gain, moved something, the sweep cap is not
// reached and no device check failed) and writes that to pinned memory, where
// the host, having launched the sweep's kernels ahead, waits for it.  The
// same loop as one CUDA graph with a while node saved about 20 us per sweep
// but took 0.3 ms to build, 0.15 ms to launch and 0.3 ms to destroy per level:
// planted graph of 10,007 vertices 1.67 ms against 1.53, R-MAT-16 level by
// level 6.6 against 6.3, R-MAT-20 28.6 against 28.4.  Launching the next sweep
// before the outcome is known (with a stop word that its kernels test) was
// slower still (LFR graph of 300,007 vertices 6.46 ms against 6.22 in lv_run).
struct LoopState {
    double q_before;
    double min_gain;
    u64 e_own;          // sum_i e_{i->C(i)} of the current state
    u64 T;
    u64 moves_total;
    double q_last;
    u64 switch_units;   // leave the loop for table sweeps when a sweep's movers have fewer row units
    int32_t max_sweeps;
    int32_t sweeps;
    int32_t changed;
    int32_t switched;
};

__global__ void sweep_end_kernel(const SweepBlock *blk, LoopState *ls, volatile int32_t *flag, int32_t number) {
    const Totals *t = &blk->tot;
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x != 0) return;
    ls->e_own += t->dE;
    const double q = q_from_parts_dev(ls->T, ls->e_own, t->s2[0], t->s2[1]);
    ls->sweeps += 1;
    ls->moves_total += t->moves;
    const double gain = __dsub_rn(q, ls->q_before);
    if (gain > 0) ls->changed = 1;
    ls->q_before = q;
    ls->q_last = q;
    bool more = gain >= ls->min_gain && t->moves != 0 &&
                !(ls->max_sweeps > 0 && ls->sweeps >= ls->max_sweeps) && t->err == 0;
    if (more && ls->switch_units) {
        u64 units = 0;
        for (int b = 0; b < NBUCKETS; ++b) units += blk->movers[b] >> 32;
        if (units < ls->switch_units) {
            ls->switched = 1;
            more = false;
        }
    }
    flag[0] = more ? 1 : 0;
    __threadfence_system();
    flag[1] = number;
}

// Tables pay off on levels whose sweeps are bound by their rows: below this many
// entries the tables save less than their checks and builds cost.  Runs without
// tables / from 2^21 / from 2^18 entries, ms: R-MAT scale 16 (1.8 million
// entries) 8.59 / 8.58 / 8.80, 17 (with edge factor 16, 3.7 million) 15.54 / 13.45
// / 13.46, 18 (7.6 million) 16.55 / 14.45 / 14.35, planted graph of 3000 vertices and
// 0.8 million entries 0.56 / 0.56 / 0.62.  Where one sweep is left after the switch
// they cost a little (20,000 vertices, 5.6 million entries 1.14 / 1.35), and the
// checks alone up to 2 % (LFR graph of 300,007 vertices 4.89 / 5.01).
constexpr int64_t NCT_MIN_ENTRIES = LV_NCT_MIN_ENTRIES;
// ... once the movers' rows, which the table updates visit with random
// accesses, are a small part of the entries: lv_run of R-MAT-24 takes 240 / 236
// / 233.4 / 233.4 ms when tables start below 0.02 / 0.05 / 0.1 / 0.2 (273 ms
// without tables) ...
constexpr double NCT_SWITCH = LV_NCT_SWITCH;
// ... and when the tables hold far fewer slots than the rows hold entries
// (R-MAT-24: 0.12 slots per entry on the second level; over 0.5 on the first,
// where a table sweep took 51 ms against 18), estimated from sampled rows.
constexpr double NCT_MAX_SLOTS = LV_NCT_MAX_SLOTS;
constexpr int32_t NCT_SAMPLES = 4096;

// Prepares table sweeps of the current level; *ok = 0 when its rows do not
// allow them (an entry without its mirror entry, or of weight zero) or there is
// no memory for the tables.
int nct_begin(lv_handle *h, int *ok) {
    *ok = 0;
    LV_TRY(reset_totals(h));
    u64 *tot = h->tot_d->s2;   // two words
    launch_nct_sample(h->cur_rowptr, h->cur_rowend, h->cur_col, h->comm, h->list + h->cls_off[CLS_B4],
                      h->cls_off[CLS_HG] - h->cls_off[CLS_B4], NCT_SAMPLES, tot, h->stream);
    LV_TRY(read_totals(h));
    if ((double)h->tot_h->s2[0] > NCT_MAX_SLOTS * (double)h->tot_h->s2[1]) return LV_OK;
    LV_TRY(reset_totals(h));
    auto check = [&](auto g) {
        for (int c = 0; c < NCLS; ++c)
            launch_row_reduce(c, 2, g, h->comm, nullptr, tot, h->list + h->cls_off[c],
                              h->cls_off[c + 1] - h->cls_off[c], h->di, h->stream);
    };
    if (h->cur_w) check(view_of<u64>(h));
    else check(view_of<float>(h));
    LV_TRY(read_totals(h));
    if (h->tot_h->s2[0] || h->tot_h->s2[1]) return LV_OK;
    // without memory for tables the sweeps go on from the rows
    NctView &t = h->nct;
    const size_t V = (size_t)h->V0 + 1;
    if ((!t.lg && !dalloc_optional(h, &t.lg, V)) || (!t.off && !dalloc_optional(h, &t.off, V)) ||
        (!t.queue && !dalloc_optional(h, &t.queue, V)) || (!t.cursor && !dalloc_optional(h, &t.cursor, 4)))
        return LV_OK;
    // half a slot per entry of the level: rows with many communities that do
    // not fit go on being summed from the row
    u64 want = (u64)h->E / 2 + 1024;
    if (h->table_limit > 0 && want > (u64)h->table_limit) want = (u64)h->table_limit;
    if (want > h->nct_alloc) {
        dfree(h, t.slots);
        h->nct_alloc = 0;
        if (!dalloc_optional(h, &t.slots, (size_t)want)) return LV_OK;
        h->nct_alloc = want;
    }
    h->nct.cap = want;
    LV_CUDA(h, cudaMemsetAsync(h->nct.lg, 0, (size_t)h->V, h->stream));
    LV_CUDA(h, cudaMemsetAsync(h->nct.cursor, 0, 4 * sizeof(u64), h->stream));
    *ok = 1;
    return LV_OK;
}

// Runs sweeps (from tables when `tables`) from the state *ls until one ends the
// loop; *ls is read back.
int run_sweeps(lv_handle *h, bool tables, LoopState *ls) {
    LoopState *ld = (LoopState *)h->loop_d;
    const int32_t sweeps0 = ls->sweeps;
    const u64 moves0 = ls->moves_total;
    LV_CUDA(h, cudaMemcpyAsync(ld, ls, sizeof(*ls), cudaMemcpyHostToDevice, h->stream));
    clear_move_state(h->fb, h->hub_move.view, h->stream);
    h->flag_h[0] = 0;
    h->flag_h[1] = 0;
    Timer tm(h, 100);
    h->in_loop = true;   // one timed region for the loop, none per sweep
    int rc = LV_OK;
    for (int32_t number = 1;; ++number) {
        rc = reset_totals(h);
        if (rc) break;
        if (tables) LV_BY_WEIGHT(h, enqueue_sweep_tables, h);
        else LV_BY_WEIGHT(h, enqueue_sweep, h);
        launch_s2(h->S, h->V, h->tot_d->s2, h->stream);
        launch_pdl(sweep_end_kernel, 1, 32, 0, h->stream, h->blk_d, ld, h->flag_h, number);
        note_launches(1);
        // the flag arrives some microseconds before a copy or a synchronisation would return
        for (uint32_t spin = 1; h->flag_h[1] != number; ++spin) {
            if ((spin & 0xFFF) != 0) continue;
            const cudaError_t e = cudaStreamQuery(h->stream);
            if (e == cudaErrorNotReady || h->flag_h[1] == number) continue;
            rc = fail(h, LV_ERR_CUDA, std::string("sweep: ") + cudaGetErrorString(e));
            break;
        }
        if (rc || !h->flag_h[0]) break;
    }
    h->in_loop = false;
    tm.stop();
    LV_TRY(rc);
    LV_CUDA(h, cudaMemcpyAsync(ls, ld, sizeof(*ls), cudaMemcpyDeviceToHost, h->stream));
    LV_CUDA(h, cudaMemcpyAsync(h->tot_h, h->tot_d, sizeof(Totals), cudaMemcpyDeviceToHost, h->stream));
    u64 *cur = reinterpret_cast<u64 *>(h->small_h);
    if (tables)
        LV_CUDA(h, cudaMemcpyAsync(cur, h->nct.cursor, 4 * sizeof(u64), cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    LV_TRY(check_device_error(h, h->tot_h->err));
    const int32_t ran = ls->sweeps - sweeps0;
    if (tables) {
        h->table_sweeps += ran;
        cur[0] = std::min(cur[0], h->nct.cap);   // refused requests count as well
        h->table_slots += (int64_t)cur[0];
        h->table_without += (int64_t)cur[1];
        if (cur[2]) h->table_full = 1;
        if (cur[3]) h->table_stale = 1;
        // rows of up to 32 entries every time, the others once and then their tables
        double wide = 0;
        for (int c = CLS_B4; c < NCLS; ++c) wide += (double)h->cls_edges[c];
        h->st.move_bytes += ran * (12.0 * ((double)h->E - wide) + 20.0 * (double)h->V) + 12.0 * wide +
                            (ran - 1) * sizeof(GSlot) * (double)cur[0];
    }
    h->e_own_cur = ls->e_own;
    h->st.sweeps += ran;
    h->st.edge_sweeps += h->E * (int64_t)ran;
    h->st.moves += (int64_t)(ls->moves_total - moves0);
    return LV_OK;
}

// A level's sweep loop with the decisions taken on the device.
int sweep_loop_device(lv_handle *h, float min_gain, double q_start, int *ch) {
    if (!h->loop_d) {
        LoopState *p = nullptr;
        LV_TRY(dalloc(h, &p, 1));
        h->loop_d = p;
    }
    LoopState ls{};
    ls.q_before = q_start;
    ls.min_gain = (double)min_gain;
    ls.e_own = h->e_own_cur;
    ls.T = h->T;
    ls.q_last = q_start;
    ls.max_sweeps = h->opts.max_sweeps;
    if (h->E >= NCT_MIN_ENTRIES) ls.switch_units = (u64)(NCT_SWITCH * (double)h->E / 32.0);
    LV_TRY(run_sweeps(h, false, &ls));
    if (ls.switched) {
        ls.switched = 0;
        ls.switch_units = 0;
        int ok = 0;
        LV_TRY(nct_begin(h, &ok));
        LV_TRY(run_sweeps(h, ok != 0, &ls));
    }
    *ch = ls.changed;
    return LV_OK;
}

// ---------------------------------------------------------------------------
// learned active set (lv_opts.active_set) and move traces (trace_sample)
// ---------------------------------------------------------------------------
// Levels with fewer vertices than this run plain sweeps in learned mode: their
// sweeps are short and the device-side sweep loop (no host round trip per
// sweep) is cheaper than proposing.
constexpr int32_t ACTIVE_MIN_VERTICES = 1 << 16;

bool learned_mode(const lv_handle *h) {
    return h->opts.trace_sample > 0.0f || (h->opts.active_set != 0 && h->V >= ACTIVE_MIN_VERTICES);
}

int ensure_active(lv_handle *h) {
    if (h->active_ready) return LV_OK;
    const size_t V = (size_t)h->V0 + 1;
    LV_TRY(dalloc(h, &h->feat, 2 * V));
    LV_TRY(dalloc(h, &h->moved, V));
    LV_TRY(dalloc(h, &h->nmoved, V));
    LV_TRY(dalloc(h, &h->pred, V));
    LV_TRY(dalloc(h, &h->fresh, V));
    LV_CUDA(h, cudaMemsetAsync(h->fresh, 0, V, h->stream));
    LV_TRY(dalloc(h, &h->comm_prev, V));
    LV_TRY(dalloc(h, &h->alist, V));
    LV_TRY(dalloc(h, &h->acnt, (size_t)NCLS));
    LV_TRY(dalloc(h, &h->actr, 4));
    LV_CUDA(h, cudaMemsetAsync(h->actr, 0, 4 * sizeof(u64), h->stream));
    if (h->opts.trace_sample > 0.0f) {
        const double r = h->opts.trace_sample < 1.0f ? h->opts.trace_sample : 1.0;
        h->tr_cap = (int64_t)std::ceil(r * (double)h->V0 * 48.0) + 1024;
        LV_TRY(dalloc(h, &h->tr_x, (size_t)h->tr_cap * LV_ACTIVE_FEATURES));
        LV_TRY(dalloc(h, &h->tr_v, (size_t)h->tr_cap));
        LV_TRY(dalloc(h, &h->tr_y, (size_t)h->tr_cap));
    }
    h->active_ready = true;
    return LV_OK;
}

// One sweep over the proposed vertices only (per-class counts cnt, lists at
// the classes' offsets in alist); giants are always in the list.
template <typename WT>
void enqueue_sweep_active(lv_handle *h, const int32_t *cnt) {
    GraphView<WT> g = view_of<WT>(h);
    StateView st = state_of(h);
    u64 *dE = &h->tot_d->dE;
    Timer tm(h, 100);
    int64_t verts = 0;
    for (int b = 0; b < NBUCKETS; ++b) {
        const int c0 = b, c1 = (b < 6) ? b + 1 : NCLS;
        int64_t any = 0;
        for (int c = c0; c < c1; ++c) any += cnt[c];
        if (!any) continue;
        st.mv_cnt = h->blk_d->movers + b;
        next_round(h, st);
        if (b < 4) {
            launch_move_class<WT>(b, g, st, h->alist + h->cls_off[b], cnt[b], dE, h->stream,
                                  narrow_weights<WT>(h));
        } else {
            for (int c = c0; c < c1; ++c) {
                if (c == CLS_HG || !cnt[c]) continue;
                const int32_t maxdeg = c == CLS_B4 ? 84 : (c == CLS_B5 ? 319 : (c == CLS_H1 ? 1024 : h->giant_degree));
                // sets 0..3: classes B4, B5, H1, H2 (H2 shares its large queue with the giants)
                launch_move_wide<WT>(g, st, h->alist + h->cls_off[c], cnt[c], queues_on(h, c - CLS_B4), h->di, dE,
                                     h->stream, maxdeg, narrow_weights<WT>(h), c == CLS_H2 && cnt[CLS_HG] > 0);
            }
            if (b == 6 && cnt[CLS_HG])
                launch_move_giants<WT>(g, st, h->hub_move.view, queues_on(h, CLS_H2 - CLS_B4), h->di, dE, h->stream,
                                       narrow_weights<WT>(h));
        }
        for (int c = c0; c < c1; ++c)
            if (b >= 4) launch_collect_movers<WT>(g, st, h->alist + h->cls_off[c], cnt[c], h->stream);
        launch_movers<WT>(g, st, (int32_t)any, h->di, dE, &h->tot_d->moves, h->stream);
        verts += any;
    }
    tm.bytes = 20.0 * (double)verts;
    tm.stop();
}

// One sweep of the learned / traced loop: full (every vertex) or over the
// proposed vertices; predict = run the predictor first (the proposal of an
// active sweep, or the flags whose recall a full sweep measures).
int sweep_learned(lv_handle *h, bool full, bool predict, int64_t *moves, double *q, int64_t *movers,
                  int64_t *hits, int64_t *fresh_movers) {
    LV_TRY(reset_totals(h));
    clear_move_state(h->fb, h->hub_move.view, h->stream);
    LV_CUDA(h, cudaMemsetAsync(h->actr, 0, 2 * sizeof(u64), h->stream));
    LV_CUDA(h, cudaMemsetAsync(h->actr + 3, 0, sizeof(u64), h->stream));
    const int32_t n = h->cls_off[NCLS];
    ActiveClassOffsets co;
    for (int c = 0; c <= NCLS; ++c) co.off[c] = h->cls_off[c];
    const int32_t *rowend = h->cur_rowend ? h->cur_rowend : h->cur_rowptr + 1;
    int32_t cnt[NCLS];
    const bool tracing = h->opts.trace_sample > 0.0f && h->tr_x;
    // the neighbours that moved in the last sweep, a feature: only where it is
    // read (a first sweep of 1,000,003 vertices, whose movers' rows are most
    // of the graph, does without 90 us)
    if (predict || (tracing && h->tr_sweep > 0))
        launch_nbr_moved(h->cur_rowptr, rowend, h->cur_col, h->V, h->moved, h->nmoved, h->stream);
    if (predict) {
        if (!full) LV_CUDA(h, cudaMemsetAsync(h->acnt, 0, NCLS * sizeof(int32_t), h->stream));
        launch_active_select(h->list, n, co, h->cur_rowptr, rowend, h->feat, h->moved, h->nmoved, h->model, h->logit_thr,
                             CLS_HG, full ? nullptr : h->alist, h->acnt, h->pred, h->fresh, h->stream);
        if (!full) {
            LV_CUDA(h, cudaMemcpyAsync(h->small_h, h->acnt, NCLS * sizeof(int32_t), cudaMemcpyDeviceToHost,
                                       h->stream));
            LV_TRY(sync(h));
            for (int c = 0; c < NCLS; ++c) cnt[c] = h->small_h[c];
        }
    }
    if (tracing && h->tr_sweep > 0) {
        const double r = h->opts.trace_sample < 1.0f ? h->opts.trace_sample : 1.0;
        const u64 thr = r >= 1.0 ? ~0ull : (u64)(r * 18446744073709551616.0);
        launch_trace_sample(h->V, h->cur_rowptr, rowend, h->feat, h->moved, h->nmoved, thr,
                            0x7A11ull * (h->tr_sweep + 1) ^ ((u64)h->level << 40), h->tr_x, h->tr_v, h->tr_cap,
                            h->actr + 2, h->stream);
    }
    LV_CUDA(h, cudaMemcpyAsync(h->comm_prev, h->comm, sizeof(int32_t) * (size_t)h->V, cudaMemcpyDeviceToDevice,
                               h->stream));
    if (full) {
        LV_BY_WEIGHT(h, enqueue_sweep, h);
        h->act_evaluated += n;
        h->act_full += 1;
    } else {
        LV_BY_WEIGHT(h, enqueue_sweep_active, h, cnt);
        for (int c = 0; c < NCLS; ++c) h->act_evaluated += cnt[c];
        h->act_active += 1;
    }
    {
        Timer tm(h, 101);
        launch_s2(h->S, h->V, h->tot_d->s2, h->stream);
        tm.stop();
    }
    launch_active_moved(h->comm, h->comm_prev, h->V, h->moved, predict && full ? h->pred : nullptr, h->fresh,
                        h->actr, h->stream);
    if (tracing && h->tr_sweep > 0)
        launch_trace_label(h->tr_v, h->moved, h->tr_rows, h->actr + 2, h->tr_cap, h->tr_y, h->stream);
    u64 ctr[4];
    LV_CUDA(h, cudaMemcpyAsync(h->small_h, h->actr, sizeof(ctr), cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(read_totals(h));
    std::memcpy(ctr, h->small_h, sizeof(ctr));
    if (tracing) {
        if (h->tr_sweep > 0) h->tr_rows = (int64_t)ctr[2] < h->tr_cap ? (int64_t)ctr[2] : h->tr_cap;
        h->tr_sweep += 1;
    }
    h->e_own_cur += h->tot_h->dE;
    Totals t = *h->tot_h;
    t.e_own = h->e_own_cur;
    *moves = (int64_t)t.moves;
    *movers = (int64_t)ctr[0];
    *hits = (int64_t)ctr[1];
    *fresh_movers = (int64_t)ctr[3];
    *q = q_from_totals(h->T, t);
    h->st.sweeps += 1;
    h->st.edge_sweeps += h->E;
    h->st.moves += *moves;
    return LV_OK;
}

// optimiseModularity with the learned proposal: sweeps are full until one
// moves fewer than active_start of the level's vertices (the early sweeps,
// where most vertices move, stay exactly the plain method's); after that
// every active_full_every-th sweep evaluates every vertex and the others only
// the proposed ones.  A full sweep after a proposal measures its recall over
// the vertices evaluated since the previous full sweep (movers the predictor
// proposes now / movers among them); below active_min_recall the plain sweep
// takes over for the rest of the level.  An active sweep that gains less than
// min_gain (or moves nothing) is followed by a full sweep, and the level ends
// as the plain loop does, on a full sweep.  Without a model (trace recording
// only) every sweep is full and the result equals the plain loop's.
int optimise_level_learned(lv_handle *h, float min_gain, int32_t *changed) {
    LV_TRY(ensure_active(h));
    LV_CUDA(h, cudaMemsetAsync(h->feat, 0, sizeof(float) * 2 * (size_t)h->V, h->stream));
    LV_CUDA(h, cudaMemsetAsync(h->moved, 0, (size_t)h->V, h->stream));
    LV_CUDA(h, cudaMemsetAsync(h->nmoved, 0, sizeof(int32_t) * (size_t)h->V, h->stream));
    LV_CUDA(h, cudaMemsetAsync(h->fresh, 0, (size_t)h->V, h->stream));
    h->tr_sweep = 0;
    double q_before = 0, q_after = 0;
    LV_TRY(modularity(h, &q_before));
    const bool learned = h->opts.active_set != 0 && h->has_model;
    const int K = h->opts.active_full_every > 0 ? h->opts.active_full_every : 4;
    const double rmin = h->opts.active_min_recall > 0.0f ? (double)h->opts.active_min_recall : 0.9;
    const double start = h->opts.active_start > 0.0f ? (double)h->opts.active_start : 0.05;
    bool plain_rest = !learned, force_full = true, proposing = false;
    int since_full = 0, sweeps = 0, ch = 0;
    for (;;) {
        if (h->opts.max_sweeps > 0 && sweeps >= h->opts.max_sweeps) break;
        const bool full = force_full || plain_rest || !proposing || since_full + 1 >= K;
        const bool predict = learned && !plain_rest && proposing;
        int64_t moves = 0, movers = 0, hits = 0, fresh_movers = 0;
        LV_TRY(sweep_learned(h, full, predict, &moves, &q_after, &movers, &hits, &fresh_movers));
        sweeps++;
        const double gain = q_after - q_before;
        if (gain > 0) ch = 1;
        q_before = q_after;
        const bool stall = !(gain >= (double)min_gain) || moves == 0;
        if (full) {
            since_full = 0;
            force_full = false;
            if ((double)movers < start * (double)h->V) proposing = true;
            if (predict) {
                // recall over the movers whose features are current (evaluated
                // since the last full sweep): what the predictor caught, not
                // the moves it postponed
                // (no fresh mover while others moved: the proposals caught
                // nothing, recall 0; nothing moved at all: recall 1)
                h->act_recall = fresh_movers > 0 ? (double)hits / (double)fresh_movers : (movers > 0 ? 0.0 : 1.0);
                if (h->act_recall < rmin) {
                    plain_rest = true;
                    h->act_fell_back = 1;
                }
            }
            if (stall) break;
        } else {
            since_full++;
            if (stall) force_full = true;
        }
    }
    launch_compose_map(h->orig2comm, h->comm, h->V0, h->stream);
    h->st.levels += 1;
    h->st.final_vertices = h->V;
    if (changed) *changed = ch;
    return sync(h);
}

int optimise_level(lv_handle *h, float min_gain, int32_t *changed) {
    LV_TRY(ensure_setup(h));
    h->singletons = false;
    if (learned_mode(h)) return optimise_level_learned(h, min_gain, changed);
    double q_before = 0, q_after = 0;
    LV_TRY(modularity(h, &q_before));
    if (h->opts.sweep_graph && !h->opts.profile && !h->opts.verify && !h->opts.trace) {
        int ch = 0;
        LV_TRY(sweep_loop_device(h, min_gain, q_before, &ch));
        launch_compose_map(h->orig2comm, h->comm, h->V0, h->stream);
        h->st.levels += 1;
        h->st.final_vertices = h->V;
        if (changed) *changed = ch;
        return sync(h);
    }
    double gain = (double)min_gain;
    int ch = 0, sweeps = 0;
    while (gain >= (double)min_gain) {
        if (h->opts.max_sweeps > 0 && sweeps >= h->opts.max_sweeps) break;
        int64_t moves = 0;
        LV_TRY(sweep_and_q(h, &moves, &q_after));
        sweeps++;
        gain = q_after - q_before;
        if (gain > 0) ch = 1;
        q_before = q_after;
        if (moves == 0) break;
    }
    launch_compose_map(h->orig2comm, h->comm, h->V0, h->stream);
    h->st.levels += 1;
    h->st.final_vertices = h->V;
    if (changed) *changed = ch;
    return sync(h);
}

// ---------------------------------------------------------------------------
// aggregation
// ---------------------------------------------------------------------------
int ensure_agg(lv_handle *h) {
    if (h->agg_ready) return LV_OK;
    const size_t V = (size_t)h->V0, E = (size_t)(h->E0 > 0 ? h->E0 : 1);
    AggBuffers &a = h->ab;
    LV_TRY(dalloc(h, &a.flag, V + 1));
    LV_TRY(dalloc(h, &a.cdeg, V + 1));
    LV_TRY(dalloc(h, &a.mstart, V + 1));
    LV_TRY(dalloc(h, &a.cursor, V + 16));
    LV_TRY(dalloc(h, &a.members, V + 1));
    LV_TRY(dalloc(h, &a.lab, V + 1));
    LV_TRY(dalloc(h, &a.clist, V + 1));
    LV_TRY(dalloc(h, &a.newdeg, V + 1));
    LV_TRY(dalloc(h, &a.epos_new, V + 1));
    LV_TRY(dalloc(h, &a.scan_tmp, (size_t)scan_tmp_elems((int64_t)V + 1) + 16));
    LV_TRY(dalloc(h, &a.scalars, 64));
    LV_TRY(dalloc(h, &h->mslot, V + 1));
    LV_TRY(dalloc(h, &h->degm, V + 1));
    LV_TRY(dalloc(h, &h->P, V + 1));
    for (int b = 0; b < 2; ++b) {
        LV_TRY(dalloc(h, &h->lvl_start[b], V + 1));
        LV_TRY(dalloc(h, &h->lvl_end[b], V + 1));
        LV_TRY(dalloc(h, &h->lvl_col[b], E));
        LV_TRY(dalloc(h, &h->lvl_w[b], E));
        LV_TRY(dalloc(h, &h->lvl_w32[b], E));
    }
    h->agg_ready = true;
    return LV_OK;
}

template <typename WT>
int aggregate_t(lv_handle *h) {
    Timer tm(h, 102);
    AggBuffers &ab = h->ab;
    const int32_t V = h->V;
    // the next level's rows are built in the other ping-pong buffer
    const int nb = (h->cur_buf == 0) ? 1 : 0;
    int32_t *vkey = h->lvl_col[nb];
    u64 *vw = h->lvl_w[nb];
    uint32_t *vw32 = h->lvl_w32[nb];
    int32_t *hiflag = ab.scalars + 12;   // set when a merged sum is 2^32 or more
    // the permuted inter-community weights are the current level's
    // non-self-loop weights: below 2^32 when the move phase reads them narrow
    const bool narrow = h->cur_w32 || narrow_weights<WT>(h);
    agg_prepare(h->cur_rowptr, h->cur_rowend, h->comm, h->size, V, ab, h->mslot, h->degm, h->P,
                h->stream);
    LV_CUDA(h, cudaMemcpyAsync(h->small_h, ab.scalars, sizeof(int32_t) * (2 + NAC),
                               cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    const int32_t newV = h->small_h[0];
    int32_t aoff[NAC + 1];
    aoff[0] = 0;
    for (int c = 0; c < NAC; ++c) aoff[c + 1] = aoff[c] + h->small_h[2 + c];
    agg_classify(h->size, V, ab, h->P, aoff, h->stream);
    const int32_t nbig = aoff[NAC] - aoff[NAC - 1];
    std::vector<int32_t> ids(nbig), deg(nbig);
    if (nbig > 0) {
        launch_gather_cdeg(ab.mstart, h->P, ab.clist + aoff[NAC - 1], nbig, ab.cdeg, h->stream);
        LV_CUDA(h, cudaMemcpyAsync(ids.data(), ab.clist + aoff[NAC - 1], sizeof(int32_t) * nbig,
                                   cudaMemcpyDeviceToHost, h->stream));
        LV_CUDA(h, cudaMemcpyAsync(deg.data(), ab.cdeg, sizeof(int32_t) * nbig,
                                   cudaMemcpyDeviceToHost, h->stream));
        LV_TRY(sync(h));
    }
    LV_TRY(build_layout(h, h->hub_agg, ids, deg, newV, true, HG_EDGE_CHUNK, true));
    GraphView<WT> g = view_of<WT>(h);
    for (int c = 0; c < NCLS; ++c)
        agg_permute<WT>(c, g, ab, h->mslot, h->P, h->list + h->cls_off[c],
                        h->cls_off[c + 1] - h->cls_off[c], vkey, vw, h->di.sms, h->stream);
    agg_new_vertices(h->size, h->S, V, ab, h->P, h->k, h->stream);
    LV_CUDA(h, cudaMemsetAsync(hiflag, 0, sizeof(int32_t), h->stream));
    for (int c = 0; c < NAC - 1; ++c)
        agg_merge_class(c, ab, h->P, ab.clist + aoff[c], aoff[c + 1] - aoff[c], vkey, vw, vw32,
                        &h->tot_d->err, hiflag, h->di.sms, h->stream, narrow);
    agg_merge_global(h->hub_agg.view, ab, h->P, vkey, vw, vw32, &h->tot_d->err, hiflag, h->stream,
                     narrow);
    agg_row_bounds(ab, newV, h->lvl_start[nb], h->lvl_end[nb], h->stream);
    // E' = number of stored entries (P is free again after the merges)
    scan_exclusive_i32(ab.newdeg, h->P, newV, h->P + newV, ab.scan_tmp, h->stream);
    LV_CUDA(h, cudaMemcpyAsync(h->small_h, h->P + newV, sizeof(int32_t), cudaMemcpyDeviceToHost,
                               h->stream));
    LV_CUDA(h, cudaMemcpyAsync(h->small_h + 1, hiflag, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    launch_compose_map(h->orig2comm, ab.flag, h->V0, h->stream);
    LV_CUDA(h, cudaMemcpyAsync(h->tot_h, h->tot_d, sizeof(Totals), cudaMemcpyDeviceToHost, h->stream));
    tm.stop();
    LV_TRY(sync(h));
    if (h->opts.trace)
        std::fprintf(stderr, "[lv] aggregate: newV=%d big_communities=%d agg_ms_total=%.3f\n", newV, nbig,
                     h->st.aggregate_ms);
    LV_TRY(check_device_error(h, h->tot_h->err));
    const int64_t newE = h->small_h[0];
    h->cur_buf = nb;
    h->cur_rowptr = h->lvl_start[nb];
    h->cur_rowend = h->lvl_end[nb];
    h->cur_col = h->lvl_col[nb];
    h->cur_w = h->lvl_w[nb];
    h->cur_w32 = h->opts.wide_weights || h->small_h[1] ? nullptr : h->lvl_w32[nb];
    h->V = newV;
    h->E = newE;
    h->level += 1;
    h->e_own_valid = false;
    h->singletons = false;
    h->setup_due = SETUP_ALL;
    if (team_fits(h)) return LV_OK;   // as in to_level0
    return ensure_setup(h);
}

int aggregate(lv_handle *h) {
    LV_TRY(ensure_setup(h));
    LV_TRY(ensure_agg(h));
    const int rc = h->cur_w ? aggregate_t<u64>(h) : aggregate_t<float>(h);
    // the level stays, but its giants' layout may point to staging buffers that
    // the aggregation outgrew before it failed
    if (rc && !h->setup_due) h->setup_due = SETUP_LISTS;
    return rc;
}

// ---------------------------------------------------------------------------
// small levels: the rest of the level loop in one launch
// ---------------------------------------------------------------------------
// A level this small spends its time on launches and host round trips (0.3 to
// 0.6 ms per level and 0.1 ms per sweep), not on its rows.
// lv_run of planted graphs of 500 / 2000 / 3500 vertices (6 / 27 / 58 thousand
// entries) takes 0.87 / 0.81 / 0.63 ms in one launch; 2000 vertices took 1.97
// ms level by level, and at 10,007 vertices (171 thousand entries) the two
// are even (1.60 against 1.69 ms).
bool team_fits(const lv_handle *h) {
    return h->V > 0 && h->E > 0 && h->V <= TEAM_RUN_MAX_V && h->E <= TEAM_RUN_MAX_E && h->opts.sweep_graph &&
           !h->opts.profile && !h->opts.verify && !h->opts.trace && !(h->opts.trace_sample > 0.0f);
}

// Runs the level loop of lv_run to its end from the current level (whose
// communities are singletons); *done = 0 when the launch could not be made.
int team_finish(lv_handle *h, double min_gain, double *q, int *done) {
    *done = 0;
    const size_t bytes = team_arena_bytes(h->V, h->E);
    if (bytes > h->team_bytes) {
        unsigned char *old = (unsigned char *)h->team_arena, *nd = nullptr;
        h->team_arena = nullptr;
        h->team_bytes = 0;
        dfree(h, old);
        LV_TRY(dalloc(h, &nd, bytes));
        h->team_arena = nd;
        h->team_bytes = bytes;
    }
    TeamJob j{};
    j.rs = h->cur_rowptr;
    j.re = h->cur_rowend;
    j.col = h->cur_col;
    j.w = h->cur_w ? nullptr : h->in_w;
    j.w64 = h->cur_w;
    j.V = h->V;
    j.E = h->E;
    j.scale = h->scale_d;
    j.narrow = h->w0_narrow;
    j.min_gain = min_gain;
    j.max_sweeps = h->opts.max_sweeps;
    j.comm = h->comm;
    j.newc = h->newc;
    j.size = h->size;
    j.k = h->k;
    j.S = h->S;
    TeamRows rows;
    {
        Timer tm(h, 100);
        if (!team_run(j, h->team_arena, h->device, h->stream, &rows)) return LV_OK;
        tm.stop();
    }
    launch_compose_map(h->orig2comm, rows.o2c, h->V0, h->stream);
    TeamResult *r = reinterpret_cast<TeamResult *>(h->small_h);
    LV_CUDA(h, cudaMemcpyAsync(r, rows.result, sizeof(TeamResult), cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    if (r->status != LV_OK) return fail(h, LV_ERR_DEVICE, "device check failed in the small-graph launch");
    h->st.levels += r->levels;
    h->st.final_vertices = r->V;
    h->st.sweeps += r->sweeps;
    h->st.edge_sweeps += r->edge_sweeps;
    h->st.moves += r->moves;
    h->st.move_bytes += 12.0 * (double)r->edge_sweeps + 20.0 * (double)r->vertex_sweeps;
    h->level += r->levels - 1;
    h->V = r->V;
    h->E = r->E;
    if (r->cur >= 0) {
        h->cur_rowptr = rows.rs[r->cur];
        h->cur_rowend = rows.re[r->cur];
        h->cur_col = rows.col[r->cur];
        h->cur_w = rows.w64[r->cur];
        h->cur_w32 = nullptr;
        h->cur_buf = -1;
    }
    h->e_own_valid = false;
    h->singletons = false;
    h->setup_due = SETUP_LISTS;
    *q = r->q;
    *done = 1;
    return LV_OK;
}

// ---------------------------------------------------------------------------
// creation
// ---------------------------------------------------------------------------
int to_level0(lv_handle *h) {
    h->level = 0;
    h->V = h->V0;
    h->E = h->E0;
    h->cur_rowptr = h->in_rowptr;
    h->cur_rowend = h->in_rowptr + 1;
    h->cur_col = h->in_col;
    h->cur_w = nullptr;
    h->cur_w32 = nullptr;
    h->cur_buf = -1;
    h->e_own_valid = false;
    launch_iota_i32(h->orig2comm, h->V0, h->stream);
    h->setup_due = SETUP_ALL;
    // a level that lv_run hands to one launch needs no class lists
    if (team_fits(h)) return LV_OK;
    return ensure_setup(h);
}

// Buffers of the move phase (class lists, degree sort, fallback queues).
int ensure_move(lv_handle *h) {
    if (h->move_ready) return LV_OK;
    const size_t V = (size_t)h->V0;
    LV_TRY(dalloc(h, &h->list, V + 1));
    LV_TRY(dalloc(h, &h->mv_list, 4 * V + 1));
    LV_CUDA(h, cudaMemsetAsync(h->mv_list + 3 * V, 0, sizeof(int32_t) * V, h->stream));
    h->mv_round = 0;
    LV_TRY(dalloc(h, &h->sort_buf, 3 * V + 16));
    h->sort_temp_bytes = sort_by_degree_temp_bytes((int32_t)V, HG_MIN_DEG_HI) + 256;
    {
        unsigned char *t = nullptr;
        LV_TRY(dalloc(h, &t, h->sort_temp_bytes));
        h->sort_temp = t;
    }
    {
        // fallback work lists of the move phase.  Only vertices of degree
        // > warp_limit are queued (at most E / warp_limit of them at any
        // level); a large item covers FB_KEYS edges of a vertex of degree
        // > FBQ_MAXDEG(NFBQ - 1), or as many staged pairs of a giant.
        FallbackSet &fs = h->fb;
        LV_TRY(dalloc(h, &fs.hint, V + 1));
        LV_CUDA(h, cudaMemsetAsync(fs.hint, 0, V + 1, h->stream));
        const size_t cap_row = (size_t)(h->E0 / fs.warp_limit) + 64;
        const size_t cap_large = (size_t)(2 * (h->E0 / FBQ_MAXDEG(NFBQ - 1) + h->E0 / FB_KEYS)) + 64;
        for (int q = 0; q <= NFBQ; ++q) {
            Fallback &f = fs.q[q];
            const size_t cap = q < NFBQ ? cap_row : cap_large;
            f.cap = (int32_t)cap;
            LV_TRY(dalloc(h, &f.v, cap));
            if (q < NFBQ) continue;
            LV_TRY(dalloc(h, &f.p, cap));
            LV_TRY(dalloc(h, &f.P, cap));
            LV_TRY(dalloc(h, &f.first, cap));
            LV_TRY(dalloc(h, &f.src, cap));
            LV_TRY(dalloc(h, &f.done, cap));
            LV_TRY(dalloc(h, &f.gd, cap));
            LV_TRY(dalloc(h, &f.e, cap));
            LV_TRY(dalloc(h, &f.S, cap));
            LV_TRY(dalloc(h, &f.eo, cap));
            LV_TRY(dalloc(h, &f.c, cap));
            LV_TRY(dalloc(h, &f.cnt, cap));
            LV_CUDA(h, cudaMemsetAsync(f.done, 0, cap * sizeof(int32_t), h->stream));
        }
    }
    h->move_ready = true;
    return LV_OK;
}

int finish_create(lv_handle *h) {
    const size_t V = (size_t)h->V0;
    if (h->opts.trace)
        std::fprintf(stderr, "[lv] device %d memory pool: %s\n", h->device,
                     mem_pooled(h->device) ? "on" : "off (cudaMalloc per buffer)");
    LV_TRY(dalloc(h, &h->comm, V + 1));
    LV_TRY(dalloc(h, &h->newc, V + 1));
    LV_TRY(dalloc(h, &h->size, V + 1));
    LV_TRY(dalloc(h, &h->orig2comm, V + 1));
    LV_TRY(dalloc(h, &h->k, V + 1));
    LV_TRY(dalloc(h, &h->S, V + 1));
    LV_TRY(dalloc(h, &h->cls_scratch, V + SCRATCH_OFF + 16));
    LV_TRY(dalloc(h, &h->blk_d, 1));
    h->tot_d = &h->blk_d->tot;
    LV_CUDA(h, cudaMemsetAsync(h->blk_d, 0, sizeof(SweepBlock), h->stream));
    LV_TRY(pinned_take(h));
    // CSR checks, fixed-point scale (same rule as the oracle's orc_choose_scale)
    // and total weight; one read back
    int32_t *ws = h->cls_scratch;
    u64 *tw = (u64 *)(h->tot_d);   // reuse e_own slot
    launch_csr_scan(h->in_rowptr, h->in_col, h->in_w, h->V0, h->E0, &h->tot_d->err, ws, nullptr, 0, h->stream);
    launch_total_weight(h->in_w, h->E0, &h->tot_d->err, ws, tw, h->stream);
    LV_CUDA(h, cudaMemcpyAsync(h->tot_h, h->tot_d, sizeof(Totals), cudaMemcpyDeviceToHost, h->stream));
    LV_CUDA(h, cudaMemcpyAsync(h->small_h, ws, sizeof(int32_t) * 3, cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    if (h->tot_h->err) return fail(h, LV_ERR_INVALID, "malformed CSR (offsets or column ids)");
    if (h->small_h[2]) return fail(h, LV_ERR_WEIGHT, "negative, NaN or infinite edge weight");
    const int need = h->small_h[0];
    const int top = h->small_h[1] ? h->small_h[1] - 1024 : 0;
    const int s = scale_of_scan(h->small_h, h->E0);
    if (s < 0) return fail(h, LV_ERR_TOO_LARGE, "total edge weight exceeds the fixed-point range");
    h->scale = s;
    h->exact = (s == need);
    // every fixed-point weight is at most 2^(top + 1 + scale) (rounding included)
    h->w0_narrow = !h->small_h[1] || top + 1 + s <= 31;
    h->scale_d = std::ldexp(1.0, s);
    h->T = h->tot_h->e_own;
    LV_CUDA(h, cudaMemsetAsync(h->tot_d, 0, sizeof(Totals), h->stream));
    return to_level0(h);
}

int begin_create(const lv_opts *opts, int32_t V, int64_t E, lv_handle **out, lv_handle **hp) {
    if (!out) return LV_ERR_INVALID;
    *out = nullptr;
    if (V < 0 || E < 0) return LV_ERR_INVALID;
    if (E > 0x7fffffffLL || V >= 0x7fffffff) return LV_ERR_TOO_LARGE;
    lv_handle *h = new lv_handle();
    lv_default_opts(&h->opts);
    if (opts) {
        size_t n = opts->struct_size && opts->struct_size < sizeof(lv_opts) ? opts->struct_size : sizeof(lv_opts);
        std::memcpy(&h->opts, opts, n);
        h->opts.struct_size = sizeof(lv_opts);
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        delete h;
        return LV_ERR_NO_DEVICE;
    }
    if (h->opts.device < 0 || h->opts.device >= ndev) {
        delete h;
        return LV_ERR_INVALID;
    }
    // work-mapping knobs (0 = default); results never depend on them
    if (h->opts.giant_degree != 0 &&
        (h->opts.giant_degree < HG_MIN_DEG_LO || h->opts.giant_degree > HG_MIN_DEG_HI)) {
        delete h;
        return LV_ERR_INVALID;
    }
    if (h->opts.warp_limit != 0 && (h->opts.warp_limit < WARP_LIMIT_MIN || h->opts.warp_limit > WARP_LIMIT_MAX)) {
        delete h;
        return LV_ERR_INVALID;
    }
    h->giant_degree = h->opts.giant_degree ? h->opts.giant_degree : HG_MIN_DEG;
    h->fb.warp_limit = h->opts.warp_limit ? h->opts.warp_limit : WARP_LIMIT;
    h->fb.hint_set = (h->fb.warp_limit * 3) / 4;
    h->device = h->opts.device;
    cudaSetDevice(h->device);
    h->mem.dev = h->device;
    if (stream_take(h->device, &h->stream) != cudaSuccess) {
        cudaGetLastError();
        delete h;
        return LV_ERR_CUDA;
    }
    static bool attrs_done[64] = {false};
    init_kernel_attributes(h->di);
    if (h->device < 64 && !attrs_done[h->device]) {
        init_agg_attributes();
        attrs_done[h->device] = true;
    }
    h->V0 = V;
    h->E0 = E;
    h->launch_base = launches_total();
    *hp = h;
    return LV_OK;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

void lv_default_opts(lv_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->struct_size = sizeof(lv_opts);
    o->device = 0;
    o->max_sweeps = 0;
    o->sweep_graph = 1;
    o->profile = 0;
}

const char *lv_status_string(int s) {
    switch (s) {
    case LV_OK: return "ok";
    case LV_ERR_INVALID: return "invalid argument or malformed CSR";
    case LV_ERR_WEIGHT: return "negative, NaN or infinite weight";
    case LV_ERR_TOO_LARGE: return "graph too large for int32 ids or the fixed-point grid";
    case LV_ERR_NOMEM: return "out of memory";
    case LV_ERR_CUDA: return "CUDA error";
    case LV_ERR_DEVICE: return "device-side check failed";
    case LV_ERR_IO: return "I/O or parse error";
    case LV_ERR_NO_DEVICE: return "no CUDA device";
    default: return "unknown status";
    }
}

int lv_trim_device_memory(int32_t device) {
    if (device < 0 || device >= 64) return LV_ERR_INVALID;
    return mem_trim(device) == cudaSuccess ? LV_OK : LV_ERR_CUDA;
}

const char *lv_version(void) { return "louvain_b200 0.1 (sm_100a)"; }

int lv_destroy(lv_handle *h) {
    if (!h) return LV_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    // every buffer goes back: the stream has drained
    h->mem.give_all(h->stream);
    pinned_give(h);
    for (const Pending &p : h->pend) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
    for (cudaEvent_t e : h->ev_free) cudaEventDestroy(e);
    stream_give(h->device, h->stream);
    delete h;
    return LV_OK;
}

int lv_create(const int32_t *rowptr, const int32_t *col, const float *w, int32_t V, int64_t E,
              const lv_opts *opts, lv_handle **out) {
    if (!rowptr || (E > 0 && (!col || !w))) return LV_ERR_INVALID;
    lv_handle *h = nullptr;
    int rc = begin_create(opts, V, E, out, &h);
    if (rc) return rc;
    h->owns_input = true;
    rc = dalloc(h, &h->in_rowptr, (size_t)V + 1);
    if (!rc) rc = dalloc(h, &h->in_col, (size_t)E);
    if (!rc) rc = dalloc(h, &h->in_w, (size_t)E);
    if (!rc && cudaMemcpyAsync(h->in_rowptr, rowptr, sizeof(int32_t) * ((size_t)V + 1),
                               cudaMemcpyHostToDevice, h->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc && E > 0 &&
        cudaMemcpyAsync(h->in_col, col, sizeof(int32_t) * (size_t)E, cudaMemcpyHostToDevice,
                        h->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc && E > 0 &&
        cudaMemcpyAsync(h->in_w, w, sizeof(float) * (size_t)E, cudaMemcpyHostToDevice,
                        h->stream) != cudaSuccess)
        rc = LV_ERR_CUDA;
    if (!rc) rc = finish_create(h);
    if (rc) {
        lv_destroy(h);
        return rc;
    }
    *out = h;
    return LV_OK;
}

int lv_create_device(const int32_t *d_rowptr, const int32_t *d_col, const float *d_w, int32_t V,
                     int64_t E, const lv_opts *opts, lv_handle **out) {
    if (!d_rowptr || (E > 0 && (!d_col || !d_w))) return LV_ERR_INVALID;
    lv_handle *h = nullptr;
    int rc = begin_create(opts, V, E, out, &h);
    if (rc) return rc;
    h->owns_input = false;
    h->in_rowptr = const_cast<int32_t *>(d_rowptr);
    h->in_col = const_cast<int32_t *>(d_col);
    h->in_w = const_cast<float *>(d_w);
    rc = finish_create(h);
    if (rc) {
        lv_destroy(h);
        return rc;
    }
    *out = h;
    return LV_OK;
}

const char *lv_last_error(const lv_handle *h) { return h ? h->err.c_str() : "null handle"; }

int lv_reset(lv_handle *h) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    return to_level0(h);
}

int lv_optimise_level(lv_handle *h, float min_gain, int32_t *changed) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    return optimise_level(h, min_gain, changed);
}

int lv_aggregate(lv_handle *h) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    return aggregate(h);
}

int lv_modularity(lv_handle *h, double *q) {
    if (!h || !q) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    LV_TRY(ensure_setup(h));
    return modularity(h, q);
}

int lv_sweep(lv_handle *h, int64_t *moves) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    int64_t m = 0;
    LV_TRY(ensure_setup(h));
    LV_TRY(sweep_and_q(h, &m, nullptr));
    if (moves) *moves = m;
    return LV_OK;
}

int lv_run(lv_handle *h, float min_gain, double *q) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    double qq = 0;
    for (;;) {
        if ((double)min_gain >= TEAM_RUN_MIN_GAIN && team_fits(h) &&
            (h->singletons || h->setup_due == SETUP_ALL)) {
            int done = 0;
            LV_TRY(team_finish(h, (double)min_gain, &qq, &done));
            if (done) {
                if (q) *q = qq;
                return LV_OK;
            }
        }
        int32_t changed = 0;
        LV_TRY(optimise_level(h, min_gain, &changed));
        if (!changed) break;
        LV_TRY(aggregate(h));
    }
    LV_TRY(modularity(h, &qq));
    if (q) *q = qq;
    return LV_OK;
}

int lv_get_original_to_community(lv_handle *h, int32_t *out, int32_t *num_communities) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    if (out && h->V0 > 0)
        LV_CUDA(h, cudaMemcpyAsync(out, h->orig2comm, sizeof(int32_t) * (size_t)h->V0,
                                   cudaMemcpyDeviceToHost, h->stream));
    LV_TRY(sync(h));
    if (num_communities) *num_communities = h->V;
    return LV_OK;
}

int lv_get_communities(lv_handle *h, int32_t *out) {
    if (!h || !out) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    if (h->setup_due == SETUP_ALL) LV_TRY(ensure_setup(h));
    if (h->V > 0)
        LV_CUDA(h, cudaMemcpyAsync(out, h->comm, sizeof(int32_t) * (size_t)h->V,
                                   cudaMemcpyDeviceToHost, h->stream));
    return sync(h);
}

int lv_set_communities(lv_handle *h, const int32_t *comm) {
    if (!h || !comm) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    if (h->V == 0) return LV_OK;
    if (h->setup_due == SETUP_ALL) LV_TRY(ensure_setup(h));
    h->singletons = false;
    int32_t *tmp = h->cls_scratch + SCRATCH_OFF;   // V0 entries of scratch
    LV_CUDA(h, cudaMemcpyAsync(tmp, comm, sizeof(int32_t) * (size_t)h->V, cudaMemcpyHostToDevice,
                               h->stream));
    LV_CUDA(h, cudaMemsetAsync(&h->tot_d->err, 0, sizeof(int), h->stream));
    launch_set_communities(tmp, h->comm, h->newc, h->size, h->k, h->S, h->V, &h->tot_d->err, h->stream);
    h->e_own_valid = false;
    LV_TRY(read_totals(h));
    return LV_OK;
}

int lv_set_test_limits(lv_handle *h, int32_t fail_alloc, int64_t table_slots) {
    if (!h || fail_alloc < 0 || table_slots < 0) return LV_ERR_INVALID;
    h->mem.fail_at = fail_alloc;
    h->table_limit = table_slots;
    return LV_OK;
}

int lv_get_table_stats(lv_handle *h, int64_t *sweeps, int64_t *slots, int64_t *without, int32_t *pool_full,
                       int32_t *stale) {
    if (!h) return LV_ERR_INVALID;
    if (sweeps) *sweeps = h->table_sweeps;
    if (slots) *slots = h->table_slots;
    if (without) *without = h->table_without;
    if (pool_full) *pool_full = h->table_full;
    if (stale) *stale = h->table_stale;
    return LV_OK;
}

int lv_get_level_info(lv_handle *h, int32_t *V, int64_t *E, int32_t *level) {
    if (!h) return LV_ERR_INVALID;
    if (V) *V = h->V;
    if (E) *E = h->E;
    if (level) *level = h->level;
    return LV_OK;
}

int lv_get_level_classes(lv_handle *h, int32_t *vertices, int64_t *entries) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    LV_TRY(ensure_setup(h));
    for (int c = 0; c < NCLS; ++c) {
        if (vertices) vertices[c] = h->cls_off[c + 1] - h->cls_off[c];
        if (entries) entries[c] = h->cls_edges[c];
    }
    return LV_OK;
}

int lv_get_device_name(int32_t device, char *name, int32_t len) {
    if (!name || len <= 0) return LV_ERR_INVALID;
    cudaDeviceProp p;
    if (cudaGetDeviceProperties(&p, device) != cudaSuccess) {
        cudaGetLastError();
        return LV_ERR_NO_DEVICE;
    }
    std::snprintf(name, (size_t)len, "%s (sm_%d%d, %d SMs)", p.name, p.major, p.minor, p.multiProcessorCount);
    return LV_OK;
}

int lv_get_csr(lv_handle *h, int32_t *rowptr, int32_t *col, int64_t *wfix) {
    if (!h) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    if (h->level == 0) {
        if (rowptr)
            LV_CUDA(h, cudaMemcpyAsync(rowptr, h->cur_rowptr, sizeof(int32_t) * ((size_t)h->V + 1),
                                       cudaMemcpyDeviceToHost, h->stream));
        if (col && h->E > 0)
            LV_CUDA(h, cudaMemcpyAsync(col, h->cur_col, sizeof(int32_t) * (size_t)h->E,
                                       cudaMemcpyDeviceToHost, h->stream));
        if (wfix && h->E > 0) {
            MemBlock tb;
            if (mem_take(h->device, sizeof(int64_t) * (size_t)h->E, h->stream, &tb) != cudaSuccess)
                return fail(h, LV_ERR_NOMEM, "device allocation");
            int64_t *tmp = (int64_t *)tb.p;
            launch_weights_to_fixed<float>(h->in_w, h->E, h->scale_d, tmp, h->stream);
            cudaError_t e = cudaMemcpyAsync(wfix, tmp, sizeof(int64_t) * (size_t)h->E,
                                            cudaMemcpyDeviceToHost, h->stream);
            cudaStreamSynchronize(h->stream);
            mem_give(h->device, tb, h->stream);
            if (e != cudaSuccess) return fail(h, LV_ERR_CUDA, cudaGetErrorString(e));
        }
        return sync(h);
    }
    // aggregated level: gather the (possibly non-contiguous) rows on the host
    const size_t V = (size_t)h->V;
    std::vector<int32_t> st(V + 1), en(V + 1);
    if (V) {
        LV_CUDA(h, cudaMemcpyAsync(st.data(), h->cur_rowptr, sizeof(int32_t) * V, cudaMemcpyDeviceToHost,
                                   h->stream));
        LV_CUDA(h, cudaMemcpyAsync(en.data(), h->cur_rowend, sizeof(int32_t) * V, cudaMemcpyDeviceToHost,
                                   h->stream));
    }
    LV_TRY(sync(h));
    int32_t span = 0;
    for (size_t v = 0; v < V; ++v) span = en[v] > span ? en[v] : span;
    std::vector<int32_t> c((size_t)span);
    std::vector<u64> w((size_t)span);
    if (span) {
        LV_CUDA(h, cudaMemcpyAsync(c.data(), h->cur_col, sizeof(int32_t) * (size_t)span,
                                   cudaMemcpyDeviceToHost, h->stream));
        LV_CUDA(h, cudaMemcpyAsync(w.data(), h->cur_w, sizeof(u64) * (size_t)span, cudaMemcpyDeviceToHost,
                                   h->stream));
    }
    LV_TRY(sync(h));
    int64_t at = 0;
    for (size_t v = 0; v < V; ++v) {
        if (rowptr) rowptr[v] = (int32_t)at;
        for (int32_t e = st[v]; e < en[v]; ++e, ++at) {
            if (col) col[at] = c[(size_t)e];
            if (wfix) wfix[at] = (int64_t)w[(size_t)e];
        }
    }
    if (rowptr) rowptr[V] = (int32_t)at;
    return LV_OK;
}

int lv_get_scale(lv_handle *h, int32_t *scale, uint64_t *total_weight, int32_t *exact) {
    if (!h) return LV_ERR_INVALID;
    if (scale) *scale = h->scale;
    if (total_weight) *total_weight = h->T;
    if (exact) *exact = h->exact;
    return LV_OK;
}

int lv_set_active_model(lv_handle *h, const uint16_t *model, int32_t n_params, float logit_threshold) {
    if (!h || !model || n_params != LV_ACTIVE_MODEL_SIZE) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    if (!h->model) LV_TRY(dalloc(h, &h->model, (size_t)LV_ACTIVE_MODEL_SIZE));
    LV_CUDA(h, cudaMemcpyAsync(h->model, model, sizeof(uint16_t) * LV_ACTIVE_MODEL_SIZE, cudaMemcpyHostToDevice,
                               h->stream));
    h->logit_thr = logit_threshold;
    h->has_model = true;
    return sync(h);
}

int lv_get_traces(lv_handle *h, float *features, uint8_t *labels, int64_t cap, int64_t *n) {
    if (!h || cap < 0) return LV_ERR_INVALID;
    cudaSetDevice(h->device);
    const int64_t rows = h->tr_rows;
    if (n) *n = rows;
    const int64_t m = rows < cap ? rows : cap;
    if (m > 0 && features)
        LV_CUDA(h, cudaMemcpyAsync(features, h->tr_x, sizeof(float) * LV_ACTIVE_FEATURES * (size_t)m,
                                   cudaMemcpyDeviceToHost, h->stream));
    if (m > 0 && labels)
        LV_CUDA(h, cudaMemcpyAsync(labels, h->tr_y, (size_t)m, cudaMemcpyDeviceToHost, h->stream));
    return sync(h);
}

int lv_get_active_stats(lv_handle *h, int64_t *evaluated, int64_t *full_sweeps, int64_t *active_sweeps,
                        double *last_recall, int32_t *fell_back) {
    if (!h) return LV_ERR_INVALID;
    if (evaluated) *evaluated = h->act_evaluated;
    if (full_sweeps) *full_sweeps = h->act_full;
    if (active_sweeps) *active_sweeps = h->act_active;
    if (last_recall) *last_recall = h->act_recall;
    if (fell_back) *fell_back = h->act_fell_back;
    return LV_OK;
}

int lv_get_stats(lv_handle *h, lv_stats *s) {
    if (!h || !s) return LV_ERR_INVALID;
    LV_TRY(sync(h));
    *s = h->st;
    s->kernel_launches = launches_total() - h->launch_base;
    return LV_OK;
}

int lv_get_class_stats(lv_handle *h, lv_class_stats *s) {
    if (!h || !s) return LV_ERR_INVALID;
    LV_TRY(sync(h));
    *s = h->cst;
    return LV_OK;
}

int lv_clear_stats(lv_handle *h) {
    if (!h) return LV_ERR_INVALID;
    LV_TRY(sync(h));
    std::memset(&h->st, 0, sizeof(h->st));
    std::memset(&h->cst, 0, sizeof(h->cst));
    h->launch_base = launches_total();
    h->act_evaluated = h->act_full = h->act_active = 0;
    h->act_recall = -1.0;
    h->act_fell_back = 0;
    h->table_sweeps = h->table_slots = h->table_without = 0;
    h->table_full = h->table_stale = 0;
    return LV_OK;
}

}  // extern "C"
