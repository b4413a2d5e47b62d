// lv_nct.cuh -- neighbour-community tables: the late sweeps of a level.
// Included by lv_move.cu after the move phase's shared helpers.
//
// After a level's first sweeps few vertices move, yet every sweep sums every
// row by community again: on an R-MAT-24 graph's second level 24 of 28 sweeps
// move under 10 % of the vertices and each reads 482 million entries (4.1 ms).
// Once few row entries belong to movers, each vertex of degree > 32 keeps its
// sums e_{v,C} in a table in global memory (its own community included), built
// at its next evaluation.  From then on it is evaluated from the table, a few
// dozen slots instead of hundreds of row entries with their gathers and shared
// atomics, and every committed move adds its entry's weight to the new and
// takes it from the old community in its neighbours' tables.  Sums are exact
// integers, so the values, and with them every decision, are those of a pass
// over the rows.  This needs each entry to have its mirror entry (the mover's
// row updates the neighbours' sums) and no entry of weight zero (a slot whose
// sum returns to zero is no neighbour); the engine checks both per level.
//
// A table has 2^lg slots, at least twice the distinct communities at its
// build.  A community that finds no free slot near its hash makes the table
// stale (lg = 0), and the vertex's next evaluation builds a new one; so does
// an exhausted slot pool, each time.  Vertices with more than FB_KEYS distinct
// communities never get one (lg = NCT_NEVER) and keep the partition paths.
#pragma once

constexpr int NCT_LG = 8, NCT_SLOTS = 1 << NCT_LG;   // a warp's build table
constexpr int NCT_U = 2;
constexpr int NCT_CLAIMS = 160;   // distinct communities a warp builds; more go to a CTA
static_assert(NCT_CLAIMS + 32 * NCT_U < NCT_SLOTS, "a step's claims fit the build table");
static_assert(NCT_CLAIMS >= 84, "bucket 4 needs no CTA builds");
constexpr uint32_t NCT_PROBES = 32;

// Adds w to community c's sum; false when no slot is free near its hash.
__device__ __forceinline__ bool nct_add(GSlot *tb, int lg, int32_t c, u64 w, uint32_t probes) {
    const uint32_t mask = (1u << lg) - 1u, key1 = (uint32_t)c + 1u;
    uint32_t s = hash_slot(c, lg);
    for (uint32_t p = 0; p <= mask && p < probes; ++p) {
        const uint32_t k = ((volatile GSlot *)tb)[s].key1;
        if (k == key1) { atomicAdd(&tb[s].val, w); return true; }
        if (k == 0) {
            const uint32_t prev = atomicCAS(&tb[s].key1, 0u, key1);
            if (prev == 0 || prev == key1) { atomicAdd(&tb[s].val, w); return true; }
        }
        s = (s + 1u) & mask;
    }
    return false;
}

// Sets a word to 1 (a store only the first time).
__device__ __forceinline__ void nct_flag(u64 *p) {
    if (*(volatile u64 *)p == 0) *(volatile u64 *)p = 1;
}

// A neighbour of j, over an entry of weight w, moves between communities.
__device__ __forceinline__ void nct_move(const NctView &t, int32_t j, int32_t from, int32_t to, u64 w) {
    const int lg = ((volatile uint8_t *)t.lg)[j];
    if (lg == 0 || lg == NCT_NEVER) return;
    GSlot *tb = t.slots + t.off[j];
    const uint32_t mask = (1u << lg) - 1u, key1 = (uint32_t)from + 1u;
    uint32_t s = hash_slot(from, lg);
    bool ok = false;
    for (uint32_t p = 0; p <= mask; ++p) {
        const uint32_t k = ((volatile GSlot *)tb)[s].key1;
        if (k == key1) {
            atomicAdd(&tb[s].val, (u64)0 - w);
            ok = true;
            break;
        }
        if (k == 0) break;
        s = (s + 1u) & mask;
    }
    if (ok) ok = nct_add(tb, lg, to, w, NCT_PROBES);
    if (!ok) {
        t.lg[j] = 0;   // stale: the next evaluation reads the row again
        nct_flag(t.cursor + 3);
    }
}

// Would tables be small?  A warp per sampled vertex (n of them, evenly spaced in
// list[0 .. m)) counts the row's distinct communities: out[0] += the slots its
// table would take (as if all were distinct when there are more than
// NCT_SAMPLE_MAX), out[1] += its entries.
constexpr int NCT_SAMPLE_MAX = 352;

__global__ void __launch_bounds__(256) nct_sample_kernel(const int32_t *__restrict__ rowptr,
                                                         const int32_t *__restrict__ rowend,
                                                         const int32_t *__restrict__ col,
                                                         const int32_t *__restrict__ comm,
                                                         const int32_t *__restrict__ list, int32_t m, int32_t n,
                                                         u64 *out) {
    constexpr int LG = 9;
    __shared__ int32_t skeys[8 << LG];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int32_t *keys = skeys + (wid << LG);
    for (int s = lane; s < (1 << LG); s += 32) keys[s] = -1;
    __syncwarp();
    const int32_t i = (int32_t)blockIdx.x * 8 + wid;
    if (i >= n) return;
    const int32_t v = list[(int64_t)i * m / n];
    const int32_t r0 = rowptr[v], r1 = rowend[v];
    int32_t d = 0;
    for (int32_t b0 = r0; b0 < r1 && d <= NCT_SAMPLE_MAX; b0 += 32) {
        bool fresh = false;
        if (b0 + lane < r1) {
            const int32_t c = comm[__ldg(col + b0 + lane)];
            uint32_t s = hash_slot(c, LG);
            for (;;) {   // at most NCT_SAMPLE_MAX + 32 of the 512 slots are ever taken
                const int32_t prev = atomicCAS(keys + s, -1, c);
                fresh = prev < 0;
                if (fresh || prev == c) break;
                s = (s + 1u) & ((1u << LG) - 1u);
            }
        }
        d += __popc(__ballot_sync(FULL, fresh));
    }
    if (lane == 0) {
        if (d > NCT_SAMPLE_MAX) d = r1 - r0;
        atomicAdd(out, 1ull << max(5, ceil_log2_i(2 * (int64_t)(d + 1))));
        atomicAdd(out + 1, (u64)(r1 - r0));
    }
}

// Slots for a table of d communities from the pool (one thread): the offset,
// or false when the pool is used up.
__device__ __forceinline__ bool nct_alloc(const NctView &t, int32_t d, int *lg, uint32_t *off) {
    *lg = max(5, ceil_log2_i(2 * (int64_t)d));
    const u64 cap = 1ull << *lg;
    if (*((volatile u64 *)t.cursor) + cap <= t.cap) {
        const u64 at = atomicAdd(t.cursor, cap);
        *off = (uint32_t)at;
        if (at + cap <= t.cap) return true;
    }
    nct_flag(t.cursor + 2);
    return false;
}

// A warp per vertex of list[0 .. n) (one update bucket, degree > 32), 32
// headers loaded at a time.  Built vertices are decided from their tables;
// the others from their rows, leaving a table, or queued for a CTA
// (nct_build_kernel) when the row is a giant's or shows more than NCT_CLAIMS
// communities.  Bound by the latency of header -> slots -> Sigma_tot.
template <typename WT>
__global__ void __launch_bounds__(256) nct_eval_kernel(GraphView<WT> g, StateView st,
                                                       const int32_t *__restrict__ list, int32_t n, NctView t,
                                                       Fallback large, int32_t giant_degree, u64 *dE) {
    __shared__ u64 svals[8 * NCT_SLOTS];
    __shared__ int32_t skeys[8 * NCT_SLOTS];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u64 *vals = svals + wid * NCT_SLOTS;
    int32_t *keys = skeys + wid * NCT_SLOTS;
    for (int s = lane; s < NCT_SLOTS; s += 32) { keys[s] = -1; vals[s] = 0; }
    __syncwarp();
    const int32_t nw = (int32_t)gridDim.x * 8, w = (int32_t)blockIdx.x * 8 + wid;
    const int32_t rounds = (int32_t)(((int64_t)n + (int64_t)nw * 32 - 1) / ((int64_t)nw * 32));
    const int32_t cs = (int32_t)(((int64_t)n + (int64_t)nw * rounds - 1) / ((int64_t)nw * rounds));   // <= 32
    u64 delta_acc = 0;
    for (int64_t c0 = (int64_t)w * cs; c0 < n; c0 += (int64_t)nw * cs) {
        const int cnt = (int)imin64(cs, n - c0);
        int32_t hv = 0, hown = 0, hlg = 0, hsz = 0;
        uint32_t hoff = 0;
        u64 hk = 0, hS = 0;
        if (lane < cnt) {
            hv = list[c0 + lane];
            hlg = t.lg[hv];
            hoff = t.off[hv];
            hown = __ldg(st.comm + hv);
            hk = __ldg(st.k + hv);
            hS = __ldg(st.S + hown);
            hsz = __ldg(st.size + hown);
        }
        for (int i = 0; i < cnt; ++i) {
            const int32_t v = __shfl_sync(FULL, hv, i), own = __shfl_sync(FULL, hown, i);
            const int lg = __shfl_sync(FULL, hlg, i);
            const u64 kv = __shfl_sync(FULL, hk, i), sown = __shfl_sync(FULL, hS, i);
            const MoveCtx m = move_ctx(own, __shfl_sync(FULL, hsz, i) == 1, st.T, kv, sown);
            Best b = best_init(own);
            if (lg != 0 && lg != NCT_NEVER) {
                const GSlot *tb = t.slots + __shfl_sync(FULL, hoff, i);
                const int32_t cap = 1 << lg;
                for (int32_t s0 = lane; s0 < cap; s0 += 64) {
                    uint4 x[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        x[u] = s0 + 32 * u < cap ? *reinterpret_cast<const uint4 *>(tb + s0 + 32 * u)
                                                 : make_uint4(0, 0, 0, 0);
                    u64 SS[2];
                    int32_t zz[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int32_t c = (int32_t)x[u].x - 1;
                        const bool cand = x[u].x != 0 && (x[u].z | x[u].w) != 0 && c != own;
                        SS[u] = cand ? __ldg(st.S + c) : 0;
                        zz[u] = cand && guard_needs_size(m, c) ? __ldg(st.size + c) : 0;
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const u64 e = ((u64)x[u].w << 32) | (u64)x[u].z;
                        if (x[u].x != 0 && e != 0) eval_loaded((int32_t)x[u].x - 1, e, SS[u], zz[u], m, b);
                    }
                }
            } else {
                const int32_t r0 = g.rowptr[v], r1 = g.rowend[v], d = r1 - r0;
                if (lg == NCT_NEVER) {
                    // giants: the staged path; others: partitions in the large queue
                    if (d <= giant_degree && lane == 0) enqueue_large(large, v, d, st.err);
                    continue;
                }
                bool over = d > giant_degree;
                u64 e_own = 0;
                int32_t claims = 0;
                for (int32_t b0 = r0; b0 < r1 && !over; b0 += 32 * NCT_U) {
                    int32_t jj[NCT_U];
                    u64 ww[NCT_U];
#pragma unroll
                    for (int u = 0; u < NCT_U; ++u) {
                        const int32_t e = b0 + lane + 32 * u;
                        jj[u] = -1;
                        ww[u] = 0;
                        if (e < r1) { jj[u] = __ldg(g.col + e); ww[u] = gw(g, e); }
                    }
                    unsigned mine = 0;
                    int32_t cc[NCT_U];
#pragma unroll
                    for (int u = 0; u < NCT_U; ++u) cc[u] = (jj[u] >= 0 && jj[u] != v) ? __ldg(st.comm + jj[u]) : -1;
#pragma unroll
                    for (int u = 0; u < NCT_U; ++u) {
                        if (cc[u] < 0) continue;
                        if (cc[u] == own) e_own += ww[u];
                        else mine += table_insert_claim(keys, vals, NCT_LG, cc[u], ww[u], st.err) >= 0 ? 1u : 0u;
                    }
                    claims += (int32_t)__reduce_add_sync(FULL, mine);
                    over = claims > NCT_CLAIMS;
                }
                __syncwarp();
                if (over) {
                    for (int s = lane; s < NCT_SLOTS; s += 32) {
                        if (keys[s] >= 0) { keys[s] = -1; vals[s] = 0; }
                    }
                    if (lane == 0) t.queue[atomicAdd(t.qctr, 1)] = v;
                    __syncwarp();
                    continue;
                }
                e_own = warp_sum_u64(e_own);
                int nlg = 0;
                uint32_t noff = 0;
                int ok = 0;
                if (lane == 0) ok = nct_alloc(t, claims + 1, &nlg, &noff) ? 1 : 0;
                ok = __shfl_sync(FULL, ok, 0);
                nlg = __shfl_sync(FULL, nlg, 0);
                GSlot *tb = t.slots + __shfl_sync(FULL, noff, 0);
                if (ok) {
                    for (int s = lane; s < (1 << nlg); s += 32)
                        *reinterpret_cast<uint4 *>(tb + s) = make_uint4(0, 0, 0, 0);
                    __syncwarp();
                    if (lane == 0 && e_own) nct_add(tb, nlg, own, e_own, 1u << nlg);
                }
                if (lane == 0) b.eo = e_own;
                for (int s = lane; s < NCT_SLOTS; s += 32) {
                    const int32_t c = keys[s];
                    if (c < 0) continue;
                    const u64 e = vals[s];
                    keys[s] = -1;
                    vals[s] = 0;
                    eval_loaded(c, e, __ldg(st.S + c), guard_needs_size(m, c) ? __ldg(st.size + c) : 0, m, b);
                    if (ok) nct_add(tb, nlg, c, e, 1u << nlg);
                }
                __syncwarp();
                if (ok && lane == 0) {
                    t.off[v] = noff;
                    t.lg[v] = (uint8_t)nlg;
                }
            }
            group_reduce_best(m, b, 32);
            if (lane == 0) {
                u64 delta = 0;
                st.newc[v] = move_decision(m, b, &delta);
                delta_acc += delta;
            }
            __syncwarp();
        }
    }
    if (lane == 0 && delta_acc) atomicAdd(dE, delta_acc);
}

// The queued vertices, a CTA each: the row in a shared table of FB_CAP slots.
template <typename WT>
__global__ void __launch_bounds__(FB_THREADS) nct_build_kernel(GraphView<WT> g, StateView st, NctView t,
                                                               Fallback large, int32_t giant_degree, u64 *dE) {
    constexpr int LG = ilog2_c(FB_CAP), OCC_CAP = FB_CAP / 2;
    static_assert(FB_KEYS + FB_THREADS <= OCC_CAP, "a step's claims fit the occupied list");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64 *vals = reinterpret_cast<u64 *>(smem_raw);
    int32_t *keys = reinterpret_cast<int32_t *>(vals + FB_CAP);
    int32_t *occ = keys + FB_CAP;
    __shared__ int32_t nocc, item_sh;
    __shared__ int nlg, ok;
    __shared__ uint32_t noff;
    const int32_t count = t.qctr[0];
    if ((int32_t)blockIdx.x >= count) return;   // at most one CTA per item
    for (int s = threadIdx.x; s < FB_CAP; s += FB_THREADS) { keys[s] = -1; vals[s] = 0; }
    if (threadIdx.x == 0) nocc = 0;
    __syncthreads();
    u64 delta_acc = 0;
    for (;;) {
        if (threadIdx.x == 0) item_sh = atomicAdd(t.qctr + 1, 1);
        __syncthreads();
        const int32_t item = item_sh;
        if (item >= count) break;
        const int32_t v = t.queue[item];
        const int32_t own = __ldg(st.comm + v);
        const int32_t r0 = g.rowptr[v], r1 = g.rowend[v];
        u64 e_own = 0;
        bool over = false;
        for (int32_t b0 = r0; b0 < r1; b0 += FB_THREADS) {
            if (b0 - r0 >= FB_KEYS) {   // fewer entries cannot hold more communities
                __syncthreads();
                const int32_t so_far = nocc;
                __syncthreads();
                over = so_far > FB_KEYS;
                if (over) break;
            }
            const int32_t e = b0 + (int32_t)threadIdx.x;
            if (e >= r1) continue;
            const int32_t j = __ldg(g.col + e);
            if (j == v) continue;
            const int32_t c = __ldg(st.comm + j);
            if (c == own) e_own += gw(g, e);
            else table_insert_occ_capped(keys, vals, LG, c, gw(g, e), st.err, occ, &nocc, OCC_CAP);
        }
        __syncthreads();
        const int32_t nd = min(nocc, OCC_CAP);
        if (nd > FB_KEYS) over = true;
        if (over) {
            for (int32_t i = threadIdx.x; i < nd; i += FB_THREADS) {
                keys[occ[i]] = -1;
                vals[occ[i]] = 0;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                nocc = 0;
                t.lg[v] = NCT_NEVER;
                atomicAdd(t.cursor + 1, 1ull);   // vertices without tables
                if (r1 - r0 <= giant_degree) enqueue_large(large, v, r1 - r0, st.err);
            }
            __syncthreads();
            continue;
        }
        if (threadIdx.x == 0) ok = nct_alloc(t, nd + 1, &nlg, &noff) ? 1 : 0;
        __syncthreads();
        const int have = ok, lg = nlg;
        GSlot *tb = t.slots + noff;
        if (have) {
            for (int s = threadIdx.x; s < (1 << lg); s += FB_THREADS)
                *reinterpret_cast<uint4 *>(tb + s) = make_uint4(0, 0, 0, 0);
            __syncthreads();
        }
        const MoveCtx m = move_ctx(own, __ldg(st.size + own) == 1, st.T, __ldg(st.k + v), __ldg(st.S + own));
        Best b = best_init(own);
        b.eo = e_own;
        for (int32_t i = threadIdx.x; i < nd; i += FB_THREADS) {
            const int32_t sl = occ[i];
            const int32_t c = keys[sl];
            const u64 e = vals[sl];
            keys[sl] = -1;
            vals[sl] = 0;
            eval_loaded(c, e, __ldg(st.S + c), guard_needs_size(m, c) ? __ldg(st.size + c) : 0, m, b);
            if (have) nct_add(tb, lg, c, e, 1u << lg);
        }
        cta_reduce_best<FB_THREADS>(m, b);
        if (threadIdx.x == 0) {
            u64 delta = 0;
            st.newc[v] = move_decision(m, b, &delta);
            delta_acc += delta;
            nocc = 0;
            if (have) {
                if (b.eo) nct_add(tb, lg, own, b.eo, 1u << lg);
                t.off[v] = noff;
                t.lg[v] = (uint8_t)lg;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && delta_acc) atomicAdd(dE, delta_acc);
}
