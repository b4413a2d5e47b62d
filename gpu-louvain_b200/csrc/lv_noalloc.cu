// lv_noalloc.cu -- modularity of a given partition without any device
// allocation (lv_modularity_noalloc).
//
// Some callers cannot allocate device memory at the moment they want a
// modularity value: a process whose device memory is wholly owned by another
// allocator (a framework's caching allocator, or a fixed pool sized to the
// whole GPU), or a latency-critical loop that cannot afford the device-wide
// synchronisation that cudaMalloc / cudaFree imply.  lv_create and
// lv_modularity allocate their working set per handle, so this entry point
// computes the same number with its working memory in one file-scope device
// array instead.
//
// The computation is the engine's modularity reduction (sum_i e_{i->C(i)} over
// the CSR, Sigma_tot per community, sum of Sigma_tot^2) on the same
// fixed-point grid and with the same FP64 formula, so for the same CSR and
// partition it returns exactly what lv_create_device + lv_set_communities +
// lv_modularity return.
#include <cmath>
#include <cstdio>

#include "../../include/louvain_b200.h"
#include "lv_internal.h"

namespace lv {
namespace {

// Working memory shared by every call on a device: a header (the weight
// scan words, error bits and the exact totals) followed by Sigma_tot of up
// to LV_NOALLOC_MAX_VERTICES communities.  Every GPU that loads the library
// holds it until the process exits.
struct NoallocHeader {
    int32_t scan[4];   // max fractional bits, top exponent + 1024, bad-weight flag, unused
    int32_t err;       // CSR check bits (1, 2) and community-id check bit (4)
    int32_t pad;
    u64 T;             // total weight on the fixed grid
    u64 e_own;         // sum_i e_{i->C(i)}
    u64 s2[2];         // hi, lo of sum_C Sigma_tot^2
};
constexpr int NOALLOC_HEADER_BYTES = 256;
static_assert(sizeof(NoallocHeader) <= NOALLOC_HEADER_BYTES, "header fits its slot");
constexpr size_t NOALLOC_BYTES = NOALLOC_HEADER_BYTES + sizeof(u64) * (size_t)LV_NOALLOC_MAX_VERTICES;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

// k_v (row weight) and the weight to the own community; Sigma_tot[C(v)] += k_v,
// T = sum of k.  Community ids outside [0, V) set error bit 4.  The grid comes
// from the scan words, and nothing is read beyond the offsets when the scan
// rejected the CSR.
//
// Every warp takes the same number of items, an item being an entry or a
// vertex: row v owns the items rowptr[v] + v .. rowptr[v + 1] + v, so a warp
// finds its first row by a search and a long row is shared by many warps (all
// sums are exact, whoever adds them).  Four rows at a time take eight lanes
// each; a part of a row longer than NA_LONG takes the warp.  With equal vertex
// ranges per CTA and eight lanes for any row, a call on an R-MAT-20 graph took
// 15.1 ms, its hubs being left to few lanes; now 0.79 ms.  Sigma_tot is summed
// in a shared table per CTA first: an atomic per vertex on the few cache lines
// of 256 communities took 46 us on 200,003 vertices of about 18 entries,
// whatever the lanes per vertex; with the table that graph takes 22 us (29 MB
// read; 18 us in equal vertex ranges: the search takes 2 us, the rows cut at
// the warps' ends most of the rest), bound by the column -> community gathers.
constexpr int NA_LG = 10, NA_SLOTS = 1 << NA_LG, NA_PROBES = 8;
constexpr int NA_U = 4, NA_LONG = 8 * NA_U * 4;

// Adds up the entries [e0, e1) of a row, lanes `stride` apart: all weights to
// k, those within community cv to eo.
__device__ __forceinline__ void noalloc_entries(const int32_t *__restrict__ col, const float *__restrict__ w,
                                                const int32_t *__restrict__ comm, double scale, int32_t cv,
                                                uint32_t e0, uint32_t e1, uint32_t stride, u64 &k, u64 &eo) {
    for (; e0 < e1; e0 += stride * NA_U) {
        int32_t jj[NA_U];
        u64 xx[NA_U];
#pragma unroll
        for (int u = 0; u < NA_U; ++u) {
            const uint32_t e = e0 + stride * u;
            jj[u] = -1;
            xx[u] = 0;
            if (e < e1) {
                jj[u] = __ldg(col + e);
                xx[u] = wfix(w, e, scale);
            }
        }
        int32_t cc[NA_U];
#pragma unroll
        for (int u = 0; u < NA_U; ++u) cc[u] = jj[u] >= 0 ? __ldg(comm + jj[u]) : -2;
#pragma unroll
        for (int u = 0; u < NA_U; ++u) {
            k += xx[u];
            if (cc[u] == cv) eo += xx[u];
        }
    }
}

__device__ __forceinline__ void noalloc_add(int32_t *keys, u64 *vals, u64 *S, int32_t cv, u64 k) {
    uint32_t sl = hash_slot(cv, NA_LG);
    bool in = false;
    for (int p = 0; p < NA_PROBES && !in; ++p) {
        const int32_t prev = atomicCAS(keys + sl, -1, cv);
        in = prev < 0 || prev == cv;
        if (!in) sl = (sl + 1) & (NA_SLOTS - 1);
    }
    if (in) table_add(vals + sl, k);
    else atomicAdd(S + cv, k);
}

__global__ void __launch_bounds__(256) noalloc_modularity_kernel(const int32_t *__restrict__ rowptr,
                                                               const int32_t *__restrict__ col,
                                                               const float *__restrict__ w,
                                                               const int32_t *__restrict__ community,
                                                               int32_t V, int64_t E, u64 *S,
                                                               NoallocHeader *hdr) {
    __shared__ u64 part[8], tpart[8], vals[NA_SLOTS];
    __shared__ int32_t keys[NA_SLOTS];
    for (int i = threadIdx.x; i < NA_SLOTS; i += 256) {
        keys[i] = -1;
        vals[i] = 0;
    }
    const int lane = threadIdx.x & 31, gl = lane & 7;
    // the warp's items [d0, d1)
    const int64_t nw = (int64_t)gridDim.x * 8, wi = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int64_t items = (int64_t)V + E, per = (items + nw - 1) / nw;
    const int64_t d0 = min(items, wi * per), d1 = min(items, d0 + per);
    // the last row whose first item is at or before d0: 128 probes per step
    int32_t lo = 0, hi = V;
    while (hi - lo > 1) {
        const int32_t step = (hi - lo + 127) >> 7;
        int le = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t p = lo + (4 * lane + u) * step;
            le += p < hi && (int64_t)__ldg(rowptr + p) + p <= d0 ? 1 : 0;
        }
        const int q = (int)__reduce_add_sync(FULL, (unsigned)le) - 1;   // the first probe always holds
        lo += max(q, 0) * step;                                         // ... unless the offsets are malformed
        hi = min(lo + step, hi);
    }
    __syncthreads();
    const int sc = scale_of_scan(hdr->scan, E);
    if ((hdr->err & 3) || hdr->scan[2] || sc < 0) return;
    const double scale = ldexp(1.0, sc);
    u64 own_sum = 0, t_sum = 0;
    // a row's header is loaded while the four rows before it are summed
    int32_t nr0 = 0, nr1 = 0, ncv = -1;
    auto header = [&](int32_t v) {
        if (v >= V) return;
        nr0 = __ldg(rowptr + v);
        nr1 = __ldg(rowptr + v + 1);
        ncv = __ldg(community + v);
    };
    header(lo + (lane >> 3));
    for (int32_t v = lo + (lane >> 3); d0 < d1; v += 4) {
        int32_t r0 = nr0, r1 = nr1, cv = ncv;
        bool in = v < V && (int64_t)r0 + v < d1;
        if (!__any_sync(FULL, in)) break;
        header(v + 4);
        if (in && (cv < 0 || cv >= V)) {
            if (gl == 0) atomicOr(&hdr->err, 4);
            in = false;
        }
        r0 = in ? (int32_t)max((int64_t)r0, d0 - v) : 0;
        r1 = in ? (int32_t)min((int64_t)r1, d1 - v) : 0;
        unsigned longs = __ballot_sync(FULL, gl == 0 && r1 - r0 > NA_LONG);
        u64 k = 0, eo = 0;
        if (r1 - r0 <= NA_LONG)
            noalloc_entries(col, w, community, scale, cv, (uint32_t)(r0 + gl), (uint32_t)r1, 8, k, eo);
        t_sum += k;
        own_sum += eo;
        __syncwarp();
        for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(FULL, k, off);
        if (gl == 0 && k) noalloc_add(keys, vals, S, cv, k);
        for (; longs; longs &= longs - 1) {
            const int src = __ffs(longs) - 1;
            const int32_t lc = __shfl_sync(FULL, cv, src);
            const uint32_t l0 = (uint32_t)__shfl_sync(FULL, r0, src), l1 = (uint32_t)__shfl_sync(FULL, r1, src);
            u64 lk = 0, le = 0;
            noalloc_entries(col, w, community, scale, lc, l0 + lane, l1, 32, lk, le);
            t_sum += lk;
            own_sum += le;
            __syncwarp();
            lk = warp_sum_u64(lk);
            if (lane == 0 && lk) noalloc_add(keys, vals, S, lc, lk);
        }
    }
    own_sum = warp_sum_u64(own_sum);
    t_sum = warp_sum_u64(t_sum);
    if (lane == 0) {
        part[threadIdx.x >> 5] = own_sum;
        tpart[threadIdx.x >> 5] = t_sum;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NA_SLOTS; i += 256)
        if (keys[i] >= 0) atomicAdd(S + keys[i], vals[i]);
    if (threadIdx.x == 0) {
        u64 y = 0, z = 0;
        for (int i = 0; i < 8; ++i) {
            y += part[i];
            z += tpart[i];
        }
        if (y) atomicAdd(&hdr->e_own, y);
        if (z) atomicAdd(&hdr->T, z);
    }
}

inline unsigned noalloc_grid(int64_t items, int per_block) {
    const int64_t b = (items + per_block - 1) / per_block;
    return (unsigned)(b < 1 ? 1 : (b > 148 * 4 ? 148 * 4 : b));
}

int noalloc_fail(char *err, int32_t err_len, int code, const char *msg) {
    if (err && err_len > 0) std::snprintf(err, (size_t)err_len, "%s", msg);
    return code;
}

// Device address of the scratch array on the current device.  The host-side
// name of the array is not a device address, so every call asks the runtime
// for it (a cheap lookup) instead of keeping it: an address kept across calls
// would dangle after the caller resets the device (cudaDeviceReset reloads the
// module, possibly elsewhere).
int noalloc_scratch(void **out, char *err, int32_t err_len) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return noalloc_fail(err, err_len, LV_ERR_CUDA, "cudaGetSymbolAddress of the scratch array failed");
    }
    *out = p;
    return LV_OK;
}

int noalloc_read(cudaStream_t s, void *dev_hdr, NoallocHeader *h, char *err, int32_t err_len) {
    cudaError_t e = cudaMemcpyAsync(h, dev_hdr, sizeof(NoallocHeader), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        if (err && err_len > 0) std::snprintf(err, (size_t)err_len, "CUDA error: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return LV_ERR_CUDA;
    }
    return LV_OK;
}

}  // namespace
}  // namespace lv

using namespace lv;

extern "C" int lv_modularity_noalloc(const int32_t *d_rowptr, const int32_t *d_col, const float *d_w,
                                     int32_t V, int64_t E, const int32_t *d_comm, void *stream,
                                     double *q, char *err, int32_t err_len) {
    if (err && err_len > 0) err[0] = '\0';
    if (!q || V < 0 || E < 0 || (V > 0 && (!d_rowptr || !d_comm)) || (E > 0 && (!d_col || !d_w)))
        return noalloc_fail(err, err_len, LV_ERR_INVALID, "invalid argument");
    // a CSR without vertices has no entries (lv_create_device rejects it too)
    if (V == 0 && E > 0) return noalloc_fail(err, err_len, LV_ERR_INVALID, "malformed CSR: entries without vertices");
    if (V > LV_NOALLOC_MAX_VERTICES) {
        char msg[160];
        std::snprintf(msg, sizeof msg,
                      "V = %d exceeds LV_NOALLOC_MAX_VERTICES = %d (the size of the built-in scratch array)",
                      V, LV_NOALLOC_MAX_VERTICES);
        return noalloc_fail(err, err_len, LV_ERR_TOO_LARGE, msg);
    }
    if (E > 0x7fffffffLL) return noalloc_fail(err, err_len, LV_ERR_TOO_LARGE, "E exceeds 2^31 - 1");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return noalloc_fail(err, err_len, LV_ERR_NO_DEVICE, "no usable CUDA device");
    }
    void *base = nullptr;
    int rc = noalloc_scratch(&base, err, err_len);
    if (rc != LV_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    NoallocHeader *dh = (NoallocHeader *)base;
    u64 *S = (u64 *)((unsigned char *)base + NOALLOC_HEADER_BYTES);
    // the array keeps the previous call's contents: the header is cleared here,
    // Sigma_tot[0, V) by the scan
    cudaError_t ce = cudaMemsetAsync(dh, 0, NOALLOC_HEADER_BYTES, s);
    if (ce != cudaSuccess) {
        if (err && err_len > 0) std::snprintf(err, (size_t)err_len, "CUDA error: %s", cudaGetErrorString(ce));
        cudaGetLastError();
        return LV_ERR_CUDA;
    }
    if (V > 0) {
        launch_csr_scan(d_rowptr, d_col, d_w, V, E, &dh->err, dh->scan, S, V, s);
        noalloc_modularity_kernel<<<noalloc_grid((int64_t)V + E, 1024), 256, 0, s>>>(d_rowptr, d_col, d_w, d_comm, V, E,
                                                                                    S, dh);
        note_launches(1);
        launch_s2(S, V, dh->s2, s);
    }
    NoallocHeader h;
    rc = noalloc_read(s, dh, &h, err, err_len);
    if (rc != LV_OK) return rc;
    if (h.err & 3) return noalloc_fail(err, err_len, LV_ERR_INVALID, "malformed CSR (offsets or column ids)");
    if (h.scan[2]) return noalloc_fail(err, err_len, LV_ERR_WEIGHT, "negative, NaN or infinite edge weight");
    // fixed-point scale: the rule of lv_create / lv_create_device
    if (scale_of_scan(h.scan, E) < 0)
        return noalloc_fail(err, err_len, LV_ERR_TOO_LARGE, "total edge weight exceeds the fixed-point range");
    if (h.err) return noalloc_fail(err, err_len, LV_ERR_INVALID, "community id outside [0, V)");
    // the FP64 formula of lv_modularity: e_own / T - sum(S^2) / T^2
    const u128 s2 = ((u128)h.s2[0] << 64) | (u128)h.s2[1];
    const double td = (double)h.T;
    const double a = (double)h.e_own / td;
    const double b = (double)s2 / (td * td);
    *q = a - b;
    return LV_OK;
}
