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

// Eight lanes per vertex: k_v (row weight) and the weight to the own community;
// Sigma_tot[C(v)] += k_v, T = sum of k.  Community ids outside [0, V) set error
// bit 4.  The grid comes from the scan words, and nothing is read beyond the
// offsets when the scan rejected the CSR.  Each CTA takes a contiguous range of
// vertices and sums Sigma_tot in a shared table first: an atomic per vertex on
// the few cache lines of 256 communities took 46 us on 200,003 vertices of
// about 18 entries, whatever the lanes per vertex; the table takes 18 us (29
// MB read), now bound by the column -> community gathers.
constexpr int NA_LG = 10, NA_SLOTS = 1 << NA_LG, NA_PROBES = 8;
__global__ void __launch_bounds__(256) noalloc_modularity_kernel(const int32_t *__restrict__ rowptr,
                                                               const int32_t *__restrict__ col,
                                                               const float *__restrict__ w,
                                                               const int32_t *__restrict__ comm,
                                                               int32_t V, int64_t E, u64 *S,
                                                               NoallocHeader *hdr) {
    __shared__ u64 part[8], tpart[8], vals[NA_SLOTS];
    __shared__ int32_t keys[NA_SLOTS];
    constexpr int U = 4;
    for (int i = threadIdx.x; i < NA_SLOTS; i += 256) {
        keys[i] = -1;
        vals[i] = 0;
    }
    __syncthreads();
    const int sc = scale_of_scan(hdr->scan, E);
    if ((hdr->err & 3) || hdr->scan[2] || sc < 0) return;
    const double scale = ldexp(1.0, sc);
    const int lane = threadIdx.x & 31, gl = lane & 7;
    u64 own_sum = 0, t_sum = 0;
    const int32_t chunk = (V + (int32_t)gridDim.x - 1) / (int32_t)gridDim.x;
    const int32_t lo = min((int64_t)V, (int64_t)blockIdx.x * chunk), hi = min((int64_t)V, (int64_t)lo + chunk);
    for (int32_t v0 = lo + (int32_t)(threadIdx.x >> 5) * 4; v0 < hi; v0 += 32) {
        const int32_t v = v0 + (lane >> 3);
        int32_t cv = -1, r0 = 0, r1 = 0;
        if (v < hi) {
            cv = comm[v];
            r0 = rowptr[v];
            r1 = rowptr[v + 1];
            if (cv < 0 || cv >= V) {
                if (gl == 0) atomicOr(&hdr->err, 4);
                r1 = r0;
                cv = -1;
            }
        }
        u64 k = 0, eo = 0;
        for (int32_t e0 = r0 + gl; e0 < r1; e0 += 8 * U) {
            int32_t jj[U];
            u64 xx[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int32_t e = e0 + 8 * u;
                jj[u] = -1;
                xx[u] = 0;
                if (e < r1) {
                    jj[u] = __ldg(col + e);
                    xx[u] = wfix(w, e, scale);
                }
            }
            int32_t cc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) cc[u] = jj[u] >= 0 ? __ldg(comm + jj[u]) : -2;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                k += xx[u];
                if (cc[u] == cv) eo += xx[u];
            }
        }
        t_sum += k;
        own_sum += eo;
        for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(FULL, k, off);
        if (gl == 0 && k) {
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
        noalloc_modularity_kernel<<<noalloc_grid(V, 128), 256, 0, s>>>(d_rowptr, d_col, d_w, d_comm, V, E, S, dh);
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
