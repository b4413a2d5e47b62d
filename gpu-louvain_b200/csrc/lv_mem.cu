// lv_mem.cu -- device memory and streams of the library's objects.
//
// Handles, batches and the CSR builders ask for dozens of buffers, 55 GB in all
// for an R-MAT-24 run, and a program that runs one graph after another asks
// for nearly the same sizes again.  Mapping that memory anew cost 150 of 370
// ms of such a run when each graph's entry count differed a little from the
// last one's (the earlier cache matched exact sizes only), and cudaMalloc 15
// of 36 ms of building and running an R-MAT-18 graph.  So:
//   - blocks of LARGE bytes and more are rounded up to eighths of a power of
//     two and, when their owner has drained its work, kept per device for the
//     next request of about that size (at most 1/4 larger than asked for);
//   - smaller buffers are cut from 4 MB slabs, which are such blocks;
//   - streams are kept likewise, a few per device.
// Blocks in use and kept together never exceed the largest amount that was in
// use at one time by more than an eighth (blocks outgrown during a run, and
// those of a small graph between two large ones, find room there); beyond that
// the oldest go back to the stream-ordered pool they come from.  A buffer that
// a run outgrows is kept too: given to the pool, it was asked of the pool again
// by the next run, which now and then mapped it anew (the first four of twelve
// like runs of R-MAT-24 from host arrays took 753, 451, 345 and 323 ms; now
// 691, 325, 323 and 322).
// lv_trim_device_memory returns everything unused to the system.  All of it is
// safe with several threads: a block belongs to one owner from take to give,
// and is given only when no queued work uses it.
#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "lv_mem.h"

namespace lv {
namespace {

constexpr int MAX_DEVICES = 64;
constexpr size_t MAX_STREAMS = 16;

struct DeviceMemory {
    cudaMemPool_t pool = nullptr;
    std::vector<MemBlock> kept;      // oldest first
    size_t kept_bytes = 0, live_bytes = 0, peak_bytes = 0, total_bytes = 0;
    std::vector<cudaStream_t> streams;
};

std::mutex g_mu;
DeviceMemory g_dev[MAX_DEVICES];

// blocks handed to the caller of the library (lv_free_device)
struct Handed { int dev; MemBlock b; };
std::unordered_map<void *, Handed> g_handed;

// The device's pool, whose release threshold keeps freed memory mapped.  Under
// g_mu.
cudaMemPool_t pool_of(int dev) {
    DeviceMemory &d = g_dev[dev];
    if (!d.pool) {
        // an error left pending by an earlier asynchronous call would be
        // reported by the calls below; set-up is retried by the next
        // allocation if it fails
        cudaGetLastError();
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        uint64_t keep = UINT64_MAX;
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        d.pool = pool;
    }
    return d.pool;
}

// Takes the oldest blocks off the list until what is kept fits beside `live`
// bytes in use.  Under g_mu.
void evict(DeviceMemory &d, size_t live, std::vector<MemBlock> *out) {
    const size_t most = std::max(d.peak_bytes, live), limit = most + most / 8;
    size_t n = 0;
    while (n < d.kept.size() && live + d.kept_bytes > limit) {
        out->push_back(d.kept[n]);
        d.kept_bytes -= d.kept[n].bytes;
        ++n;
    }
    d.kept.erase(d.kept.begin(), d.kept.begin() + (long)n);
}

size_t rounded(size_t bytes) {
    size_t p = LARGE_BYTES;
    while (p * 2 <= bytes) p *= 2;
    const size_t step = p / 8;
    return (bytes + step - 1) / step * step;
}

void free_raw(cudaMemPool_t pool, void *p, cudaStream_t s) {
    if (pool) cudaFreeAsync(p, s);
    else cudaFree(p);
}

cudaError_t alloc_raw(cudaMemPool_t pool, void **p, size_t bytes, cudaStream_t s) {
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMalloc(p, bytes);
}

}  // namespace

cudaError_t mem_take(int dev, size_t bytes, cudaStream_t s, MemBlock *out) {
    out->p = nullptr;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    const size_t want = rounded(bytes);
    std::vector<MemBlock> old;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        DeviceMemory &d = g_dev[dev];
        size_t best = d.kept.size();
        for (size_t i = 0; i < d.kept.size(); ++i)
            if (d.kept[i].bytes >= bytes && d.kept[i].bytes <= want + want / 4 &&
                (best == d.kept.size() || d.kept[i].bytes < d.kept[best].bytes))
                best = i;
        if (best < d.kept.size()) {
            *out = d.kept[best];
            d.kept.erase(d.kept.begin() + (long)best);
            d.kept_bytes -= out->bytes;
            d.live_bytes += out->bytes;
            return cudaSuccess;
        }
        pool = pool_of(dev);
        evict(d, d.live_bytes + want, &old);
    }
    for (const MemBlock &b : old) free_raw(pool, b.p, s);
    out->bytes = want;
    cudaError_t e = alloc_raw(pool, &out->p, want, s);
    if (e != cudaSuccess) {
        // everything kept goes back first, and the pool gives up what it holds
        // unused; then the size asked for has to do
        cudaGetLastError();
        std::vector<MemBlock> kept;
        {
            std::lock_guard<std::mutex> lock(g_mu);
            kept.swap(g_dev[dev].kept);
            g_dev[dev].kept_bytes = 0;
        }
        for (const MemBlock &b : kept) free_raw(pool, b.p, s);
        cudaStreamSynchronize(s);
        if (pool) cudaMemPoolTrimTo(pool, 0);
        cudaGetLastError();
        e = alloc_raw(pool, &out->p, want, s);
        if (e != cudaSuccess && bytes < want) {
            cudaGetLastError();
            out->bytes = bytes;
            e = alloc_raw(pool, &out->p, bytes, s);
        }
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        out->p = nullptr;
        return e;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    DeviceMemory &d = g_dev[dev];
    d.live_bytes += out->bytes;
    d.peak_bytes = std::max(d.peak_bytes, d.live_bytes);
    return cudaSuccess;
}

void mem_give(int dev, const MemBlock &b, cudaStream_t s) {
    if (!b.p) return;
    std::vector<MemBlock> old;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        DeviceMemory &d = g_dev[dev];
        d.live_bytes -= b.bytes;
        d.kept.push_back(b);
        d.kept_bytes += b.bytes;
        evict(d, d.live_bytes, &old);
        pool = d.pool;
    }
    for (const MemBlock &x : old) free_raw(pool, x.p, s);
}

cudaError_t mem_trim(int dev) {
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    std::vector<MemBlock> kept;
    std::vector<cudaStream_t> streams;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        DeviceMemory &d = g_dev[dev];
        kept.swap(d.kept);
        streams.swap(d.streams);
        d.kept_bytes = 0;
        d.peak_bytes = d.live_bytes;
        pool = d.pool;
    }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(dev);
    for (const MemBlock &b : kept) free_raw(pool, b.p, 0);
    for (cudaStream_t s : streams) cudaStreamDestroy(s);
    cudaDeviceSynchronize();
    cudaSetDevice(prev);
    return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

bool mem_pooled(int dev) {
    std::lock_guard<std::mutex> lock(g_mu);
    return dev >= 0 && dev < MAX_DEVICES && pool_of(dev) != nullptr;
}

size_t mem_total(int dev) {
    if (dev < 0 || dev >= MAX_DEVICES) return 0;
    std::lock_guard<std::mutex> lock(g_mu);
    size_t avail = 0, &total = g_dev[dev].total_bytes;
    // asked once: the call takes tens of milliseconds at times
    if (!total && cudaMemGetInfo(&avail, &total) != cudaSuccess) {
        cudaGetLastError();
        total = 0;
    }
    return total;
}

cudaError_t MemSet::alloc(void **p, size_t bytes, cudaStream_t s) {
    *p = nullptr;
    if (fail_at > 0 && --fail_at == 0) return cudaErrorMemoryAllocation;
    if (bytes == 0) bytes = 1;
    if (bytes < LARGE_BYTES) {
        const size_t at = (slab_at + 255) / 256 * 256;
        if (slab && at + bytes <= slab_end) {
            *p = slab + at;
            slab_at = at + bytes;
            return cudaSuccess;
        }
        MemBlock b;
        const cudaError_t e = mem_take(dev, SLAB_BYTES, s, &b);
        if (e != cudaSuccess) return e;
        slabs.push_back(b);
        slab = (unsigned char *)b.p;
        slab_at = bytes;
        slab_end = b.bytes;
        *p = slab;
        return cudaSuccess;
    }
    return alloc_own(p, bytes, s);
}

cudaError_t MemSet::alloc_own(void **p, size_t bytes, cudaStream_t s) {
    MemBlock b;
    const cudaError_t e = mem_take(dev, bytes ? bytes : 1, s, &b);
    *p = b.p;
    if (e != cudaSuccess) return e;
    blocks.push_back(b);
    return cudaSuccess;
}

void MemSet::free(void *p, cudaStream_t s) {
    for (size_t i = 0; i < blocks.size(); ++i)
        if (blocks[i].p == p) {
            cudaStreamSynchronize(s);
            mem_give(dev, blocks[i], s);
            blocks[i] = blocks.back();
            blocks.pop_back();
            return;
        }
}

void MemSet::give_all(cudaStream_t s) {
    for (const MemBlock &b : blocks) mem_give(dev, b, s);
    for (const MemBlock &b : slabs) mem_give(dev, b, s);
    blocks.clear();
    slabs.clear();
    slab = nullptr;
}

void MemSet::hand_over(void *p) {
    for (size_t i = 0; i < blocks.size(); ++i)
        if (blocks[i].p == p) {
            std::lock_guard<std::mutex> lock(g_mu);
            g_handed[p] = Handed{dev, blocks[i]};
            blocks[i] = blocks.back();
            blocks.pop_back();
            return;
        }
}

bool mem_take_back(void *p) {
    Handed h;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        auto it = g_handed.find(p);
        if (it == g_handed.end()) return false;
        h = it->second;
        g_handed.erase(it);
    }
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(h.dev);
    cudaDeviceSynchronize();   // the caller's own work on the array, as cudaFree waits for it
    mem_give(h.dev, h.b, 0);
    cudaSetDevice(prev);
    return true;
}

cudaError_t stream_take(int dev, cudaStream_t *s) {
    *s = nullptr;
    if (dev >= 0 && dev < MAX_DEVICES) {
        std::lock_guard<std::mutex> lock(g_mu);
        auto &v = g_dev[dev].streams;
        if (!v.empty()) {
            *s = v.back();
            v.pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
}

void stream_give(int dev, cudaStream_t s) {
    if (!s) return;
    if (cudaStreamSynchronize(s) == cudaSuccess && dev >= 0 && dev < MAX_DEVICES) {
        std::lock_guard<std::mutex> lock(g_mu);
        auto &v = g_dev[dev].streams;
        if (v.size() < MAX_STREAMS) {
            v.push_back(s);
            return;
        }
    }
    cudaStreamDestroy(s);
}

}  // namespace lv
