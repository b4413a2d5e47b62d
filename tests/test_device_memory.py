"""The cache of device blocks (lv_mem.cu) on the host, with a fake of the CUDA
allocation calls that knows how much a device holds: what is kept, what goes
back, what happens when the device is full, and several threads at once."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR

SHIM = r"""
#include "lv_mem.cu"
#include <map>
#include <thread>

// ---- the fake: `room` bytes per device, every block accounted for ----
namespace {
std::mutex f_mu;
std::map<void *, size_t> f_live;
size_t f_room, f_used, f_next = 1;
long f_allocs, f_bad, f_syncs;
}
extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++f_syncs; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)0x10; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = (cudaMemPool_t)0x20; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> lock(f_mu);
    ++f_allocs;
    if (f_used + n > f_room) return cudaErrorMemoryAllocation;
    f_used += n;
    *p = (void *)(f_next++ << 20);
    f_live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> lock(f_mu);
    auto it = f_live.find(p);
    if (it == f_live.end()) { ++f_bad; return cudaErrorInvalidValue; }
    f_used -= it->second;
    f_live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t *a, size_t *t) { *t = f_room; *a = f_room - f_used; return cudaSuccess; }

void fake_room(size_t n) { f_room = n; }
size_t fake_used() { return f_used; }
long fake_allocs() { return f_allocs; }
long fake_bad() { return f_bad; }
void trim() { lv::mem_trim(0); }
size_t most() { return lv::g_dev[0].peak_bytes; }
size_t in_use() { return lv::g_dev[0].live_bytes; }
size_t kept() { return lv::g_dev[0].kept_bytes; }

lv::MemSet *set_new() { return new lv::MemSet(); }
void *set_alloc(lv::MemSet *m, size_t n) { void *p; return m->alloc(&p, n, 0) == cudaSuccess ? p : nullptr; }
void set_free(lv::MemSet *m, void *p) { m->free(p, 0); }
void set_done(lv::MemSet *m) { m->give_all(0); delete m; }

// Threads that take and give blocks of mixed sizes; a block that two of them
// hold at once is counted.
long threads(int n, int rounds) {
    std::mutex mu;
    std::map<void *, int> owner;
    long twice = 0;
    std::vector<std::thread> ts;
    for (int t = 0; t < n; ++t)
        ts.emplace_back([&, t] {
            uint64_t x = 88172645463325252ull + (uint64_t)t;
            for (int r = 0; r < rounds; ++r) {
                lv::MemSet m;
                std::vector<void *> mine;
                for (int i = 0; i < 12; ++i) {
                    x ^= x << 13, x ^= x >> 7, x ^= x << 17;
                    void *p = nullptr;
                    if (m.alloc_own(&p, (size_t)1 << (18 + x % 9), 0) != cudaSuccess) continue;
                    {
                        std::lock_guard<std::mutex> lock(mu);
                        if (owner[p]++) ++twice;
                        mine.push_back(p);
                    }
                    if (x % 5 == 0) {
                        {
                            std::lock_guard<std::mutex> lock(mu);
                            --owner[mine.back()];
                        }
                        m.free(mine.back(), 0);
                        mine.pop_back();
                    }
                }
                {
                    std::lock_guard<std::mutex> lock(mu);
                    for (void *p : mine) --owner[p];
                }
                m.give_all(0);
            }
        });
    for (auto &t : ts) t.join();
    return twice;
}
}
"""

MB = 1 << 20
GB = 1 << 30


@pytest.fixture()
def mem(tmp_path):
    (tmp_path / "shim.cpp").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    nvcc = subprocess.run(["which", "nvcc"], capture_output=True, text=True).stdout.strip()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc))) if nvcc else "/usr/local/cuda"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread",
                    "-Wl,-Bsymbolic", "-I", os.path.join(cuda, "include"),
                    "-I", os.path.join(PKG_DIR, "csrc"), str(tmp_path / "shim.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    for n in ("fake_used", "most", "in_use", "kept"):
        getattr(L, n).restype = C.c_size_t
    for n in ("fake_allocs", "fake_bad", "threads"):
        getattr(L, n).restype = C.c_long
    L.fake_room.argtypes = [C.c_size_t]
    L.set_new.restype = C.c_void_p
    L.set_alloc.restype = C.c_void_p
    L.set_alloc.argtypes = [C.c_void_p, C.c_size_t]
    L.set_free.argtypes = [C.c_void_p, C.c_void_p]
    L.set_done.argtypes = [C.c_void_p]
    L.fake_room(1 << 50)
    return L


def _bound(L):
    assert L.fake_used() == L.in_use() + L.kept()
    assert L.fake_used() <= L.most() + L.most() // 8


def _run(L, rng=None):
    """The requests of one run: fixed buffers, staging buffers outgrown once,
    small ones from slabs.  With rng the sizes differ by up to 3 %."""
    at = lambda n: int(n * (1.0 + (rng.uniform(-0.03, 0.03) if rng else 0.0)))
    m = L.set_new()
    for n in (67 * MB, 2083 * MB, 2083 * MB, 67 * MB, 134 * MB, 2000, 300000):
        assert L.set_alloc(m, at(n))
    first = [L.set_alloc(m, at(n)) for n in (319 * MB, 638 * MB)]
    assert all(first)
    assert L.set_alloc(m, at(11629 * MB))
    for p in first:
        L.set_free(m, p)
    for n in (2411 * MB, 4822 * MB, 5 * MB):
        assert L.set_alloc(m, at(n))
        _bound(L)
    L.set_done(m)
    _bound(L)


def test_like_runs_share_their_memory(mem):
    """From the second run on nothing is asked of the pool, outgrown buffers
    included."""
    _run(mem)
    n = mem.fake_allocs()
    for _ in range(5):
        _run(mem)
        assert mem.fake_allocs() == n
    assert mem.in_use() == 0 and mem.fake_bad() == 0


def test_kept_and_live_blocks_stay_within_the_most_in_use(mem):
    rng = np.random.default_rng(7)
    for _ in range(60):
        if rng.random() < 0.3:
            _run(mem, rng)
            continue
        m = mem.set_new()
        for n in np.exp(rng.uniform(np.log(1000), np.log(6e9), 8)).astype(np.int64):
            assert mem.set_alloc(m, int(n))
            _bound(mem)
        mem.set_done(m)
        _bound(mem)
    mem.trim()
    assert mem.fake_used() == 0 and mem.fake_bad() == 0


def test_a_full_device_gives_the_size_asked_for(mem):
    """1,150 MB where a rounded block would take 1,152 MB and 1,100 are idle in
    other sizes: the kept ones go back, and the size asked for has to do."""
    mem.fake_room(1151 * MB)
    m = mem.set_new()
    for _ in range(11):
        assert mem.set_alloc(m, 100 * MB)
    mem.set_done(m)
    assert mem.kept() > 0
    for _ in range(2):   # the second time from the list
        m = mem.set_new()
        assert mem.set_alloc(m, 1150 * MB)
        assert mem.set_alloc(m, 2 * MB) is None
        assert mem.in_use() == 1150 * MB and mem.kept() == 0
        mem.set_done(m)
    mem.trim()
    assert mem.fake_used() == 0 and mem.fake_bad() == 0


def test_threads_never_share_a_block(mem):
    mem.fake_room(700 * MB)   # some requests fail
    assert mem.threads(8, 200) == 0
    assert mem.in_use() == 0 and mem.fake_used() == mem.kept()
    mem.trim()
    assert mem.fake_used() == 0 and mem.fake_bad() == 0
