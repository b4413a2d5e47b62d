// lv_mem.h -- device memory and streams shared by the library's objects
// (lv_mem.cu).  Host code only.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>

#include <vector>

namespace lv {

constexpr size_t LARGE_BYTES = size_t(1) << 20;   // smaller buffers come from slabs
constexpr size_t SLAB_BYTES = size_t(4) << 20;
struct MemBlock {
    void *p = nullptr;
    size_t bytes = 0;
};
// A block of at least `bytes`, usable on stream s at once.
cudaError_t mem_take(int dev, size_t bytes, cudaStream_t s, MemBlock *out);
// Back, for the next owner: no queued work uses it any more (s: for frees).
void mem_give(int dev, const MemBlock &b, cudaStream_t s);
cudaError_t mem_trim(int dev);
bool mem_pooled(int dev);   // the device has a stream-ordered pool
size_t mem_total(int dev);  // bytes of the current device dev; 0: unknown
// The buffers of one owner.
struct MemSet {
    int dev = 0;
    std::vector<MemBlock> blocks, slabs;
    unsigned char *slab = nullptr;
    size_t slab_at = 0, slab_end = 0;
    int fail_at = 0;   // test hook: the fail_at-th alloc from now on fails (0: none)
    cudaError_t alloc(void **p, size_t bytes, cudaStream_t s);
    cudaError_t alloc_own(void **p, size_t bytes, cudaStream_t s);   // a block of its own
    // Gives p back once the work queued on s is done, which it waits for (a
    // slab's part stays with the owner).
    void free(void *p, cudaStream_t s);
    // Gives everything back: the owner's queued work is done.
    void give_all(cudaStream_t s);
    // p (from alloc_own) now belongs to the library's caller, until
    // mem_take_back.
    void hand_over(void *p);
};
bool mem_take_back(void *p);   // false: not handed over by hand_over
cudaError_t stream_take(int dev, cudaStream_t *s);
void stream_give(int dev, cudaStream_t s);

}  // namespace lv
