// Shared host-side helpers: per-thread error state and RAII device memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <string>

// Register budget of the step kernels: blocks of at most WK_FAST_MAX_THREADS threads, at least that many of them
// resident per SM. Two nodes per thread: 64 x 8 gives D3Q19 / D3Q27 128 registers (16 warps per SM), which their 38 / 54
// loads in flight need without spills. Sphere channel FP32 256x128x128, 160^3, 48^3: 110, 112, 5.6 us a step; at
// 96 registers (20 warps) 117, 117, 5.9. D2Q9 carries half the values: 64 registers and 32 warps (2048x1024:
// 22.0 us, 25.2 with 96 registers); 72 where a batch's arguments have to be read (512 channels FP32 / FP16, 32 threads: 413 /
// 345 us a step, 431 / 375 with 80 registers, 418 / 342 with 64; 60 channels 50.9 / 39.7, 52.5 / 41.7, 51.8 / 41.3).
// The FP32 D3Q27 MRT takes 168 with Smagorinsky's tau and in a batch: with 128 it spills 2.2 KB a thread (256^3 box with
// Smagorinsky 664 us a step, 920 with 128; batch of two 160^3 boxes 345, 473).
#ifndef WK_PAIRS27_MIN_BLOCKS
#define WK_PAIRS27_MIN_BLOCKS 5
#endif
#ifndef WK_FAST_MAX_THREADS
#define WK_FAST_MAX_THREADS 64
#endif
#ifndef WK_PAIRS_MIN_BLOCKS
#define WK_PAIRS_MIN_BLOCKS 8
#endif
#ifndef WK_PAIRS9_MIN_BLOCKS
#define WK_PAIRS9_MIN_BLOCKS 16
#endif
#ifndef WK_PAIRS9_BATCH_MIN_BLOCKS
#define WK_PAIRS9_BATCH_MIN_BLOCKS 14
#endif

namespace wk {

int set_error(int code, const std::string& msg);
void clear_error();

// Return with a failed call's error, and take it from the runtime: the check of the next launch would report it again.
#define WK_CUDA(call)                                                                                      \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) {                                                                           \
            (void)cudaGetLastError();                                                                      \
            return ::wk::set_error(-2, std::string(#call) + ": " + cudaGetErrorString(e_));                \
        }                                                                                                  \
    } while (0)

// Device blocks are taken from, and may be handed back to, a process-wide cache
// (alloc_cache.cpp). cudaFree synchronises the whole device, so an object whose
// work is known to be finished (its stream synchronised) returns its blocks with
// release() instead: a serving loop can then retire jobs and start new ones while
// other streams keep running, and a new lattice reuses the retired one's memory
// without a cudaMalloc. reset() keeps the synchronous cudaFree for blocks whose
// last use is not known to have finished.
cudaError_t cache_alloc(void** p, std::size_t bytes, std::size_t* block_bytes);
void cache_release(void* p, std::size_t block_bytes);
std::size_t cache_trim();         // cudaFree every cached block of the current device; bytes freed
std::size_t cache_held_bytes();   // bytes held by the cache on the current device

// Device allocation owned by one object. Nothing is allocated until ensure().
struct DevMem {
    void* p = nullptr;
    std::size_t bytes = 0;
    DevMem() = default;
    DevMem(const DevMem&) = delete;
    DevMem& operator=(const DevMem&) = delete;
    ~DevMem() { reset(); }
    void reset() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    // Hand the block to the cache; only when no queued work can still touch it.
    void release() {
        if (p) cache_release(p, bytes);
        p = nullptr;
        bytes = 0;
    }
    // Grow to at least b bytes when no queued work can still use the current block: the old
    // block goes back to the cache instead of a cudaFree (which would wait for the whole device).
    cudaError_t grow(std::size_t b) {
        if (p && bytes >= b) return cudaSuccess;
        release();
        return ensure(b);
    }
    // (Re)allocate when the current block is smaller than b. Returns cudaSuccess or the error.
    cudaError_t ensure(std::size_t b) {
        if (p && bytes >= b) return cudaSuccess;
        reset();
        if (b == 0) return cudaSuccess;
        cudaError_t e = cache_alloc(&p, b, &bytes);
        if (e != cudaSuccess) {
            p = nullptr;
            bytes = 0;
            (void)cudaGetLastError();
            return e;
        }
        return cudaSuccess;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

}  // namespace wk
