// launch.cuh -- host helpers of the launches, shared by the sources of the library.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include "agb_dev.cuh"

// Values fixed for the life of a device (its SM count, the resident blocks of one
// kernel) are read on the device current at the call and cached per device index.
// Host threads making their first call at the same time store the same value, so
// relaxed atomics are enough.
#define AGB_MAX_DEVICES 64

inline int current_device()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= AGB_MAX_DEVICES) d = 0;
    return d;
}

inline std::atomic<int> g_num_sms[AGB_MAX_DEVICES];

inline int num_sms()
{
    const int dev = current_device();
    int v = g_num_sms[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        g_num_sms[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

// resident blocks per SM of `kernel` at `threads` threads, cached per device in `cache`
template <typename K>
inline int blocks_per_sm(std::atomic<int>* cache, K kernel, int threads)
{
    const int dev = current_device();
    int b = cache[dev].load(std::memory_order_relaxed);
    if (b == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, 0) != cudaSuccess || b < 1)
            b = 1;
        cache[dev].store(b, std::memory_order_relaxed);
    }
    return b;
}

constexpr size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// eval.cu: the thread's last error (returns code), and a launch's status, counted
int agb_set_error(int code, const char* what);
int agb_check_launch(const char* what);

// launch-shape bits of out_flags (blocks per slot, threads per block, points per thread)
#define AGB_OUT_SHAPE_BITS ((15 << AGB_OUT_GRID_SHIFT) | (3 << AGB_OUT_BLOCK_SHIFT) | (15 << AGB_OUT_PPT_SHIFT))

// split.cu: launches the split kernel (a few points per block, the harmonics shared by its
// warps) where that is the better shape for this call; false where it is not
bool agb_launch_split(int mode, bool mixed, EvalArgs& a, cudaStream_t st);

// cyl.cu: the same for trees whose expansions are CylSplines
bool agb_launch_cyl(int mode, bool mixed, EvalArgs& a, cudaStream_t st);
