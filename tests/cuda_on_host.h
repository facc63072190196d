// Runs a block of a CUDA kernel on the CPU, one std::thread per CUDA thread and
// a pthread barrier for __syncthreads, so that ThreadSanitizer sees every access
// to shared and global memory that no barrier orders (test infrastructure: the
// kernels' own source is compiled against this header).
#pragma once
#include <math.h>
#include <pthread.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <functional>
#include <thread>
#include <type_traits>
#include <utility>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __align__(n)

struct dim3 {
    unsigned x, y, z;
    dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {}
};
struct float2 { float x, y; };
struct double2 { double x, y; };
static thread_local dim3 blockIdx, threadIdx;
static dim3 blockDim, gridDim;
static pthread_barrier_t block_bar;
static std::vector<pthread_barrier_t> warp_bar;
alignas(16) unsigned char shared_raw[227 * 1024];

static inline void __syncthreads() { pthread_barrier_wait(&block_bar); }
static inline void __syncwarp() { pthread_barrier_wait(&warp_bar[threadIdx.x >> 5]); }
static inline size_t __cvta_generic_to_shared(const void* p) { return (const unsigned char*)p - shared_raw; }
static inline int __float2int_rz(float x) { return (int)x; }
static inline float __fdividef(float a, float b) { return a / b; }
using std::min;
template <typename T>
T __shfl_up_sync(unsigned, T v, int) { abort(); return v; }
template <typename T>
T __shfl_down_sync(unsigned, T v, int) { abort(); return v; }

// cp.async: the destination is unknown from the issue on and holds the data
// once the group has been waited for
struct Copy { unsigned char* dst; const void* src; };
static thread_local std::vector<std::vector<Copy>> groups;
static thread_local std::vector<Copy> open_group;
static inline void cp_async16_full(uint32_t saddr, const void* g) {
    if (saddr % 16 || (size_t)g % 16 || saddr + 16 > sizeof shared_raw) { fprintf(stderr, "cp.async: bad address\n"); abort(); }
    memset(shared_raw + saddr, 0xff, 16);
    open_group.push_back({shared_raw + saddr, g});
}
static inline void cp_async_commit() { groups.push_back(std::move(open_group)); open_group.clear(); }
template <int N>
static inline void cp_async_wait_newest() {
    while ((int)groups.size() > N) {
        for (const Copy& c : groups.front()) memcpy(c.dst, c.src, 16);
        groups.erase(groups.begin());
    }
}
static inline void cp_async_wait_all_groups() { cp_async_wait_newest<0>(); }

// one launch, block after block
static void launch(dim3 grid, unsigned threads, const std::function<void()>& kernel) {
    gridDim = grid;
    blockDim = dim3(threads);
    warp_bar.resize((threads + 31) / 32);
    for (unsigned z = 0; z < grid.z; z++)
        for (unsigned y = 0; y < grid.y; y++)
            for (unsigned x = 0; x < grid.x; x++) {
                memset(shared_raw, 0xff, sizeof shared_raw);
                pthread_barrier_init(&block_bar, nullptr, threads);
                for (auto& b : warp_bar) pthread_barrier_init(&b, nullptr, 32);
                std::vector<std::thread> t;
                for (unsigned i = 0; i < threads; i++)
                    t.emplace_back([&, i] {
                        blockIdx = dim3(x, y, z);
                        threadIdx = dim3(i, 0, 0);
                        kernel();
                    });
                for (auto& th : t) th.join();
                pthread_barrier_destroy(&block_bar);
                for (auto& b : warp_bar) pthread_barrier_destroy(&b);
            }
}
