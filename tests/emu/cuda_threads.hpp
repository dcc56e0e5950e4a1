// Runs one CTA of a CUDA kernel on host threads: enough of the device
// vocabulary for the bucket kernel (barriers, warp shuffles up, an atomic
// counter, vector types). Shared arrays become statics, so one CTA at a time.
#pragma once
#include <algorithm>
#include <barrier>
#include <cstdint>
#include <memory>
#include <thread>
#include <vector>
using std::max;
using std::min;
#define __host__
#define __device__
#define __global__
#define __shared__ static
#define __constant__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)
#define ZG_HD inline
struct uint4 {
  uint32_t x, y, z, w;
};
struct uint2 {
  uint32_t x, y;
};
inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return {a, b, c, d}; }
inline uint2 make_uint2(uint32_t a, uint32_t b) { return {a, b}; }
struct Dim3 {
  unsigned x, y, z;
};
inline thread_local Dim3 threadIdx, blockIdx;
inline std::unique_ptr<std::barrier<>> g_block, g_warp[32];
inline uint32_t g_lane[1024];
inline void __syncthreads() { g_block->arrive_and_wait(); }
inline void __syncwarp() { g_warp[threadIdx.x >> 5]->arrive_and_wait(); }
inline uint32_t __shfl_up_sync(uint32_t, uint32_t v, unsigned d) {
  const unsigned t = threadIdx.x;
  g_lane[t] = v;
  __syncwarp();
  const uint32_t r = (t & 31) >= d ? g_lane[t - d] : v;
  __syncwarp();
  return r;
}
inline uint32_t atomicAdd(uint32_t* p, uint32_t v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
// the FP64 product is compiled but not run here
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __fma_rz(double a, double b, double c) { return a * b + c; }
inline double __fma_rn(double a, double b, double c) { return a * b + c; }
inline double __hiloint2double(int, int) { return 0; }
inline long long __double_as_longlong(double) { return 0; }
inline uint32_t __funnelshift_r(uint32_t, uint32_t, uint32_t) { return 0; }

template <class F>
void run_block(unsigned threads, F f) {
  g_block = std::make_unique<std::barrier<>>(threads);
  for (unsigned w = 0; w < threads / 32; ++w) g_warp[w] = std::make_unique<std::barrier<>>(32);
  std::vector<std::thread> all;
  for (unsigned t = 0; t < threads; ++t)
    all.emplace_back([=] {
      threadIdx = {t, 0, 0};
      blockIdx = {0, 0, 0};
      f();
    });
  for (auto& x : all) x.join();
}
