// The CUDA built-ins that csrc/owner_pass.cuh uses, for one thread block on the
// CPU: a host thread per CUDA thread, barriers for the warp collectives.
#pragma once
#include <pthread.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <thread>
#include <type_traits>
#include <vector>

#define __device__
#define __forceinline__ inline
#define __shared__
#define __align__(n) __attribute__((aligned(n)))

struct int2 {
  int x, y;
};
inline int2 make_int2(int x, int y) { return int2{x, y}; }
struct Dim {
  unsigned x;
};
inline Dim blockDim, gridDim;
inline thread_local Dim threadIdx, blockIdx;
using std::max;
using std::min;

struct Warp {
  pthread_barrier_t bar;
  uint64_t word[32];
};
inline std::vector<Warp> g_warps;
inline pthread_barrier_t g_block;

inline void __syncthreads() { pthread_barrier_wait(&g_block); }
inline void __syncwarp() { pthread_barrier_wait(&g_warps[threadIdx.x / 32].bar); }
template <class T>
T lane_value(T v, int from) {
  Warp &w = g_warps[threadIdx.x / 32];
  uint64_t bits = 0;
  std::memcpy(&bits, &v, sizeof v);
  w.word[threadIdx.x & 31] = bits;
  __syncwarp();
  if (from >= 0) std::memcpy(&v, &w.word[from], sizeof v);
  __syncwarp();
  return v;
}
template <class T>
T __shfl_sync(unsigned, T v, int from) { return lane_value(v, from & 31); }
template <class T>
T __shfl_xor_sync(unsigned, T v, int mask) { return lane_value(v, static_cast<int>(threadIdx.x & 31) ^ mask); }
template <class T>
T __shfl_up_sync(unsigned, T v, int by) { return lane_value(v, static_cast<int>(threadIdx.x & 31) - by); }
inline unsigned __ballot_sync(unsigned, bool p) {
  Warp &w = g_warps[threadIdx.x / 32];
  w.word[threadIdx.x & 31] = p;
  __syncwarp();
  unsigned m = 0;
  for (int i = 0; i < 32; ++i) m |= static_cast<unsigned>(w.word[i]) << i;
  __syncwarp();
  return m;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __ffs(unsigned x) { return __builtin_ffs(static_cast<int>(x)); }
inline int atomicAdd(int *p, int v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
inline unsigned atomicOr(unsigned *p, unsigned v) { return __atomic_fetch_or(p, v, __ATOMIC_SEQ_CST); }
inline int atomicMax(int *p, int v) {
  int old = __atomic_load_n(p, __ATOMIC_SEQ_CST);
  while (old < v && !__atomic_compare_exchange_n(p, &old, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
  return old;
}
template <class T>
T __ldcg(const T *p) { return *p; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline int __float_as_int(float f) {
  int i;
  std::memcpy(&i, &f, 4);
  return i;
}

namespace dlp {
struct SumBarrier;
inline float label_recip(float, bool) { return 0.0f; }
inline bool recip_serves(float, float) { return false; }
inline float label_by_recip(float, float, float) { return 0.0f; }
inline float updated_label(float w, float l, float old, bool) {
  return std::fmin(std::fmax(w > 1e-10f ? l / w : old, 0.0f), 1.0f);
}
}  // namespace dlp

// Runs f() on every thread of one block.
template <class F>
void run_block(unsigned block, unsigned threads, F f) {
  blockDim.x = threads;
  g_warps = std::vector<Warp>(threads / 32);
  for (Warp &w : g_warps) pthread_barrier_init(&w.bar, nullptr, 32);
  pthread_barrier_init(&g_block, nullptr, threads);
  std::vector<std::thread> ts;
  for (unsigned t = 0; t < threads; ++t)
    ts.emplace_back([=] {
      threadIdx.x = t;
      blockIdx.x = block;
      f();
    });
  for (std::thread &t : ts) t.join();
}
