// Shared host and device helpers of the GB300 DynLP library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "dlp_gb300.h"

namespace dlp {

// ---------------------------------------------------------------------------
// Host-side error plumbing: every C-ABI call returns a status and leaves a
// message for the calling thread.
// ---------------------------------------------------------------------------
void set_error(const std::string &msg);
void clear_error();
int fail(int status, const std::string &msg);
int cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define DLP_CUDA_TRY(call)                                                    \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) return ::dlp::cuda_fail(e_, #call, __FILE__, __LINE__); \
  } while (0)

#define DLP_TRY(call)                \
  do {                               \
    int s_ = (call);                 \
    if (s_ != DLP_OK) return s_;     \
  } while (0)

// Threads per block of the persistent kernels (a build setting: 512 or 1024).
#ifndef DLP_BLOCK
#define DLP_BLOCK 1024
#endif
constexpr int kBlockThreads = DLP_BLOCK;
static_assert(kBlockThreads == 512 || kBlockThreads == 1024, "the persistent kernels are tuned for 512 or 1024 threads");

// Checks that a GPU of compute capability 10.3 is current.
int require_device();

// Vertex status values of the reference (headers/graphTypes.h:191-195).
constexpr int kActive = 0;
constexpr int kDeleted = 1;
constexpr int kGroundTruth = 2;

// ---------------------------------------------------------------------------
// Device primitives.
// ---------------------------------------------------------------------------

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acq_rel_u32(unsigned *p, unsigned v) {
  unsigned old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;"
               : "=r"(old)
               : "l"(p), "r"(v)
               : "memory");
  return old;
}
__device__ __forceinline__ int ld_relaxed_i32(const int *p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier over the first `nblocks` blocks of a cooperative launch (all blocks
// co-resident). Arrivals are counted in two levels — groups of 16 blocks, then
// the groups — so they do not all serialise on one counter; the last block to
// arrive advances the generation, the others wait for it with a time limit. A
// block that runs out of time records DLP_ERR_TIMEOUT in *err and every block
// leaves at its next barrier, so no wait is unbounded.
constexpr int kBarrierGroup = 16;
constexpr int kBarrierMaxGroups = 128;

struct GridBarrier {
  unsigned count;
  unsigned gen;
  unsigned group[kBarrierMaxGroups];
};

__device__ __forceinline__ bool grid_sync_n(GridBarrier *bar, unsigned nblocks, int *err, uint64_t timeout_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned gen = ld_acquire_u32(&bar->gen);
    const unsigned ngroups = (nblocks + kBarrierGroup - 1) / kBarrierGroup;
    bool last = false;
    if (ngroups <= 1 || ngroups > kBarrierMaxGroups) {
      last = atom_add_acq_rel_u32(&bar->count, 1u) == nblocks - 1;
      if (last) bar->count = 0;
    } else {
      const unsigned grp = blockIdx.x / kBarrierGroup;
      const unsigned gsize = min(static_cast<unsigned>(kBarrierGroup), nblocks - grp * kBarrierGroup);
      if (atom_add_acq_rel_u32(&bar->group[grp], 1u) == gsize - 1) {
        bar->group[grp] = 0;  // ordered before the release of the next arrival
        last = atom_add_acq_rel_u32(&bar->count, 1u) == ngroups - 1;
        if (last) bar->count = 0;
      }
    }
    int ok = 1;
    if (last) {
      st_release_u32(&bar->gen, gen + 1);
    } else {
      const uint64_t t0 = global_timer_ns();
      unsigned spins = 0;
      while (ld_acquire_u32(&bar->gen) == gen) {
        if (((++spins) & 63u) == 0 && global_timer_ns() - t0 > timeout_ns) {
          atomicCAS(err, 0, DLP_ERR_TIMEOUT);
          ok = 0;
          break;
        }
        __nanosleep(20);
      }
    }
    s_ok = ok && (ld_relaxed_i32(err) == 0);
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ bool grid_sync(GridBarrier *bar, int *err, uint64_t timeout_ns) {
  return grid_sync_n(bar, gridDim.x * gridDim.y * gridDim.z, err, timeout_ns);
}

// Barrier over all blocks of a cooperative launch, in one hop: every block adds
// one word to a counter and one thread of it polls that counter, so an arrival
// is seen after one addition and one load instead of two dependent atomics, a
// release and a poll. The word is 64 bits of fields that the addition sums over
// the blocks (arrivals, rows, blocks that moved a label, that want to stop,
// that failed), which saves the loads that would follow the barrier. Four
// counters take turns: block 0 clears the one used two generations ago, which
// every block has read before it arrived at this one, and which is added to
// again two generations on.
//
// Measured on 152 blocks of 1,024 threads, full-grid passes of replays: 5.1 us
// a pass at 5,000 vertices, 7.5 to 8.0 at 50,000 and 16.2 at 500,000, against
// 7.1 to 7.2, 9.4 to 10.1 and 17.7 to 18 with GridBarrier. (A word per block
// polled by all blocks, 152 words each, gave 5.3 to 8.1 and 8 to 11 us: the
// polls of 760 warps queue up in the L2 slices that hold the words.)
//
// The counters start at zero in every launch. Every wait has a time limit; a
// block that runs out records DLP_ERR_TIMEOUT and leaves, and so do the blocks
// that then wait for it.
constexpr int kSumBlocks = 255;  // blocks at most
constexpr unsigned long long kSumArrival = 1ull << 56, kSumError = 1ull << 48, kSumStop = 1ull << 40,
                             kSumMoved = 1ull << 32;  // the low 32 bits sum a count

struct SumBarrier {
  struct {
    unsigned long long v;
    unsigned long long pad[15];
  } word[4];
};

struct SumState {  // in shared memory, one per block
  unsigned gen;    // barriers passed
  unsigned long long sum;
};

// All threads of all blocks call. mine() is evaluated by thread 0 after the
// block's own barrier; `sum` receives the fields summed over the blocks. False
// when a block sent kSumError or a wait ran out.
template <class Mine>
__device__ __forceinline__ bool sum_sync(SumBarrier *bar, SumState &f, int *err, uint64_t timeout_ns, Mine mine,
                                         unsigned long long &sum) {
  __syncthreads();
  if (gridDim.x == 1) {  // a launch of one block
    if (threadIdx.x == 0) f.sum = mine();
    __syncthreads();
    sum = f.sum;
    __syncthreads();  // before the next call's
    return (sum & (0xffull * kSumError)) == 0;
  }
  if (threadIdx.x == 0) {
    const unsigned gen = f.gen;
    unsigned long long *word = &bar->word[gen & 3].v;
    const unsigned long long add = kSumArrival | mine();
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(add) : "memory");
    const unsigned long long want = static_cast<unsigned long long>(gridDim.x) << 56;
    unsigned long long v;
    uint64_t t0 = 0;
    for (unsigned spins = 1;; ++spins) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
      if (v >= want) break;
      if ((spins & 63u) == 0) {
        const uint64_t now = global_timer_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > timeout_ns) {
          atomicCAS(err, 0, DLP_ERR_TIMEOUT);
          v = kSumError;
          break;
        }
      }
    }
    if (blockIdx.x == 0) bar->word[(gen + 2) & 3].v = 0;
    f.gen = gen + 1;
    f.sum = v;
  }
  __syncthreads();
  sum = f.sum;
  return (sum & (0xffull * kSumError)) == 0;
}

// *p if c, else d; the load is predicated, not branched around, so that several are in
// flight together.
__device__ __forceinline__ int load_if(bool c, const int *p, int d) {
  int v;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.s32 p, %2, 0;\n\t"
      "mov.b32 %0, %3;\n\t"
      "@p ld.global.b32 %0, [%1];\n\t"
      "}" : "=&r"(v) : "l"(p), "r"(static_cast<int>(c)), "r"(d));
  return v;
}
__device__ __forceinline__ int2 load_if(bool c, const int2 *p, int d) {
  int2 v;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.s32 p, %3, 0;\n\t"
      "mov.b32 %0, %4;\n\t"
      "mov.b32 %1, %4;\n\t"
      "@p ld.global.v2.b32 {%0, %1}, [%2];\n\t"
      "}" : "=&r"(v.x), "=&r"(v.y) : "l"(p), "r"(static_cast<int>(c)), "r"(d));
  return v;
}

__device__ __forceinline__ unsigned load_if(bool c, const uint8_t *p, unsigned d) {
  unsigned v;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.s32 p, %2, 0;\n\t"
      "mov.b32 %0, %3;\n\t"
      "@p ld.global.u8 %0, [%1];\n\t"
      "}" : "=&r"(v) : "l"(p), "r"(static_cast<int>(c)), "r"(d));
  return v;
}

// Appends the set lanes' values to list[*count ...] with one atomic per warp.
// Must be called by all lanes of the warp (convergent).
__device__ __forceinline__ void warp_append(bool pred, int value, int *list, int *count) {
  const unsigned mask = __ballot_sync(0xffffffffu, pred);
  if (mask == 0) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) list[base + __popc(mask & ((1u << lane) - 1u))] = value;
}

// Same, growing downward from list[cap - 1] (for a second list sharing the array).
__device__ __forceinline__ void warp_append_back(bool pred, int value, int *list, int cap,
                                                 int *count) {
  const unsigned mask = __ballot_sync(0xffffffffu, pred);
  if (mask == 0) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) list[cap - 1 - (base + __popc(mask & ((1u << lane) - 1u)))] = value;
}

__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// 32.32 fixed point for exact, order-independent supernode weight sums.
__device__ __forceinline__ long long to_fixed(float w) {
  return __double2ll_rn(static_cast<double>(w) * 4294967296.0);
}
__device__ __forceinline__ float from_fixed(long long q) {
  return __double2float_rn(__ll2double_rn(q) * (1.0 / 4294967296.0));
}

// New label from the two row sums (src/iterativePropagation.cu:153-168) with an
// IEEE round-to-nearest division.
// The quotient of a weighted average. Default: IEEE round-to-nearest, the
// oracle's arithmetic. fast: the CUDA fast division (__fdividef), the division
// that the reference's -use_fast_math build makes of its `/`
// (src/iterativePropagation.cu:160, src/labelInitialization.cu:137; Makefile:52).
__device__ __forceinline__ float quotient(float num, float den, bool fast) {
  return fast ? __fdividef(num, den) : __fdiv_rn(num, den);
}

__device__ __forceinline__ float updated_label(float w_all, float w_label, float old, bool fast = false) {
  float nl = (w_all > 1e-10f) ? quotient(w_label, w_all, fast) : old;
  return fminf(fmaxf(nl, 0.0f), 1.0f);
}

// a / b, correctly rounded, from y = RN(1 / b): q1 is a/b to within an ulp, its
// remainder is exact, and one more correction by y rounds correctly (P.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990). 1e-10 < b <= kDivHi, and a is 0
// or in [kDivLo, kDivHi], so that nothing here underflows or overflows. The
// reciprocal can be known before the numerator, which leaves five dependent
// multiply-adds of the division; and a zero numerator, which is common where all
// neighbours have label 0, takes no other path.
constexpr float kDivLo = 0x1p-40f, kDivHi = 0x1p40f;
__device__ __forceinline__ float divide(float a, float b, float y) {
  const float q0 = __fmul_rn(a, y);
  const float q1 = __fmaf_rn(__fmaf_rn(-b, q0, a), y, q0);
  return __fmaf_rn(__fmaf_rn(-b, q1, a), y, q1);
}

// updated_label from the reciprocal of the weight sum: label_recip is 0, and
// recip_serves false, where updated_label has to be called instead.
__device__ __forceinline__ float label_recip(float w_all, bool fast) {
  return !fast && w_all > 1e-10f && w_all <= kDivHi ? __frcp_rn(w_all) : 0.0f;
}
__device__ __forceinline__ bool recip_serves(float recip, float w_label) {
  return (recip != 0.0f) & ((w_label == 0.0f) | ((w_label >= kDivLo) & (w_label <= kDivHi)));
}
__device__ __forceinline__ float label_by_recip(float w_all, float recip, float w_label) {
  return fminf(fmaxf(divide(w_label, w_all, recip), 0.0f), 1.0f);
}

// The current device's context: an id that no other context of the process has had, 0
// when there is none to be asked. What a host function keeps for a device (a pool,
// an address, a kernel's attributes) is lost with the context, which
// cudaDeviceReset ends, and is kept by this id. 12 ns.
unsigned long long context_id();

// Launch helper: cooperative launch of `kernel` with `args` on `stream`.
int launch_cooperative(const void *kernel, int grid, int block, void **args, size_t smem,
                       cudaStream_t stream);

}  // namespace dlp
