// The reference's five step launchers on caller-owned device arrays in the
// reference's layout (packed CSR with separate colInd / values, int32 status,
// gtClass and isAffected arrays). C ABI group 3 in dlp_gb300.h.
//
// Each launcher keeps the reference's argument meaning and its outputs,
// including the soft-delete (-1) entries and the final isAffected state, but
// runs as GB300 kernels: group-per-row walks instead of a 256-thread block per
// row, a single cooperative kernel for the whole Shiloach-Vishkin loop and for
// the whole propagation loop (no host round trip per round), and stream-ordered
// temporaries (cudaMallocAsync) instead of cudaMalloc/cudaFree per round. They
// synchronise the stream only to return a scalar through a pointer
// (numSubEdges, numComponents, iterationsUsed), as the reference's int&
// outputs require.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "owner_pass.cuh"
#include "row_stint.cuh"
#include "row_sums.cuh"

namespace dlp {
namespace ref_layout {
namespace {

// Division of the label updates in the launchers (dlp_set_launcher_arithmetic).
std::atomic<int> g_launcher_arith{DLP_ARITH_IEEE};

constexpr int kBlock = 256;
constexpr int kGroup = 8;               // lanes per row in the row walks
constexpr int kMaxHookRounds = 100;     // src/connectedComponents.cu:209
constexpr int kNarrowMax = 32;

__device__ __forceinline__ bool in_range(int v, int n) {
  return static_cast<unsigned>(v) < static_cast<unsigned>(n);
}

int grid_for(long long items, int per_block) {
  long long g = (items + per_block - 1) / per_block;
  return static_cast<int>(std::max<long long>(1, std::min<long long>(g, 152LL * 32)));
}

// The launchers' temporaries come from a stream-ordered pool of the library's
// own, one per device, that holds on to at most kPoolBytes between calls. (The
// default pool gives everything back to the system at each device
// synchronisation, and the next call maps it again: 200 us a call for a caller
// that synchronises the device between calls.) The driver orders its blocks
// between streams and threads; what a call allocates beyond the limit goes back
// at the next synchronisation, the rest with the device's context.
constexpr unsigned long long kPoolBytes = 32ull << 20;

// What the launchers keep for a device's context, made when it is first asked for.
struct ContextFacts {
  bool pool_asked = false;
  cudaMemPool_t pool = nullptr;  // null: the default pool serves
  bool shape_asked = false;
  int owned_grid = 0;            // blocks of the owned kernels, 0 when they do not fit
  size_t owned_fixed = 0, owned_smem = 0;  // their static shared memory, the most of the dynamic one
  void *scratch = nullptr;       // of dlp_iterative_propagation_noalloc
};

// fn on the facts of the current device's context, one thread at a time; false when
// the context cannot be told.
template <class Fn>
bool with_context(Fn fn) {
  static std::mutex mu;
  // not destroyed at the end of the process, when the contexts are gone already
  static auto &known = *new std::map<std::pair<int, unsigned long long>, ContextFacts>();
  int dev = -1;
  const unsigned long long id = context_id();
  if (id == 0 || cudaGetDevice(&dev) != cudaSuccess) return false;
  std::lock_guard<std::mutex> lock(mu);
  fn(known[{dev, id}], dev);
  return true;
}

// The current device's pool, null for the default one.
cudaMemPool_t tmp_pool() {
  cudaMemPool_t pool = nullptr;
  with_context([&](ContextFacts &f, int dev) {
    if (!f.pool_asked) {
      f.pool_asked = true;
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      unsigned long long keep = kPoolBytes;
      // in a thread that captures a stream, too: the pool is no part of the graph
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (cudaMemPoolCreate(&f.pool, &props) != cudaSuccess) f.pool = nullptr;
      else cudaMemPoolSetAttribute(f.pool, cudaMemPoolAttrReleaseThreshold, &keep);
      cudaThreadExchangeStreamCaptureMode(&mode);
      cudaGetLastError();
    }
    pool = f.pool;
  });
  return pool;
}

template <class T>
int tmp_alloc(T **p, size_t count, cudaStream_t s) {
  const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
  cudaMemPool_t pool = tmp_pool();
  if (pool) DLP_CUDA_TRY(cudaMallocFromPoolAsync(reinterpret_cast<void **>(p), bytes, pool, s));
  else DLP_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void **>(p), bytes, s));
  return DLP_OK;
}

// ------------------------------------------------------- mark deletions ----
// src/sparsifySubgraph.cu:58-83: neighbours of each deleted vertex's row are
// affected, the row is soft-deleted, the vertex becomes DELETED.
__global__ void mark_deleted_rows(const int *row_ptr, int *col, int *status, int *affected,
                                  const int *deleted, int count, int n) {
  const int lane = threadIdx.x & 31, gl = lane & (kGroup - 1);
  const int group = (blockIdx.x * blockDim.x + threadIdx.x) / kGroup;
  const int groups = gridDim.x * blockDim.x / kGroup;
  for (int i = group; i < count; i += groups) {
    const int u = deleted[i];
    if (!in_range(u, n)) continue;
    const int rs = row_ptr[u], re = row_ptr[u + 1];
    for (int e = rs + gl; e < re; e += kGroup) {
      const int v = col[e];
      if (in_range(v, n)) atomicMax(&affected[v], 1);
      col[e] = -1;
    }
    if (gl == 0) status[u] = kDeleted;
  }
}

// src/sparsifySubgraph.cu:92-111: entries pointing at a DELETED vertex, in the
// rows of vertices that are not DELETED themselves. A warp takes 32 rows, whose
// entries are one contiguous range: it is read coalesced whatever the row
// lengths are, and only a range with a deleted vertex's entries in it looks up
// which row an entry is in. Bound by the status gathers (a sector each).
// Measured on 2 million rows of 2.1 entries on average: 27 us, against 63 us
// with eight lanes per row.
__global__ void clean_incoming(const int *row_ptr, int *col, const int *status, int n) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int u0 = warp * 32; u0 < n; u0 += nwarps * 32) {
    const int u = u0 + lane;
    const int rs = row_ptr[min(u, n)], end = row_ptr[min(u0 + 32, n)];
    const int re = min(u + 1, n) == n ? row_ptr[n] : row_ptr[u + 1];
    const bool gone = u < n && status[u] == kDeleted && re > rs;
    const unsigned skip = __ballot_sync(0xffffffffu, gone);
    const int begin = __shfl_sync(0xffffffffu, rs, 0);
    for (int e = begin + lane; e - lane < end; e += 32) {
      const int v = e < end ? col[e] : -1;
      bool hit = in_range(v, n) && status[v] == kDeleted;
      if (skip) {  // the last row that starts at or before the entry and is not empty
        int r = 0;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
          const int s = __shfl_sync(0xffffffffu, rs, r + o);
          if (s <= e) r += o;
        }
        hit = hit && !((skip >> r) & 1u);
      }
      if (hit) col[e] = -1;
    }
  }
}

// ---------------------------------------------------------- sparsify -------
struct SparsifyArgs {
  const int *src, *dst;
  const float *w;
  int m;
  const int *is_new;
  int n;
  float tau;
};

__device__ __forceinline__ bool kept_edge(const SparsifyArgs &a, int i, int &u, int &v, float &w, bool &bad) {
  u = a.src[i];
  v = a.dst[i];
  w = a.w[i];
  if (!in_range(u, a.n) || !in_range(v, a.n)) {
    bad = true;
    return false;
  }
  return a.is_new[u] && a.is_new[v] && w > a.tau;
}

// Blocks of the step kernels below: one cooperative launch each, with a barrier
// between their phases (SumBarrier: 1.3 us) instead of a launch. A few thousand
// items per block; small steps take one block, whose barrier is __syncthreads.
constexpr int kStepBlock = 1024;
struct StepScratch {       // zeroed before the launch of more than one block
  SumBarrier bar;
  int out[16];             // kStep*
  int count[kSumBlocks + 1];  // per block
};
enum { kStepError = 0, kStepTotal = 1 };

__shared__ SumState s_step;

// Every step kernel's first statement.
__device__ __forceinline__ void step_begin(StepScratch *sc) {
  if (threadIdx.x != 0) return;
  s_step.gen = 0;
  if (gridDim.x == 1) sc->out[kStepError] = sc->out[kStepTotal] = 0;
}
__device__ __forceinline__ bool step_sync(StepScratch *sc, unsigned long long mine, unsigned long long &sum) {
  return sum_sync(&sc->bar, s_step, &sc->out[kStepError], 2000000000ull, [&] { return mine; }, sum);
}
__device__ __forceinline__ bool step_sync(StepScratch *sc) {
  unsigned long long sum;
  return step_sync(sc, 0ull, sum);
}

// Exclusive prefix of v over the block's threads; total receives the sum.
__device__ __forceinline__ int block_prefix(int v, int &total) {
  __shared__ int s_warp[kStepBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();  // s_warp's last readers
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int w = s_warp[lane], wi = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, wi, o);
    if (lane >= o) wi += t;
  }
  total = __shfl_sync(0xffffffffu, wi, 31);
  return incl - v + __shfl_sync(0xffffffffu, wi - w, warp);
}

// Sum of count[0 .. blocks) before this block, by all threads of the block.
__device__ __forceinline__ int blocks_before(const int *count) {
  int total;
  block_prefix(threadIdx.x < blockIdx.x ? __ldcg(count + threadIdx.x) : 0, total);
  return total;
}

// src/sparsifySubgraph.cu:119-179 in one launch: every block counts the kept
// edges of its range, then writes them in raw order (both directions) behind
// those of the blocks before it, with the clipped endpoint marks (numNodes =
// numInserted, :259-263). Nothing is written when an endpoint is invalid.
__global__ void __launch_bounds__(kStepBlock, 1)
    sparsify_kernel(SparsifyArgs a, StepScratch *sc, int *affected, int mark_limit, int *sub_col, float *sub_val) {
  step_begin(sc);
  const int per = (a.m + gridDim.x - 1) / gridDim.x;
  const int lo = min(static_cast<int>(blockIdx.x) * per, a.m), hi = min(lo + per, a.m);
  bool bad = false;
  int kept = 0, u, v;
  float w;
  for (int i = lo + threadIdx.x; i < hi; i += kStepBlock) kept += kept_edge(a, i, u, v, w, bad);
  int mine;
  block_prefix(kept, mine);
  bad = __syncthreads_or(bad) != 0;
  if (threadIdx.x == 0) sc->count[blockIdx.x] = mine;
  unsigned long long sum;
  if (!step_sync(sc, static_cast<unsigned>(mine) | (bad ? kSumStop : 0ull), sum)) return;
  if (sum & (0xffull * kSumStop)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->out[kStepError] = DLP_ERR_INVALID_ARGUMENT;
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->out[kStepTotal] = 2 * static_cast<int>(static_cast<unsigned>(sum));
  int at = blocks_before(sc->count);
  for (int base = lo; base < hi; base += kStepBlock) {
    const int i = base + threadIdx.x;
    const bool k = i < hi && kept_edge(a, i, u, v, w, bad);
    int total;
    const int pos = at + block_prefix(k, total);
    at += total;
    if (k) {
      sub_col[2 * pos] = v;
      sub_col[2 * pos + 1] = u;
      sub_val[2 * pos] = w;
      sub_val[2 * pos + 1] = w;
    }
    if (i < hi && w > a.tau) {
      if (u >= 0 && u < mark_limit) atomicMax(&affected[u], 1);
      if (v >= 0 && v < mark_limit) atomicMax(&affected[v], 1);
    }
  }
}

// ------------------------------------------------- connected components ----
struct CcArgs {
  const int *es, *ed;
  int m;
  const int *ins;
  int I, n;
  int *par;         // n
  int *comp;        // n: component ids
  unsigned *bits;   // a bit per vertex: roots
  int *prefix;      // roots before each word of bits
  StepScratch *sc;
};

// The whole components step in one launch: clear and validate, parents of the
// inserted vertices (src/connectedComponents.cu:64-71), rounds of hooking
// (atomicMin of the larger root under the smaller, :79-100) and full pointer
// jumping (:108-121) until a hook pass changes nothing, then ids by the rank of
// the root among the roots in ascending vertex order (:264-283). par holds -1
// for vertices that are not inserted, and such a root gives id -1; the
// isRoot[-1] write of the reference is dropped. A round is bound by its random
// accesses to par; the rest is streaming. Measured on 200,000 inserted vertices
// of 2 million and 700,000 edges: 44 us, against 142 us with five kernels, whose
// scan of the root bits ran on one block.
__global__ void __launch_bounds__(kStepBlock, 1) cc_kernel(CcArgs a) {
  step_begin(a.sc);
  const int t = blockIdx.x * kStepBlock + threadIdx.x, nt = gridDim.x * kStepBlock;
  const int words = (a.n + 31) / 32;
  bool bad = false;
  for (int i = t; i < a.n; i += nt) {
    a.par[i] = -1;
    a.comp[i] = -1;
  }
  for (int i = t; i < words; i += nt) a.bits[i] = 0;
  for (int i = t; i < a.m; i += nt) bad |= !in_range(a.es[i], a.n) || !in_range(a.ed[i], a.n);
  for (int i = t; i < a.I; i += nt) bad |= !in_range(a.ins[i], a.n);
  bad = __syncthreads_or(bad) != 0;
  unsigned long long sum;
  if (!step_sync(a.sc, bad ? kSumStop : 0ull, sum)) return;
  if (sum & (0xffull * kSumStop)) {
    if (t == 0) a.sc->out[kStepError] = DLP_ERR_INVALID_ARGUMENT;
    return;
  }
  for (int i = t; i < a.I; i += nt) a.par[a.ins[i]] = a.ins[i];
  if (!step_sync(a.sc)) return;
  for (int r = 0; r < kMaxHookRounds; ++r) {
    bool changed = false;
    for (int i = t; i < a.m; i += nt) {
      const int ru = a.par[a.es[i]];
      const int rv = a.par[a.ed[i]];
      if (ru != rv) {
        const int hi = max(ru, rv), lo = min(ru, rv);
        if (atomicMin(&a.par[hi], lo) != lo) changed = true;
      }
    }
    changed = __syncthreads_or(changed) != 0;
    if (!step_sync(a.sc, changed ? kSumMoved : 0ull, sum)) return;
    if ((sum & (0xffull * kSumMoved)) == 0) break;  // par is as the last jump left it
    for (int i = t; i < a.I; i += nt) {
      const int v = a.ins[i];
      int p = a.par[v];
      while (p >= 0) {  // par[-1] reads as -1
        const int q = a.par[p];
        if (q == p) break;
        p = q;
      }
      a.par[v] = p;
    }
    if (!step_sync(a.sc)) return;
  }
  for (int i = t; i < a.I; i += nt) {
    const int v = a.ins[i];
    if (a.par[v] == v) atomicOr(&a.bits[v >> 5], 1u << (v & 31));
  }
  if (!step_sync(a.sc)) return;
  // ranks: a range of words per block, a run of words per thread
  const int per = (words + gridDim.x - 1) / gridDim.x;
  const int lo = min(static_cast<int>(blockIdx.x) * per, words), hi = min(lo + per, words);
  const int run = (hi - lo + kStepBlock - 1) / kStepBlock;
  const int wlo = min(lo + static_cast<int>(threadIdx.x) * run, hi), whi = min(wlo + run, hi);
  int roots = 0, mine;
  for (int w = wlo; w < whi; ++w) roots += __popc(__ldcg(a.bits + w));
  const int before = block_prefix(roots, mine);
  if (threadIdx.x == 0) a.sc->count[blockIdx.x] = mine;
  if (!step_sync(a.sc, static_cast<unsigned>(mine), sum)) return;
  if (t == 0) a.sc->out[kStepTotal] = static_cast<int>(static_cast<unsigned>(sum));
  int at = blocks_before(a.sc->count) + before;
  for (int w = wlo; w < whi; ++w) {
    a.prefix[w] = at;
    at += __popc(__ldcg(a.bits + w));
  }
  if (!step_sync(a.sc)) return;
  for (int i = t; i < a.I; i += nt) {
    const int v = a.ins[i];
    const int r = a.par[v];
    if (r >= 0) a.comp[v] = a.prefix[r >> 5] + __popc(a.bits[r >> 5] & ((1u << (r & 31)) - 1u));
  }
}

// ---------------------------------------------------- label init ----------
struct InitArgs {
  const int *row_ptr, *col;
  const float *val;
  float *labels;
  const int *comp;
  int num_comp;
  const int *gt, *ins;
  int I, n;
  long long *acc;  // 2 per component
  int fast_div;
};

// src/labelInitialization.cu:59-88: supernode weights per component in exact
// fixed-point sums. A lane per row: 155,000 rows in flight instead of 19,000 with
// eight lanes each, and the step is bound by the dependent loads of a row (vertex,
// component and row start, entries, classes). Rows beyond kLaneRow entries are
// shared by the warp.
__device__ __forceinline__ void init_weights(const InitArgs &a, int t, int nt) {
  constexpr int kLaneRow = 64, kAhead = 4;
  const int lane = threadIdx.x & 31;
  auto add = [&](int c, long long q0, long long q1) {
    if (q0) atomicAdd(reinterpret_cast<unsigned long long *>(&a.acc[2 * c]), static_cast<unsigned long long>(q0));
    if (q1) atomicAdd(reinterpret_cast<unsigned long long *>(&a.acc[2 * c + 1]), static_cast<unsigned long long>(q1));
  };
  for (int base = t - lane; base < a.I; base += nt) {
    const int i = base + lane;
    int c = -1, rs = 0, len = 0;
    if (i < a.I) {
      const int u = a.ins[i];
      if (in_range(u, a.n)) {
        c = a.comp[u];
        rs = a.row_ptr[u];
        len = a.row_ptr[u + 1] - rs;
        if (c < 0 || c >= a.num_comp) len = 0;  // out-of-range ids are treated as no component
      }
    }
    long long q0 = 0, q1 = 0;
    for (int e = 0; e < len && len <= kLaneRow; e += kAhead) {
      int v[kAhead], g[kAhead];
      float w[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const int at = rs + min(e + j, len - 1);
        v[j] = a.col[at];
        w[j] = a.val[at];
        if (e + j >= len) v[j] = -1;
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) g[j] = in_range(v[j], a.n) ? a.gt[v[j]] : -1;
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if (g[j] == 0) q0 += to_fixed(w[j]);
        else if (g[j] == 1) q1 += to_fixed(w[j]);
      }
    }
    if (q0 | q1) add(c, q0, q1);
    for (unsigned todo = __ballot_sync(0xffffffffu, len > kLaneRow); todo; todo &= todo - 1) {
      const int from = __ffs(todo) - 1;
      const int cq = __shfl_sync(0xffffffffu, c, from), rq = __shfl_sync(0xffffffffu, rs, from),
                lq = __shfl_sync(0xffffffffu, len, from);
      long long p0 = 0, p1 = 0;
      for (int e = lane; e < lq; e += 32) {
        const int v = a.col[rq + e];
        const int g = in_range(v, a.n) ? a.gt[v] : -1;
        if (g == 0) p0 += to_fixed(a.val[rq + e]);
        else if (g == 1) p1 += to_fixed(a.val[rq + e]);
      }
      p0 = warp_sum_ll(p0);
      p1 = warp_sum_ll(p1);
      if (lane == 0) add(cq, p0, p1);
    }
  }
}

// src/labelInitialization.cu:99-142.
__device__ __forceinline__ void init_labels(const InitArgs &a, int t, int nt) {
  for (int i = t; i < a.I; i += nt) {
    const int u = a.ins[i];
    if (!in_range(u, a.n)) continue;
    const int g = a.gt[u];
    if (g == 0) { a.labels[u] = 0.0f; continue; }
    if (g == 1) { a.labels[u] = 1.0f; continue; }
    const int c = a.comp[u];
    if (c < 0 || c >= a.num_comp) { a.labels[u] = 0.5f; continue; }
    const float w0 = from_fixed(__ldcg(a.acc + 2 * c));
    const float w1 = from_fixed(__ldcg(a.acc + 2 * c + 1));
    const float den = w0 + w1;
    a.labels[u] = den > 1e-10f ? quotient(w1, den, a.fast_div) : 0.5f;
  }
}

// The step returns nothing to the host, so nothing in it may fail on the device:
// two ordinary launches, no grid barrier whose wait could run out unseen. What
// one block takes is one launch.
__global__ void __launch_bounds__(kStepBlock, 1) init_weights_kernel(InitArgs a) {
  init_weights(a, blockIdx.x * kStepBlock + threadIdx.x, gridDim.x * kStepBlock);
}
__global__ void __launch_bounds__(kStepBlock, 1) init_labels_kernel(InitArgs a) {
  init_labels(a, blockIdx.x * kStepBlock + threadIdx.x, gridDim.x * kStepBlock);
}
__global__ void __launch_bounds__(kStepBlock, 1) init_kernel(InitArgs a) {
  for (int i = threadIdx.x; i < 2 * max(a.num_comp, 1); i += kStepBlock) a.acc[i] = 0;
  __syncthreads();
  init_weights(a, threadIdx.x, kStepBlock);
  __syncthreads();
  init_labels(a, threadIdx.x, kStepBlock);
}

// ------------------------------------------------------- propagation -------
struct PropArgs {
  const int *row_ptr, *col;
  const float *val;
  float *labels, *buffer;
  const int *status, *gt;
  int *affected;
  int n;
  float delta;
  int max_iter;
  unsigned *stamp;     // n, zeroed
  int *lists;          // 2n: the list of pass k in half k & 1
  int *counts;         // [3][2]
  int *out;            // [0] passes, [1] last mark stamp, [2] next pass after a block-0 stint
  GridBarrier *bar;
  int *err;
  unsigned long long timeout_ns;
  int fast_div;        // the division of the label updates (dlp_set_launcher_arithmetic)
};

// Frontier loop of src/iterativePropagation.cu:274-327 in one cooperative
// launch; per pass, the frontier is the set of vertices marked in the previous
// pass that are ACTIVE and not ground truth.
__global__ void __launch_bounds__(kBlock) prop_kernel(PropArgs a) {
  constexpr int G = kGroup;  // lanes per row of at most kNarrowMax entries
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31, gwarp = t >> 5, nwarps = nt >> 5;
  const int n = a.n;
  if (ld_relaxed_i32(a.err) != 0) return;
  auto append = [&](bool pred, int v, int set, int half) {
    bool wide = false;
    if (pred) wide = a.row_ptr[v + 1] - a.row_ptr[v] > kNarrowMax;
    int *list = a.lists + static_cast<size_t>(half) * n;
    warp_append(pred && !wide, v, list, &a.counts[2 * set]);
    warp_append_back(pred && wide, v, list, n, &a.counts[2 * set + 1]);
  };
  // seed: src/iterativePropagation.cu:63-78
  for (int base = gwarp * 32; base < n; base += nwarps * 32) {
    const int v = base + lane;
    const bool ok = v < n && a.affected[v] == 1 && a.status[v] == kActive && a.gt[v] < 0;
    append(ok, v, 0, 0);
  }
  if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;

  constexpr int GPW = 32 / G;
  const int grp = lane / G, gl = lane & (G - 1);
  // The rows of pass k (nn narrow, nw wide) by the warps
  // [w0, w0 + nws) of the launch; marks go to the list of pass k + 1.
  auto rows = [&](int k, int nn, int nw, int w0, int nws) {
    const float *src = (k & 1) ? a.buffer : a.labels;
    float *dst = (k & 1) ? a.labels : a.buffer;
    const unsigned stamp = static_cast<unsigned>(k) + 1u;
    const int nset = (k + 1) % 3;
    const int *cur = a.lists + static_cast<size_t>(k & 1) * n;
    auto mark = [&](bool cand, int v) {
      bool fresh = false;
      if (cand) fresh = atomicMax(&a.stamp[v], stamp) < stamp;
      append(fresh && a.status[v] == kActive && a.gt[v] < 0, v, nset, (k + 1) & 1);
    };
    for (int base = w0 * GPW; base < nn; base += nws * GPW) {
      const int item = base + grp;
      const bool valid = item < nn;
      int u = 0, rs = 0, len = 0;
      if (valid) {
        u = cur[item];
        rs = a.row_ptr[u];
        len = a.row_ptr[u + 1] - rs;
      }
      auto load = [&](int e, int &v, float &w) {
        v = a.col[rs + e];
        w = a.val[rs + e];
        if (v >= 0 && a.status[v] == kDeleted) v = -1;
      };
      float tw, tl;
      int cols[32 / G];
      group_row_sums<G>(len, gl, load, src, tw, tl, cols);
      int changed = 0;
      if (valid && gl == 0) {
        const float old = src[u];
        const float nl = updated_label(tw, tl, old, a.fast_div);
        dst[u] = nl;
        changed = fabsf(nl - old) > a.delta;
      }
      changed = __shfl_sync(0xffffffffu, changed, 0, G);
#pragma unroll
      for (int r = 0; r < 32 / G; ++r) mark(changed && cols[r] >= 0 && a.gt[cols[r]] < 0, cols[r]);
      mark(changed && gl == 0 && a.gt[u] < 0, u);
    }
    for (int wi = w0; wi < nw; wi += nws) {
      const int u = cur[n - 1 - wi];
      const int rs = a.row_ptr[u], len = a.row_ptr[u + 1] - rs;
      auto load = [&](int e, int &v, float &w) {
        v = a.col[rs + e];
        w = a.val[rs + e];
        if (v >= 0 && a.status[v] == kDeleted) v = -1;
      };
      float tw, tl;
      warp_row_sums(len, lane, load, src, tw, tl);
      int changed = 0;
      if (lane == 0) {
        const float old = src[u];
        const float nl = updated_label(tw, tl, old, a.fast_div);
        dst[u] = nl;
        changed = fabsf(nl - old) > a.delta;
      }
      changed = __shfl_sync(0xffffffffu, changed, 0);
      if (changed) {
        for (int e0 = 0; e0 < len; e0 += 32) {
          const int e = e0 + lane;
          int v = e < len ? a.col[rs + e] : -1;
          if (v >= 0 && a.status[v] == kDeleted) v = -1;
          mark(v >= 0 && a.gt[v] < 0, v);
        }
        mark(lane == 0 && a.gt[u] < 0, u);
      }
    }
  };
  // A frontier of narrow rows that one block takes in one round runs on
  // block 0 alone, pass after pass with block barriers, while the other
  // blocks wait at the next grid barrier: a pass then costs a block barrier
  // instead of a grid barrier. The stint ends when the frontier empties,
  // outgrows one round or gets a wide row, at maxIter, or after 100 ms (the
  // waiting blocks' barrier has a 2 s limit); block 0 publishes the next pass.
  constexpr int kSmallFront = kBlock / G;
  __shared__ int s_stop;
  int k = 0;
  for (;;) {
    const int set = k % 3;
    const int nn = ld_relaxed_i32(&a.counts[2 * set]);
    const int nw = ld_relaxed_i32(&a.counts[2 * set + 1]);
    if (nn + nw == 0 || k >= a.max_iter) break;
    if (nw == 0 && nn <= kSmallFront) {
      if (blockIdx.x == 0) {
        const int warp = threadIdx.x >> 5;
        const uint64_t t_start = global_timer_ns();
        if (threadIdx.x == 0) s_stop = 0;
        __syncthreads();
        for (;;) {
          const int cs = k % 3;
          const int cn = ld_relaxed_i32(&a.counts[2 * cs]);
          const int cw = ld_relaxed_i32(&a.counts[2 * cs + 1]);
          // the same decision in every thread: all inputs were written
          // before the last block barrier
          if (cn + cw == 0 || cw != 0 || cn > kSmallFront || k >= a.max_iter || s_stop) break;
          if (threadIdx.x == 0) {
            a.counts[2 * ((k + 2) % 3)] = 0;
            a.counts[2 * ((k + 2) % 3) + 1] = 0;
            if ((k & 15) == 15 && global_timer_ns() - t_start > 100000000ull) s_stop = 1;
          }
          rows(k, cn, 0, warp, kBlock / 32);
          __syncthreads();
          ++k;
        }
        if (threadIdx.x == 0) a.out[2] = k;
      }
      if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
      k = ld_relaxed_i32(&a.out[2]);
      continue;
    }
    if (t == 0) {
      a.counts[2 * ((k + 2) % 3)] = 0;
      a.counts[2 * ((k + 2) % 3) + 1] = 0;
    }
    rows(k, nn, nw, gwarp, nwarps);
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
    ++k;
  }
  // final labels in the primary array, ground truth enforced
  // (src/iterativePropagation.cu:330-339); isAffected holds the last pass's marks
  for (int v = t; v < n; v += nt) {
    float l = (k & 1) ? a.buffer[v] : a.labels[v];
    const int g = a.gt[v];
    if (g == 0) l = 0.0f;
    else if (g == 1) l = 1.0f;
    a.labels[v] = l;
    if (k > 0) a.affected[v] = a.stamp[v] == static_cast<unsigned>(k) ? 1 : 0;
  }
  if (t == 0) a.out[0] = k;
}

// -------------------------------------- propagation and IrLP on owned rows --
// Graphs whose vertices the blocks can own (owner_pass.cuh) propagate as the
// resident engine does: full-grid passes on rows in shared memory, frontiers of
// up to kSmallFront vertices on one block with rows in registers
// (row_stint.cuh). Larger graphs take prop_kernel above and irlp_kernel below.
//
// Measured against prop_kernel and irlp_kernel, on the same inputs: propagation from
// 1,000 affected vertices of 50,000 (degree 5, 2,000 passes at most) 1.11 against 3.18
// ms, from 50,000 of a million (degree 7, 300 passes at most) 3.99 against 10.8 ms;
// recompute of 100,000 vertices 0.75 against 3.09 ms.
constexpr int kOwnBlock = stint::kThreads;
constexpr int kSmallFront = 512;
constexpr unsigned long long kStintNs = 100000000ull;  // the other blocks wait in a barrier with a 2 s limit

// The caller's arrays as owned passes and stints read them.
struct CsrGraph {
  static constexpr bool kCounts = false;  // nothing here reads visits, nor clears them
  const int *row_ptr, *col;
  const float *val;
  const int *status, *gt;
  int n;
  __device__ int graphs() const { return 1; }
  __device__ int nodes(int) const { return n; }
  __device__ int2 row(int, int v) const { return make_int2(row_ptr[v], row_ptr[v + 1] - row_ptr[v]); }
  __device__ bool active(int, int v) const { return gt[v] < 0 && status[v] == kActive; }
  __device__ bool markable(int, int v) const { return gt[v] < 0; }
  __device__ void entry(int, int at, int &v, float &w) const {
    v = col[at];
    w = val[at];
    if (v >= 0 && status[v] == kDeleted) v = -1;
  }
  template <int N>
  __device__ void entries(int, int start, int first, int step, int len, int (&v)[N], float (&w)[N]) const {
    int st[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = load_if(first + j * step < len, col + start + first + j * step, -1);
#pragma unroll
    for (int j = 0; j < N; ++j)
      w[j] = __int_as_float(
          load_if(first + j * step < len, reinterpret_cast<const int *>(val) + start + first + j * step, 0));
#pragma unroll
    for (int j = 0; j < N; ++j) st[j] = load_if(v[j] >= 0, status + v[j], kDeleted);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (st[j] == kDeleted) v[j] = -1;
  }
  template <int N>
  __device__ unsigned markables(int, const int (&v)[N]) const {
    unsigned can = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) can |= (load_if(v[j] >= 0, gt + v[j], 0) < 0 ? 1u : 0u) << j;
    return can;
  }
};

struct OwnedArgs {
  CsrGraph g;
  float *labels, *buffer;
  int *affected;
  float delta;
  int max_iter;
  unsigned *marks;        // 2 planes, zeroed
  int plane;              // words of a plane: whole tiles
  int *list;              // a small frontier on its way to the first block
  int *small;             // zeroed: see kOut
  SumBarrier *bar;        // zeroed
  unsigned long long timeout_ns;
  int fast_div;
  int smem_bytes;
};
// Words of OwnedArgs::small.
enum { kOutPasses = 0, kOutError = 1, kOutListed = 2, kOutPass = 3, kOutFull = 4, kOutFront = 5, kOutWords = 16 };

__shared__ SumState s_bar;

template <class Mine>
__device__ __forceinline__ bool all_sync(const OwnedArgs &a, Mine mine, unsigned long long &sum) {
  return sum_sync(a.bar, s_bar, &a.small[kOutError], a.timeout_ns, mine, sum);
}
__device__ __forceinline__ bool all_sync(const OwnedArgs &a) {
  unsigned long long sum;
  return all_sync(a, [] { return 0ull; }, sum);
}

// The block's rows; both kernels start with it.
__device__ __forceinline__ owner::Store own_rows(const OwnedArgs &a) {
  const int tid = threadIdx.x;
  const owner::Store s = owner::store(a.smem_bytes, 1, owner::owned_tiles((a.g.n + owner::kTile - 1) / owner::kTile));
  if (tid == 0) s_bar.gen = 0;
  if (s.tiles > 0) {
    owner::Head &h = s.head();
    if (tid == 0) {
      h.pool_used = 0;
      h.first_limit = a.max_iter;
      h.count = h.wide = h.wide_at = 0;
      h.moved = h.steps = 0;
      owner::Local &l = s.graph(0);
      l.lab[0] = a.labels;
      l.lab[1] = a.buffer;
      l.flat = 0;
      l.limit = a.max_iter;
      l.last = -1;
    }
    __syncthreads();
    owner::load(s, a.g);
  }
  return s;
}

// Vertices of the graph as the one-block passes from pass k0 on see them.
struct CsrStint {
  const OwnedArgs &a;
  int k0;
  __device__ void vertex(int, int v, float &even, float &odd, unsigned &meta) const {
    const float l0 = a.labels[v], l1 = a.buffer[v];
    even = k0 & 1 ? l1 : l0;
    odd = k0 & 1 ? l0 : l1;
    const bool active = a.g.active(0, v);
    meta = (active ? stint::kMarkable : 0u) | (a.g.markable(0, v) ? stint::kShown : 0u);
    if (active && a.g.row(0, v).y > kNarrowMax) meta |= stint::kWide;
  }
  __device__ int2 row(int g, int v) const { return a.g.row(g, v); }
  __device__ void entry(int g, int at, int &v, float &w) const { a.g.entry(g, at, v, w); }
};

struct StintShared {
  stint::Cache c;
  unsigned long long start;
};

// Passes from k0 on by the first block alone, over the frontier in a.list;
// leaves the next pass, its frontier's marks and what became of the labels in
// global memory.
__device__ __noinline__ void small_passes(const OwnedArgs &a, int k0, int listed) {
  StintShared &sh = *reinterpret_cast<StintShared *>(owner::g_smem);
  stint::Cache &c = sh.c;
  const int tid = threadIdx.x, warp = tid >> 5;
  const CsrStint gr{a, k0};
  stint::clear(c);
  if (tid == 0) sh.start = global_timer_ns();
  __syncthreads();
  for (int i = tid; i < listed; i += kOwnBlock) stint::seed(c, gr, 0, a.list[i]);
  __syncthreads();
  stint::Row row;
  int j = 0, full = 0;  // stint pass: pass k0 + j
  const int last = a.max_iter - k0;
  for (;;) {
    const int4 ctl = c.ctl;
    if (!stint::goes_on(ctl, j) || j >= last) break;
    if (stint::needs_rows(ctl, j) && !stint::load_rows(c, gr, row, j, a.fast_div != 0)) {
      full = 1;
      break;
    }
    const int ns = stint::short_warps(c), nl = stint::long_warps(c);
    const bool is_long = warp >= stint::kWarps - nl;
    if (warp < ns || is_long) {
      const bool leader = tid == (ns > 0 ? 0 : kOwnBlock - 32);
      auto tick = [&] { return global_timer_ns() - sh.start > kStintNs; };
      const int end = stint::run(c, row, j, last, a.delta, a.fast_div != 0, ns + nl, is_long, leader, tick, false,
                                 [](int, const stint::Row &) {});
      if (leader) c.end = end;
    }
    __syncthreads();  // the warps without rows wait here
    j = c.end;
  }
  const int k = k0 + j;
  __syncthreads();
  if (row.visits != 0 && row.lead) c.meta[row.slot] |= stint::kVisited;
  __syncthreads();
  unsigned *plane = a.marks + (k & 1 ? a.plane : 0);
  int front = 0;
  for (int i = tid; i < stint::kSlots; i += kOwnBlock) {
    if (c.key[i] == stint::kEmptyKey) continue;
    const unsigned meta = c.meta[i];
    const int v = static_cast<int>(c.key[i]);
    if (meta & stint::kVisited) {
      a.labels[v] = c.lab[k0 & 1][i];
      a.buffer[v] = c.lab[(k0 & 1) ^ 1][i];
    }
    if (stint::marked(c, i, j) && (meta & stint::kShown)) {
      plane[v] = 1;
      if (meta & stint::kMarkable) front = 1;
    }
  }
  front = __syncthreads_or(front);
  if (tid == 0) {
    a.small[kOutPass] = k;
    a.small[kOutFull] = full && j < 256;
    a.small[kOutFront] = front;
    a.small[kOutListed] = 0;
  }
}

// The passes on owned rows from k on until the frontier empties, is small or a
// limit is reached; not inlined, for its registers. TILES: see owned passes of
// the engine. -1: the launch has to end.
template <bool TILES>
__device__ __noinline__ int large_passes(const OwnedArgs &a, owner::Store s, int k, int small_from, bool &empty) {
  owner::Head &h = s.head();
  // in shared memory: the launch's arguments are memory here
  __syncthreads();
  if (threadIdx.x == 0) {
    h.marks = a.marks;
    h.plane = a.plane;
    h.delta = a.delta;
    h.fast = a.fast_div;
    h.budget = a.max_iter;
    h.solo_from = small_from;
    h.bar = a.bar;
    h.err = &a.small[kOutError];
    h.timeout_ns = a.timeout_ns;
  }
  __syncthreads();
  unsigned before = 0xffffffffu;
  for (;;) {
    if (s.tiles > 0) {
      unsigned *own = h.marks + (k & 1 ? h.plane : 0u), *next = h.marks + (k & 1 ? 0u : h.plane);
      auto each = [](int) {};
      if (TILES) owner::tile_pass(s, a.g, own, next, k, h.delta, h.fast != 0, each);
      else owner::pass(s, a.g, own, next, k, h.delta, h.fast != 0, each);
    }
    unsigned long long sum;
    const bool ok = sum_sync(h.bar, s_bar, h.err, h.timeout_ns, [&]() -> unsigned long long {
      if (s.tiles == 0) return 0ull;
      const unsigned long long mine =
          static_cast<unsigned>((h.count & 0xffff) + (h.count >> 16) + h.wide) | (h.moved ? kSumMoved : 0ull);
      h.count = h.wide = h.wide_at = 0;
      h.moved = 0;
      return mine;
    }, sum);
    if (!ok) return -1;
    ++k;
    const unsigned rows = static_cast<unsigned>(sum);
    empty = (sum & (0xffull * kSumMoved)) == 0;
    if (empty || k >= h.budget) return k;
    if (max(rows, before) <= kSmallFront && k >= h.solo_from) return k;
    before = rows;
  }
}

// src/iterativePropagation.cu:241-346 in one cooperative launch of a block per
// SM. The marks of the last pass run stay in the plane of the pass after it:
// they are the final isAffected.
__global__ void __launch_bounds__(kOwnBlock, 1) prop_owned_kernel(const __grid_constant__ OwnedArgs a) {
  const int tid = threadIdx.x, n = a.g.n;
  const int t = blockIdx.x * kOwnBlock + tid, nt = gridDim.x * kOwnBlock;
  const owner::Store s = own_rows(a);
  // both buffers start at the current labels (src/iterativePropagation.cu:268-270);
  // the first frontier (:63-78)
  int seeds = 0;
  for (int v = t; v < n; v += nt) {
    a.buffer[v] = a.labels[v];
    if (a.affected[v] == 1 && a.g.active(0, v)) {
      a.marks[v] = 1;
      ++seeds;
    }
  }
  __shared__ int s_seeds;
  if (tid == 0) s_seeds = 0;
  __syncthreads();
  if (seeds) atomicAdd(&s_seeds, seeds);
  unsigned long long sum;
  if (!all_sync(a, [&] { return static_cast<unsigned long long>(s_seeds); }, sum)) return;
  int k = 0, small_from = 0;
  unsigned rows = static_cast<unsigned>(sum);
  bool empty = rows == 0, try_small = rows <= kSmallFront;
  while (!empty && k < a.max_iter) {
    if (try_small) {
      // the marks of pass k become a list (bounded: a frontier larger than
      // thought goes back to the owned rows), the first block runs it
      unsigned *own = a.marks + (k & 1 ? a.plane : 0);
      for (int i = tid; i < s.n(); i += kOwnBlock) {
        const unsigned v = owner::flat_of(i);
        const bool marked = v < static_cast<unsigned>(n) && __ldcg(own + v) != 0;
        const bool front = marked && owner::kind_of(s, i, k) != 3;
        warp_append(front, static_cast<int>(v), a.list, &a.small[kOutListed]);
      }
      if (!all_sync(a)) return;
      const int listed = ld_relaxed_i32(&a.small[kOutListed]);
      if (listed <= kSmallFront) {
        // pass k is the first block's: its marks go
        for (int i = tid; i < s.n(); i += kOwnBlock) {
          const unsigned v = owner::flat_of(i);
          if (v < static_cast<unsigned>(n) && __ldcg(own + v) != 0) own[v] = 0;
        }
        if (!all_sync(a)) return;  // before it leaves marks of its own
        if (blockIdx.x == 0) small_passes(a, k, listed);
        if (!all_sync(a)) return;
        k = ld_relaxed_i32(&a.small[kOutPass]);
        empty = ld_relaxed_i32(&a.small[kOutFront]) == 0;
        if (ld_relaxed_i32(&a.small[kOutFull])) small_from = k + 256;
      } else {
        if (!all_sync(a)) return;  // every block has read the count
        if (t == 0) a.small[kOutListed] = 0;
      }
      try_small = false;  // at least one pass on the owned rows
      continue;
    }
    const bool tiles = s.n() <= kOwnBlock && s.head().steps <= owner::kTileSteps;
    k = tiles ? large_passes<true>(a, s, k, small_from, empty) : large_passes<false>(a, s, k, small_from, empty);
    if (k < 0) return;
    try_small = true;
  }
  // final labels in the primary array, ground truth enforced
  // (src/iterativePropagation.cu:330-339); isAffected holds the last pass's marks
  const float *lab = (k & 1) ? a.buffer : a.labels;
  const unsigned *plane = a.marks + (k & 1 ? a.plane : 0);
  for (int v = t; v < n; v += nt) {
    float l = lab[v];
    const int g = a.g.gt[v];
    if (g == 0) l = 0.0f;
    else if (g == 1) l = 1.0f;
    a.labels[v] = l;
    if (k > 0) a.affected[v] = __ldcg(plane + v) != 0;
  }
  if (t == 0) a.small[kOutPasses] = k;
}

// src/validation.cu:47-139 and :169-197 on owned rows: every active vertex
// takes its neighbours' average per pass, until no label moves by more than
// delta. The others are copied through by the reference, ground truth as 0 / 1:
// pass 0 reads the caller's labels as they are and its result has the copies, so
// these are written into the buffer before pass 0 and, ground truth, into the
// primary array during pass 1.
__global__ void __launch_bounds__(kOwnBlock, 1) irlp_owned_kernel(const __grid_constant__ OwnedArgs a) {
  const int n = a.g.n;
  const int t = blockIdx.x * kOwnBlock + threadIdx.x, nt = gridDim.x * kOwnBlock;
  const owner::Store s = own_rows(a);
  auto fixed = [&](int v) {
    const int g = a.g.gt[v];
    return g == 0 ? 0.0f : (g == 1 ? 1.0f : a.labels[v]);
  };
  for (int v = t; v < n; v += nt)
    if (!a.g.active(0, v)) a.buffer[v] = fixed(v);
  if (s.tiles > 0) {
    __syncthreads();
    owner::list_all(s);
  }
  int k = 0;
  while (k < a.max_iter) {
    if (k == 1)
      for (int v = t; v < n; v += nt)
        if (a.g.gt[v] == 0 || a.g.gt[v] == 1) a.labels[v] = fixed(v);
    if (s.tiles > 0) owner::dense_pass(s, a.g, k, a.delta);
    unsigned long long sum;
    if (!all_sync(a, [&]() -> unsigned long long {
          if (s.tiles == 0) return 0ull;
          const unsigned long long mine = s.head().moved ? kSumMoved : 0ull;
          s.head().moved = 0;
          return mine;
        }, sum))
      return;
    ++k;
    if ((sum & (0xffull * kSumMoved)) == 0) break;
  }
  // the result is the buffer written last; make it the primary array
  if (k & 1)
    for (int v = t; v < n; v += nt) a.labels[v] = __ldcg(a.buffer + v);
  if (t == 0) a.small[kOutPasses] = k;
}

// ------------------------------------------------------------------ IrLP ---
struct IrlpArgs {
  const int *row_ptr, *col;
  const float *val;
  float *labels, *buffer;
  const int *status, *gt;
  int n;
  float delta;
  int max_iter;
  int *flags;  // [3] changed per pass (triple buffered), [4] passes
  GridBarrier *bar;
  int *err;
  unsigned long long timeout_ns;
};

// src/validation.cu:47-139 and :169-197 in one cooperative launch: all
// vertices every pass; ground truth and inactive vertices are copied through
// (ground truth re-imposed as 0/1); stop after a pass with no move > delta.
__global__ void __launch_bounds__(kBlock) irlp_kernel(IrlpArgs a) {
  constexpr int G = 8;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31, gwarp = t >> 5, nwarps = nt >> 5;
  const int grp = lane / G, gl = lane & (G - 1);
  if (ld_relaxed_i32(a.err) != 0) return;
  int k = 0;
  for (; k < a.max_iter; ++k) {
    const float *src = (k & 1) ? a.buffer : a.labels;
    float *dst = (k & 1) ? a.labels : a.buffer;
    // flags[k%3] is read right after this pass's barrier; flags[(k+1)%3] was
    // last read after barrier k-2, which every block has left
    if (t == 0) a.flags[(k + 1) % 3] = 0;
    bool changed = false;
    for (int base = gwarp * (32 / G); base < a.n; base += nwarps * (32 / G)) {
      const int u = base + grp;
      const bool valid = u < a.n;
      bool compute = false;
      int rs = 0, len = 0;
      if (valid) {
        compute = a.gt[u] < 0 && a.status[u] == kActive;
        if (compute) {
          rs = a.row_ptr[u];
          len = a.row_ptr[u + 1] - rs;
        }
      }
      // one uniform path per warp: long rows fall back to a serial walk by
      // the group (still in the reference's slot order via warp_row_sums below)
      const bool any_long = __any_sync(0xffffffffu, len > kNarrowMax);
      float tw = 0.0f, tl = 0.0f;
      auto load = [&](int e, int &v, float &w) {
        v = a.col[rs + e];
        w = a.val[rs + e];
        if (v >= 0 && a.status[v] == kDeleted) v = -1;
      };
      if (!any_long) {
        int cols[32 / G];
        group_row_sums<G>(len, gl, load, src, tw, tl, cols);
      } else {
        // each group's row in turn, by the whole warp
        for (int q = 0; q < 32 / G; ++q) {
          const int uq = __shfl_sync(0xffffffffu, u, q * G);
          const int rq = __shfl_sync(0xffffffffu, rs, q * G);
          const int lq = __shfl_sync(0xffffffffu, len, q * G);
          auto lq_load = [&](int e, int &v, float &w) {
            v = a.col[rq + e];
            w = a.val[rq + e];
            if (v >= 0 && a.status[v] == kDeleted) v = -1;
          };
          float w1, l1;
          warp_row_sums(lq, lane, lq_load, src, w1, l1);
          (void)uq;
          const float w1b = __shfl_sync(0xffffffffu, w1, 0);
          const float l1b = __shfl_sync(0xffffffffu, l1, 0);
          if (grp == q) {
            tw = w1b;
            tl = l1b;
          }
        }
      }
      if (valid && gl == 0) {
        if (!compute) {
          const int g = a.gt[u];
          dst[u] = g == 0 ? 0.0f : (g == 1 ? 1.0f : src[u]);
        } else {
          const float old = src[u];
          const float nl = updated_label(tw, tl, old);
          dst[u] = nl;
          if (fabsf(nl - old) > a.delta) changed = true;
        }
      }
    }
    if (__any_sync(0xffffffffu, changed) && lane == 0) a.flags[k % 3] = 1;
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
    if (ld_relaxed_i32(&a.flags[k % 3]) == 0) {
      ++k;
      break;
    }
  }
  // the result is the buffer written last; make it the primary array
  if (k & 1)
    for (int v = t; v < a.n; v += nt) a.labels[v] = a.buffer[v];
  if (t == 0) a.flags[4] = k;
}

// Blocks of a step kernel: SMs of the current device at most, queried once per
// device; 0 when the launch is not possible.
int step_blocks() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> known[kMaxDevices];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int sms = known[dev].load(std::memory_order_relaxed);
  if (sms == 0) {
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    sms = std::min(sms, kSumBlocks);
    known[dev].store(sms, std::memory_order_relaxed);
  }
  return sms;
}

// Blocks of a step over `items`, 0 with an error.
int step_grid(long long items) {
  constexpr long long kPerBlock = 2048;
  const int most = step_blocks();
  if (most <= 0) fail(DLP_ERR_CUDA, "device query failed");
  return static_cast<int>(std::min<long long>(std::max<long long>((items + kPerBlock - 1) / kPerBlock, 1), most));
}

// One step kernel over `items`: clears its scratch (one block does it itself,
// step_begin), launches it, waits and returns kStepTotal. `invalid`: what
// DLP_ERR_INVALID_ARGUMENT from the device means.
int run_step(const void *kernel, const char *what, const char *invalid, long long items, void **args, StepScratch *sc,
             int *total, cudaStream_t s) {
  const int grid = step_grid(items);
  if (grid <= 0) return DLP_ERR_CUDA;
  if (grid == 1) {  // no barrier to clear and nothing to be resident with
    DLP_CUDA_TRY(cudaLaunchKernel(kernel, dim3(1), dim3(kStepBlock), args, 0, s));
  } else {
    DLP_CUDA_TRY(cudaMemsetAsync(sc, 0, sizeof(StepScratch), s));
    DLP_TRY(launch_cooperative(kernel, grid, kStepBlock, args, 0, s));
  }
  int host[2] = {0, 0};  // kStepError, kStepTotal
  DLP_CUDA_TRY(cudaMemcpyAsync(host, sc->out, sizeof(host), cudaMemcpyDeviceToHost, s));
  DLP_CUDA_TRY(cudaStreamSynchronize(s));
  if (host[kStepError] == DLP_ERR_INVALID_ARGUMENT) return fail(host[kStepError], invalid);
  if (host[kStepError]) return fail(host[kStepError], std::string(what) + " failed on the device");
  *total = host[kStepTotal];
  return DLP_OK;
}

// Bytes of an owned launch's counters, and of counters and barrier, in scratch.
constexpr size_t kOwnedSmall = 256, kOwnedFixed = 256 + sizeof(SumBarrier);
static_assert(sizeof(int) * kOutWords <= kOwnedSmall && kOwnedFixed % 16 == 0, "scratch layout");

// What the owned kernels' launches need to know of the device.
struct OwnedShape {
  int grid = 0;                // 0: the kernels do not fit this device
  size_t fixed = 0, smem = 0;  // static shared memory, the most of the dynamic one
};

// Sets the kernels' attributes, which a context loses.
OwnedShape ask_owned_shape(int dev) {
  OwnedShape s;
  int sms = 0, most = 0;
  bool ok = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess;
  const void *const kernels[] = {reinterpret_cast<const void *>(&prop_owned_kernel),
                                 reinterpret_cast<const void *>(&irlp_owned_kernel)};
  for (const void *kernel : kernels) {
    cudaFuncAttributes fa{};
    ok = ok && cudaFuncGetAttributes(&fa, kernel) == cudaSuccess;
    s.fixed = std::max(s.fixed, fa.sharedSizeBytes);
  }
  s.smem = (static_cast<size_t>(most) - s.fixed) & ~static_cast<size_t>(15);
  for (const void *kernel : kernels) {
    int per_sm = 0;
    ok = ok && s.smem >= sizeof(StintShared) && s.smem >= owner::bytes_of(1, owner::kMaxVertices / owner::kTile) &&
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(s.smem)) ==
             cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kOwnBlock, s.smem) == cudaSuccess &&
         per_sm > 0;
  }
  s.grid = ok ? std::min(sms, kSumBlocks) : 0;
  cudaGetLastError();
  return s;
}

OwnedShape owned_shape() {
  OwnedShape s;
  if (!with_context([&](ContextFacts &f, int dev) {
        if (!f.shape_asked) {
          const OwnedShape asked = ask_owned_shape(dev);
          f.owned_grid = asked.grid;
          f.owned_fixed = asked.fixed;
          f.owned_smem = asked.smem;
          f.shape_asked = true;
        }
        s.grid = f.owned_grid;
        s.fixed = f.owned_fixed;
        s.smem = f.owned_smem;
      })) {
    int dev = -1;
    if (cudaGetDevice(&dev) == cudaSuccess) s = ask_owned_shape(dev);
  }
  return s;
}

// Blocks that own a graph of n vertices, 0 when they cannot.
int owned_grid(int n) {
  const OwnedShape s = owned_shape();
  return s.grid > 1 && n <= (s.grid - 1) * (owner::kMaxVertices - owner::kTile) ? s.grid : 0;
}

// Shared memory that describes a block's share of n vertices, and the dynamic
// shared memory of a launch over them.
size_t owned_need(int n) {
  const size_t tiles = (static_cast<size_t>(n) + owner::kTile - 1) / owner::kTile, blocks = owned_shape().grid - 1;
  return owner::bytes_of(1, (tiles + blocks - 1) / blocks);
}
size_t owned_smem(int n) {
  const OwnedShape s = owned_shape();
  return owner::smem_of(owned_need(n), sizeof(StintShared), s.fixed, s.smem);
}

// Whether a recompute of n vertices runs on owned rows: as long as L1 keeps more than
// its last 28 KB. 30 passes over 3.5 million vertices, milliseconds: 7.5 on owned
// rows with it and 12.7 without, 10.1 with irlp_kernel.
bool irlp_owned(int n) { return owned_grid(n) > 0 && owner::leaves_l1(owned_need(n), owned_shape().fixed); }

// Words of a mark plane of n vertices: whole tiles.
int owned_plane(int n) { return (n + owner::kTile - 1) / owner::kTile * owner::kTile; }

OwnedArgs owned_args(const int *row_ptr, const int *col, const float *val, float *labels, float *buffer,
                     const int *status, const int *gt, int n, float delta, int max_iterations) {
  OwnedArgs a{};
  a.g = CsrGraph{row_ptr, col, val, status, gt, n};
  a.labels = labels;
  a.buffer = buffer;
  a.delta = delta;
  a.max_iter = max_iterations;
  a.plane = owned_plane(n);
  a.timeout_ns = 2000000000ull;
  a.smem_bytes = static_cast<int>(owned_smem(n));
  return a;
}

PropArgs prop_args(const int *row_ptr, const int *col, const float *val, float *labels, float *buffer,
                   const int *status, const int *gt, int *affected, int n, float delta, int max_iterations) {
  PropArgs a{};
  a.row_ptr = row_ptr;
  a.col = col;
  a.val = val;
  a.labels = labels;
  a.buffer = buffer;
  a.status = status;
  a.gt = gt;
  a.affected = affected;
  a.n = n;
  a.delta = delta;
  a.max_iter = max_iterations;
  a.fast_div = g_launcher_arith.load();
  return a;
}

int clear_scratch(void *p, size_t bytes, cudaStream_t s) {
  DLP_CUDA_TRY(cudaMemsetAsync(p, 0, bytes, s));
  return DLP_OK;
}

// Launches an owned kernel, waits for it and returns its pass count.
int launch_owned(const void *kernel, const OwnedArgs &a, int *passes, cudaStream_t s) {
  OwnedArgs args = a;
  void *list[] = {&args};
  DLP_TRY(launch_cooperative(kernel, owned_shape().grid, kOwnBlock, list, a.smem_bytes, s));
  int host[2] = {0, 0};  // kOutPasses, kOutError
  DLP_CUDA_TRY(cudaMemcpyAsync(host, a.small, sizeof(host), cudaMemcpyDeviceToHost, s));
  DLP_CUDA_TRY(cudaStreamSynchronize(s));
  if (host[kOutError]) return fail(host[kOutError], "propagation failed on the device");
  *passes = host[kOutPasses];
  return DLP_OK;
}

int coop_grid(const void *kernel) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0) != cudaSuccess || per_sm <= 0) {
    cudaGetLastError();
    return -1;
  }
  return sms * per_sm;
}

// Scratch of prop_kernel: `fixed` (kOwnedFixed bytes) holds counters and barrier,
// `words` (3n) the stamps and the lists. Launches it, waits and returns its pass count.
int run_lists(PropArgs a, char *fixed, unsigned *words, int *passes, cudaStream_t s) {
  constexpr size_t kCounters = 64;  // bytes: 16 words
  static_assert(kCounters + sizeof(GridBarrier) <= kOwnedFixed, "scratch layout");
  const size_t n = static_cast<size_t>(a.n);
  // both buffers start at the current labels (src/iterativePropagation.cu:268-270)
  DLP_CUDA_TRY(cudaMemcpyAsync(a.buffer, a.labels, sizeof(float) * n, cudaMemcpyDeviceToDevice, s));
  DLP_TRY(clear_scratch(fixed, kOwnedFixed, s));
  DLP_TRY(clear_scratch(words, sizeof(unsigned) * n, s));
  int *small = reinterpret_cast<int *>(fixed);
  a.counts = small;  // [0..5]
  a.out = small + 8;
  a.err = small + 12;
  a.bar = reinterpret_cast<GridBarrier *>(fixed + kCounters);
  a.stamp = words;
  a.lists = reinterpret_cast<int *>(words + n);
  a.timeout_ns = 2000000000ull;
  const void *kern = reinterpret_cast<const void *>(&prop_kernel);
  const int grid = coop_grid(kern);
  if (grid <= 0) return fail(DLP_ERR_CUDA, "occupancy query failed");
  void *args[] = {&a};
  DLP_TRY(launch_cooperative(kern, grid, kBlock, args, 0, s));
  int host[5] = {0, 0, 0, 0, 0};  // out[0] and, four words on, err
  DLP_CUDA_TRY(cudaMemcpyAsync(host, a.out, sizeof(host), cudaMemcpyDeviceToHost, s));
  DLP_CUDA_TRY(cudaStreamSynchronize(s));
  if (host[4]) return fail(host[4], "propagation failed on the device");
  *passes = host[0];
  return DLP_OK;
}

}  // namespace
}  // namespace ref_layout
}  // namespace dlp

using namespace dlp::ref_layout;

// ---------------------------------------------------------------------------
// Scratch of dlp_iterative_propagation_noalloc: the counters, the barrier and three
// words for each of at most kNoAllocMaxNodes vertices (two planes of frontier marks
// and a list; over lists, stamps and two lists): 12 MiB and less than 1 KiB. It is a
// file-scope device array, so it exists on every GPU that loads this library,
// from module load until the process exits, whether or not the entry point is
// ever called.
namespace {
constexpr int kNoAllocMaxNodes = 1 << 20;
struct NoAllocScratch {
  char fixed[kOwnedFixed];  // counters and barrier, directly before the marks: cleared with them
  unsigned words[3 * kNoAllocMaxNodes];
};
}  // namespace

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

namespace {
// The array's device address, looked up once per context (the host-side name of a
// __device__ variable is not a device address).
int noalloc_scratch(NoAllocScratch **out) {
  void *p = nullptr;
  cudaError_t e = cudaSuccess;
  if (!with_context([&](ContextFacts &f, int) {
        if (!f.scratch) e = cudaGetSymbolAddress(&f.scratch, g_noalloc_scratch);
        p = f.scratch;
      }))
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return dlp::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
  *out = static_cast<NoAllocScratch *>(p);
  return DLP_OK;
}
}  // namespace

extern "C" {

int dlp_set_launcher_arithmetic(int arithmetic) {
  dlp::clear_error();
  if (arithmetic != DLP_ARITH_IEEE && arithmetic != DLP_ARITH_REFERENCE_FAST_MATH)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "arithmetic must be DLP_ARITH_IEEE or DLP_ARITH_REFERENCE_FAST_MATH");
  g_launcher_arith.store(arithmetic);
  return DLP_OK;
}

int dlp_mark_deletions(int *d_row_ptr, int *d_col_ind, int *d_vertex_status, int *d_is_affected,
                       const int *d_deleted_nodes, int num_deleted, int num_nodes, void *stream) {
  dlp::clear_error();
  if (num_deleted == 0) return DLP_OK;  // src/sparsifySubgraph.cu:188
  if (num_deleted < 0 || num_nodes <= 0 || !d_row_ptr || !d_vertex_status || !d_is_affected || !d_deleted_nodes)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_mark_deletions");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  mark_deleted_rows<<<grid_for(static_cast<long long>(num_deleted) * kGroup, kBlock), kBlock, 0, s>>>(
      d_row_ptr, d_col_ind, d_vertex_status, d_is_affected, d_deleted_nodes, num_deleted, num_nodes);
  DLP_CUDA_TRY(cudaGetLastError());
  clean_incoming<<<grid_for(num_nodes, kBlock), kBlock, 0, s>>>(
      d_row_ptr, d_col_ind, d_vertex_status, num_nodes);
  DLP_CUDA_TRY(cudaGetLastError());
  return DLP_OK;
}

int dlp_build_sparsified_subgraph(int *d_row_ptr, int *d_col_ind, float *d_values, int *d_is_affected,
                                  const int *d_vertex_status, const int *d_new_edge_src, const int *d_new_edge_dst,
                                  const float *d_new_edge_weight, int num_new_edges, const int *d_inserted_nodes,
                                  int num_inserted, const int *d_is_new_vertex, float tau, int *d_sub_row_ptr,
                                  int *d_sub_col_ind, float *d_sub_values, int *num_sub_nodes, int *num_sub_edges,
                                  void *stream) {
  (void)d_row_ptr;
  (void)d_col_ind;
  (void)d_values;
  (void)d_vertex_status;
  (void)d_inserted_nodes;
  (void)d_sub_row_ptr;  // never written by the reference either
  dlp::clear_error();
  if (!num_sub_nodes || !num_sub_edges) return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "null outputs");
  *num_sub_nodes = num_inserted;
  *num_sub_edges = 0;
  if (num_new_edges == 0) return DLP_OK;  // src/sparsifySubgraph.cu:213-217
  if (num_new_edges < 0 || !d_new_edge_src || !d_new_edge_dst || !d_new_edge_weight || !d_is_new_vertex ||
      !d_is_affected || !d_sub_col_ind || !d_sub_values)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_build_sparsified_subgraph");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // The reference's signature carries no vertex count, so endpoints can only be
  // checked for being non-negative; the endpoint marks are clipped to ids below
  // numInserted, the numNodes the reference passes there (src/sparsifySubgraph.cu:263).
  const int n_guard = 0x7fffffff;
  StepScratch *sc = nullptr;
  DLP_TRY(tmp_alloc(&sc, 1, s));
  SparsifyArgs a{d_new_edge_src, d_new_edge_dst, d_new_edge_weight, num_new_edges, d_is_new_vertex, n_guard, tau};
  int mark_limit = num_inserted;
  void *args[] = {&a, &sc, &d_is_affected, &mark_limit, &d_sub_col_ind, &d_sub_values};
  int total = 0;
  const int st = run_step(reinterpret_cast<const void *>(&sparsify_kernel), "sparsification",
                          "edge endpoint out of range", num_new_edges, args, sc, &total, s);
  cudaFreeAsync(sc, s);
  DLP_TRY(st);
  *num_sub_edges = total;
  return DLP_OK;
}

int dlp_connected_components(const int *d_edge_src, const int *d_edge_dst, int num_edges,
                             const int *d_inserted_nodes, int num_inserted, int *d_component_id,
                             int *num_components, int num_nodes, void *stream) {
  dlp::clear_error();
  if (!num_components) return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "null num_components");
  if (num_inserted == 0) {  // src/connectedComponents.cu:167-170
    *num_components = 0;
    return DLP_OK;
  }
  if (num_inserted < 0 || num_edges < 0 || num_nodes <= 0 || !d_inserted_nodes || !d_component_id ||
      (num_edges > 0 && (!d_edge_src || !d_edge_dst)))
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_connected_components");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (num_edges == 0) {
    // src/connectedComponents.cu:191-205: ids left at -1, count = numInserted
    DLP_CUDA_TRY(cudaMemsetAsync(d_component_id, 0xff, sizeof(int) * static_cast<size_t>(num_nodes), s));
    *num_components = num_inserted;
    return DLP_OK;
  }
  const size_t words = (static_cast<size_t>(num_nodes) + 31) / 32;
  char *scratch = nullptr;
  DLP_TRY(tmp_alloc(&scratch, sizeof(StepScratch) + sizeof(int) * (2 * words + num_nodes), s));
  StepScratch *sc = reinterpret_cast<StepScratch *>(scratch);
  CcArgs a{d_edge_src, d_edge_dst, num_edges, d_inserted_nodes, num_inserted, num_nodes, nullptr, d_component_id,
           nullptr, nullptr, sc};
  a.bits = reinterpret_cast<unsigned *>(scratch + sizeof(StepScratch));
  a.prefix = reinterpret_cast<int *>(a.bits + words);
  a.par = a.prefix + words;
  void *args[] = {&a};
  int total = 0;
  const long long items = std::max<long long>(std::max(num_edges, num_inserted), num_nodes / 4);
  const int st = run_step(reinterpret_cast<const void *>(&cc_kernel), "connected components",
                          "connected components failed on the device", items, args, sc, &total, s);
  cudaFreeAsync(scratch, s);
  DLP_TRY(st);
  *num_components = total;
  return DLP_OK;
}

int dlp_label_initialization(const int *d_row_ptr, const int *d_col_ind, const float *d_values, float *d_labels,
                             const int *d_vertex_status, const int *d_component_id, int num_components,
                             const int *d_inserted_nodes, int num_inserted, const int *d_gt_class, int num_nodes,
                             void *stream) {
  (void)d_vertex_status;  // not read by the reference either
  dlp::clear_error();
  if (num_inserted == 0) return DLP_OK;  // src/labelInitialization.cu:155
  if (num_inserted < 0 || num_nodes <= 0 || !d_row_ptr || !d_labels || !d_component_id || !d_inserted_nodes ||
      !d_gt_class)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_label_initialization");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t nc = static_cast<size_t>(std::max(num_components, 1));
  const int grid = step_grid(std::max<long long>(num_inserted, nc));
  if (grid <= 0) return DLP_ERR_CUDA;
  long long *acc = nullptr;
  DLP_TRY(tmp_alloc(&acc, 2 * nc, s));
  const InitArgs a{d_row_ptr,  d_col_ind,        d_values,     d_labels,  d_component_id, num_components,
                   d_gt_class, d_inserted_nodes, num_inserted, num_nodes, acc,            g_launcher_arith.load()};
  cudaError_t e = cudaSuccess;
  if (grid == 1) {
    init_kernel<<<1, kStepBlock, 0, s>>>(a);
    e = cudaGetLastError();
  } else {
    e = cudaMemsetAsync(acc, 0, 2 * nc * sizeof(long long), s);
    if (e == cudaSuccess) {
      init_weights_kernel<<<grid, kStepBlock, 0, s>>>(a);
      init_labels_kernel<<<grid, kStepBlock, 0, s>>>(a);
      e = cudaGetLastError();
    }
  }
  cudaFreeAsync(acc, s);
  DLP_CUDA_TRY(e);
  return DLP_OK;
}

int dlp_iterative_propagation(const int *d_row_ptr, const int *d_col_ind, const float *d_values, float *d_labels,
                              float *d_labels_buffer, const int *d_vertex_status, const int *d_gt_class,
                              int *d_is_affected, int num_nodes, float delta, int max_iterations,
                              int *iterations_used, void *stream) {
  dlp::clear_error();
  if (!iterations_used) return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "null iterations_used");
  *iterations_used = 0;
  if (num_nodes <= 0 || !d_row_ptr || !d_labels || !d_labels_buffer || !d_vertex_status || !d_gt_class ||
      !d_is_affected)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_iterative_propagation");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (owned_grid(num_nodes) > 0) {
    // one block of scratch: counters, barrier, marks (zeroed), list
    const size_t n = static_cast<size_t>(num_nodes);
    char *scratch = nullptr;
    const size_t zeroed = kOwnedFixed + 2 * sizeof(unsigned) * owned_plane(num_nodes);
    DLP_TRY(tmp_alloc(&scratch, zeroed + sizeof(int) * n, s));
    OwnedArgs a = owned_args(d_row_ptr, d_col_ind, d_values, d_labels, d_labels_buffer, d_vertex_status, d_gt_class,
                             num_nodes, delta, max_iterations);
    a.affected = d_is_affected;
    a.fast_div = g_launcher_arith.load();
    a.small = reinterpret_cast<int *>(scratch);
    a.bar = reinterpret_cast<dlp::SumBarrier *>(scratch + kOwnedSmall);
    a.marks = reinterpret_cast<unsigned *>(scratch + kOwnedFixed);
    a.list = reinterpret_cast<int *>(scratch + zeroed);
    int st = clear_scratch(scratch, zeroed, s);
    if (st == DLP_OK) st = launch_owned(reinterpret_cast<const void *>(&prop_owned_kernel), a, iterations_used, s);
    cudaFreeAsync(scratch, s);
    return st;
  }
  char *scratch = nullptr;
  DLP_TRY(tmp_alloc(&scratch, kOwnedFixed + 3 * sizeof(unsigned) * static_cast<size_t>(num_nodes), s));
  const int st = run_lists(prop_args(d_row_ptr, d_col_ind, d_values, d_labels, d_labels_buffer, d_vertex_status,
                                     d_gt_class, d_is_affected, num_nodes, delta, max_iterations),
                           scratch, reinterpret_cast<unsigned *>(scratch + kOwnedFixed), iterations_used, s);
  cudaFreeAsync(scratch, s);
  return st;
}

// dlp_iterative_propagation without any device allocation: the same kernel and
// results, with its scratch in g_noalloc_scratch instead of cudaMallocAsync
// temporaries. For callers that must not allocate device memory while they run
// (a framework that owns the whole device memory pool, a service that reserves
// its memory at start-up so nothing can fail or stall later). The first call
// on a device looks the array's address up; make that call before any stream
// capture. All calls share the one array, so calls that overlap on the GPU
// (other streams, other host threads) race; serialise them. Graphs of more
// than 2^20 vertices are rejected.
int dlp_iterative_propagation_noalloc(const int *d_row_ptr, const int *d_col_ind, const float *d_values,
                                      float *d_labels, float *d_labels_buffer, const int *d_vertex_status,
                                      const int *d_gt_class, int *d_is_affected, int num_nodes, float delta,
                                      int max_iterations, int *iterations_used, void *stream) {
  dlp::clear_error();
  if (!iterations_used) return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "null iterations_used");
  *iterations_used = 0;
  if (num_nodes <= 0 || !d_row_ptr || !d_labels || !d_labels_buffer || !d_vertex_status || !d_gt_class ||
      !d_is_affected)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_iterative_propagation_noalloc");
  if (num_nodes > kNoAllocMaxNodes)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT,
                     "num_nodes " + std::to_string(num_nodes) + " exceeds the allocation-free limit of " +
                         std::to_string(kNoAllocMaxNodes) + " vertices; use dlp_iterative_propagation");
  DLP_TRY(dlp::require_device());
  NoAllocScratch *sc = nullptr;
  DLP_TRY(noalloc_scratch(&sc));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (owned_grid(num_nodes) <= 0)  // a part of a GPU, whose blocks cannot own as many vertices
    return run_lists(prop_args(d_row_ptr, d_col_ind, d_values, d_labels, d_labels_buffer, d_vertex_status, d_gt_class,
                               d_is_affected, num_nodes, delta, max_iterations),
                     sc->fixed, sc->words, iterations_used, s);
  OwnedArgs a = owned_args(d_row_ptr, d_col_ind, d_values, d_labels, d_labels_buffer, d_vertex_status, d_gt_class,
                           num_nodes, delta, max_iterations);
  a.affected = d_is_affected;
  a.fast_div = g_launcher_arith.load();
  char *scratch = reinterpret_cast<char *>(sc);
  a.small = reinterpret_cast<int *>(scratch);
  a.bar = reinterpret_cast<dlp::SumBarrier *>(scratch + kOwnedSmall);
  a.marks = sc->words;
  a.list = reinterpret_cast<int *>(sc->words + 2 * static_cast<size_t>(kNoAllocMaxNodes));
  // what must start at zero: the counters, the barrier and the marks in use
  DLP_TRY(clear_scratch(scratch, kOwnedFixed + 2 * sizeof(unsigned) * owned_plane(num_nodes), s));
  return launch_owned(reinterpret_cast<const void *>(&prop_owned_kernel), a, iterations_used, s);
}

int dlp_irlp(const int *d_row_ptr, const int *d_col_ind, const float *d_values, float *d_labels,
             const int *d_vertex_status, const int *d_gt_class, int num_nodes, float delta, int max_iterations,
             int *iterations_used, void *stream) {
  dlp::clear_error();
  if (!iterations_used) return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "null iterations_used");
  *iterations_used = 0;
  if (num_nodes <= 0 || !d_row_ptr || !d_labels || !d_vertex_status || !d_gt_class)
    return dlp::fail(DLP_ERR_INVALID_ARGUMENT, "invalid arguments to dlp_irlp");
  DLP_TRY(dlp::require_device());
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = static_cast<size_t>(num_nodes);
  if (irlp_owned(num_nodes)) {
    char *scratch = nullptr;
    DLP_TRY(tmp_alloc(&scratch, kOwnedFixed + sizeof(float) * n, s));
    OwnedArgs a = owned_args(d_row_ptr, d_col_ind, d_values, d_labels, reinterpret_cast<float *>(scratch + kOwnedFixed),
                             d_vertex_status, d_gt_class, num_nodes, delta, max_iterations);
    a.small = reinterpret_cast<int *>(scratch);
    a.bar = reinterpret_cast<dlp::SumBarrier *>(scratch + kOwnedSmall);
    int st = clear_scratch(scratch, kOwnedFixed, s);
    if (st == DLP_OK) st = launch_owned(reinterpret_cast<const void *>(&irlp_owned_kernel), a, iterations_used, s);
    cudaFreeAsync(scratch, s);
    return st;
  }
  float *buffer = nullptr;
  int *small = nullptr;
  dlp::GridBarrier *bar = nullptr;
  DLP_TRY(tmp_alloc(&buffer, n, s));
  DLP_TRY(tmp_alloc(&small, 16, s));
  DLP_TRY(tmp_alloc(&bar, 1, s));
  DLP_CUDA_TRY(cudaMemcpyAsync(buffer, d_labels, sizeof(float) * n, cudaMemcpyDeviceToDevice, s));
  DLP_CUDA_TRY(cudaMemsetAsync(small, 0, sizeof(int) * 16, s));
  DLP_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(dlp::GridBarrier), s));
  IrlpArgs a{d_row_ptr, d_col_ind, d_values, d_labels, buffer, d_vertex_status, d_gt_class, num_nodes, delta,
             max_iterations, small, bar, small + 8, 2000000000ull};
  const void *kern = reinterpret_cast<const void *>(&irlp_kernel);
  const int grid = coop_grid(kern);
  if (grid <= 0) return dlp::fail(DLP_ERR_CUDA, "occupancy query failed");
  void *args[] = {&a};
  DLP_TRY(dlp::launch_cooperative(kern, grid, kBlock, args, 0, s));
  int host[2] = {0, 0};
  DLP_CUDA_TRY(cudaMemcpyAsync(&host[0], small + 4, sizeof(int), cudaMemcpyDeviceToHost, s));
  DLP_CUDA_TRY(cudaMemcpyAsync(&host[1], small + 8, sizeof(int), cudaMemcpyDeviceToHost, s));
  DLP_CUDA_TRY(cudaStreamSynchronize(s));
  for (void *p : {static_cast<void *>(buffer), static_cast<void *>(small), static_cast<void *>(bar)})
    cudaFreeAsync(p, s);
  if (host[1]) return dlp::fail(host[1], "IrLP failed on the device");
  *iterations_used = host[0];
  return DLP_OK;
}

}  // extern "C"
