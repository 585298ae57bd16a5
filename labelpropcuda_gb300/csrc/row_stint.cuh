// Propagation passes over a small frontier on one thread block, rows held in
// registers ("row-stationary" passes).
//
// A stint starts from a frontier and runs pass after pass on one block. Every
// row that has been in the frontier during the stint belongs to a lane (up to
// 8 entries) or to four lanes (9 to 32 entries), which keep its weights and
// the shared-memory slots of its neighbours in registers. The labels of all
// vertices seen (two buffers) and a mark per vertex and pass parity live in
// shared memory. A pass is then: read the own row's mark; if set, gather the
// neighbour labels, form the sum in the reference's order, divide, store the
// new label; if it moved by more than delta, store a mark for the neighbours
// and the row itself; barrier. There are no frontier lists: the next frontier
// is the set of marks, a mark is a plain store (all writers store the same
// value), and only the warps that hold rows take part in the barrier.
//
// What bounds a pass: the dependent chain labels -> sum -> division -> stores
// -> barrier on one or two warps per scheduler, and the issue slots and bank
// conflicts beyond. Measured with every row marked: 324 cycles for 32 rows of 5
// entries (1 warp, 81 instructions: 148 cycles of arithmetic latency, 47 of
// branches, 22 of barrier), 389 for 128 (4 warps), 565 for 256 (8), 1,001 for 500
// (16); with four rows of 12 entries among 32, 389. One lane per short row is
// the shortest chain, because its sum needs no shuffles.
//
// The stint ends when the frontier empties, when a row longer than 32 entries
// is marked, when the rows no longer fit the block's lanes or the vertices the
// table, at a pass limit, on request, or when the rows of the last 512 passes
// would fit half of the warps or fewer (the caller starts another one, whose
// rows are packed: rows are never given up within a stint, and every warp that
// holds one takes part in each pass). Nothing of the arithmetic depends on
// where a row sits: slot order and summation tree are those of row_sums.cuh,
// and the weight sum of a row, which cannot change during a stint, is formed
// once when the row is loaded.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace dlp {
namespace stint {

constexpr int kThreads = kBlockThreads;    // threads of the block that runs a stint
constexpr int kWarps = kThreads / 32;
constexpr int kSlots = 4096;               // vertex-table slots (power of two)
constexpr int kSlotsUse = kSlots * 7 / 8;  // in use at most (linear probing stays short below this)
constexpr int kEntries = 8;                // row entries a lane holds
constexpr int kLongLanes = 4;              // lanes of a row of 9 to 32 entries
constexpr int kMaxRow = kEntries * kLongLanes;
constexpr int kPad = kSlots;               // slot of an empty entry: label 0, never owned
constexpr int kIdle = kSlots + 1;          // slot of a lane without a row: never marked
constexpr int kRepack = 512;               // passes between two looks at the rows in use (power of two)
constexpr int kEager = 8;                  // up to this many warps, every lane gathers before its mark is known
constexpr unsigned short kNoRow = 0xffff;
constexpr unsigned long long kEmptyKey = ~0ull;
// Cache::meta bits. kMarkable: can be in the frontier. kShown: not read here
// (what else the caller wants to know about a marked vertex).
constexpr unsigned kMarkable = 1, kWide = 2, kOwned = 4, kVisited = 8, kSwapped = 16, kShown = 32;

struct Cache {
  unsigned long long key[kSlots];  // (graph << 32) | vertex, kEmptyKey = free
  float lab[2][kSlots + 4];        // [j & 1] is read by stint pass j
  int mark[2][kSlots + 4];         // [j & 1]: j + 1 where a vertex is marked for stint pass j (see marked())
  unsigned char meta[kSlots + 4];
  unsigned short place[kThreads];  // slot of the row of each thread, kNoRow = none
  unsigned short list[kThreads];   // rows to load
  // Stamps, stint pass + 1: {the last pass with a frontier, the last one whose
  // frontier holds a vertex without a row here (or with one too long), the first
  // one that must not run}. They only grow (the third only shrinks), so a thread
  // still at the top of pass j reads the same verdict from what pass j writes for
  // pass j + 1, and nothing has to be cleared.
  alignas(16) int4 ctl;
  int used;                        // vertex-table slots in use
  int overflow;                    // a load found no room
  int num_short, num_long;         // rows held, by kind
  int pending;                     // entries of list
  int recent;                      // lanes whose row took part in the last kRepack passes
  int end;                         // first stint pass the last run did not take
};

// A lane's share of a row. Slots are shared-memory addresses of their lab[0]
// entry; lab[1] and the marks of the slot lie at fixed distances from it.
struct Row {
  float w[kEntries];
  unsigned at[kEntries];  // the neighbours
  unsigned own;           // the row's vertex
  float total = 0.0f;     // the row's weight sum
  float recip = 0.0f;     // its reciprocal, 0 where quotients take the general division
  int slot = kIdle;       // the row's vertex (kIdle: the lane holds no row)
  int len = 0;
  bool open = false;     // a neighbour it can mark has no row here
  bool lead = false;     // the lane that reports the row
  unsigned visits = 0;   // passes that updated the row
  int last = -1;         // the last of them (stint pass)
};

__device__ __forceinline__ unsigned shared_address(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// The multiplier is that of the finaliser of MurmurHash3 (A. Appleby, public domain).
__device__ __forceinline__ unsigned mix64(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  return static_cast<unsigned>(x);
}

// Slot of (g, v), inserted when absent (fresh: the caller fills it); -1 when
// the table is full.
__device__ __forceinline__ int insert(Cache &c, int g, int v, bool &fresh) {
  const unsigned long long key = (static_cast<unsigned long long>(g) << 32) | static_cast<unsigned>(v);
  unsigned h = mix64(key) & (kSlots - 1);
  fresh = false;
  for (int probe = 0; probe < kSlots; ++probe) {
    const unsigned long long prev = atomicCAS(&c.key[h], kEmptyKey, key);
    if (prev == kEmptyKey) {
      fresh = true;
      if (atomicAdd(&c.used, 1) >= kSlotsUse) c.overflow = 1;
      return static_cast<int>(h);
    }
    if (prev == key) return static_cast<int>(h);
    if (*const_cast<volatile int *>(&c.overflow)) return -1;
    h = (h + 1) & (kSlots - 1);
  }
  c.overflow = 1;
  return -1;
}

// Loads vertex (g, v) into its fresh slot h. Graph::vertex gives the label that
// stint pass 0 reads, the one it does not, and the meta bits.
template <class Graph>
__device__ __forceinline__ void fill(Cache &c, const Graph &gr, int h, int g, int v) {
  float a, b;
  unsigned meta;
  gr.vertex(g, v, a, b, meta);
  c.lab[0][h] = a;
  c.lab[1][h] = b;
  c.mark[0][h] = 0;
  c.mark[1][h] = 0;
  c.meta[h] = static_cast<unsigned char>(meta);
}

__device__ __forceinline__ void clear(Cache &c) {
  const int tid = threadIdx.x;
  for (int i = tid; i < kSlots; i += kThreads) c.key[i] = kEmptyKey;
  c.place[tid] = kNoRow;
  if (tid == 0) c.ctl = make_int4(0, 0, 0x7fffffff, 0);
  if (tid < 2) {
    for (int p = 0; p < 2; ++p) {
      c.lab[p][kPad + tid] = 0.0f;
      c.mark[p][kPad + tid] = 0;
    }
    c.meta[kPad + tid] = 0;
  }
  if (tid == 0) {
    c.used = 0;
    c.overflow = 0;
    c.num_short = 0;
    c.num_long = 0;
    c.recent = 0;
  }
}

// Whether slot h is marked for stint pass j; marks are not cleared, their value
// says for which pass they are.
__device__ __forceinline__ bool marked(const Cache &c, int h, int j) { return c.mark[j & 1][h] == j + 1; }

// A vertex of the stint's first frontier (pass 0), by one thread.
template <class Graph>
__device__ __forceinline__ void seed(Cache &c, const Graph &gr, int g, int v) {
  bool fresh;
  const int h = insert(c, g, v, fresh);
  if (h < 0) return;
  if (fresh) fill(c, gr, h, g, v);
  c.mark[0][h] = 1;
  c.ctl.x = 1;
  c.ctl.y = 1;
}

__device__ __forceinline__ int short_warps(const Cache &c) { return (c.num_short + 31) / 32; }
__device__ __forceinline__ int long_warps(const Cache &c) {
  return (c.num_long + 32 / kLongLanes - 1) / (32 / kLongLanes);
}

// What the control words say about stint pass j: its frontier is not empty and
// no request ends the stint; and whether rows have to be loaded first.
__device__ __forceinline__ bool goes_on(const int4 &ctl, int j) { return ctl.x > j && ctl.z > j + 1; }
__device__ __forceinline__ bool needs_rows(const int4 &ctl, int j) { return ctl.y == j + 1; }

// Gives every marked vertex of stint pass j without a row a place and loads
// its row. Short rows fill the lanes from warp 0 up, long rows those from the
// last warp down, so a warp holds one kind. All threads of the block call;
// false: a row is too long or there is no room (the stint has to end here; the
// marks are unchanged).
template <class Graph>
__device__ bool load_rows(Cache &c, const Graph &gr, Row &row, int j, bool fast) {
  const unsigned lab0 = shared_address(c.lab[0]);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) c.pending = 0;
  __syncthreads();  // the control words have been read by every thread
  if (tid == 0) c.ctl.y = 0;
  for (int i = tid; i < kSlots; i += kThreads) {
    if (c.key[i] == kEmptyKey || !marked(c, i, j) || (c.meta[i] & (kMarkable | kOwned)) != kMarkable) continue;
    const int at = atomicAdd(&c.pending, 1);
    if (at < kThreads) c.list[at] = static_cast<unsigned short>(i);
  }
  __syncthreads();
  const int count = c.pending;
  if (count > kThreads) return false;
  int slot = kIdle, index = 0;
  bool is_short = false;
  if (tid < count) {
    slot = c.list[tid];
    const unsigned long long key = c.key[slot];
    const int len = gr.row(static_cast<int>(key >> 32), static_cast<int>(key)).y;
    if (len > kMaxRow) {
      c.overflow = 1;
    } else {
      is_short = len <= kEntries;
      index = atomicAdd(is_short ? &c.num_short : &c.num_long, 1);
    }
  }
  __syncthreads();
  if (c.overflow || short_warps(c) + long_warps(c) > kWarps) return false;
  if (slot != kIdle) {
    c.meta[slot] |= kOwned;
    if (is_short) {
      c.place[index] = static_cast<unsigned short>(slot);
    } else {
      constexpr int kPerWarp = 32 / kLongLanes;
      const int first = (kWarps - 1 - index / kPerWarp) * 32 + (index % kPerWarp) * kLongLanes;
      for (int i = 0; i < kLongLanes; ++i) c.place[first + i] = static_cast<unsigned short>(slot);
    }
  }
  __syncthreads();
  const bool is_long = warp >= kWarps - long_warps(c);
  const bool mine = row.slot == kIdle && c.place[tid] != kNoRow;
  if (__any_sync(0xffffffffu, mine)) {
    float tw = 0.0f;
    if (mine) {
      row.slot = c.place[tid];
      row.own = lab0 + row.slot * 4;
      row.lead = !is_long || (lane & (kLongLanes - 1)) == 0;
      const unsigned long long key = c.key[row.slot];
      const int g = static_cast<int>(key >> 32);
      const int2 ri = gr.row(g, static_cast<int>(key));
      row.len = ri.y;
      int v[kEntries];
#pragma unroll
      for (int r = 0; r < kEntries; ++r) {
        const int e = is_long ? (lane & (kLongLanes - 1)) + kLongLanes * r : r;
        v[r] = -1;
        row.w[r] = 0.0f;
        if (e < ri.y) gr.entry(g, ri.x + e, v[r], row.w[r]);
        if (v[r] < 0) row.w[r] = 0.0f;
      }
      unsigned fresh = 0;
#pragma unroll
      for (int r = 0; r < kEntries; ++r) {
        bool f = false;
        int h = kPad;
        if (v[r] >= 0) {
          h = insert(c, g, v[r], f);
          if (h < 0) h = kPad;
        }
        row.at[r] = lab0 + h * 4;
        if (f) fresh |= 1u << r;
      }
#pragma unroll
      for (int r = 0; r < kEntries; ++r)
        if ((fresh >> r) & 1u) fill(c, gr, static_cast<int>(row.at[r] - lab0) / 4, g, v[r]);
      float s[kEntries];
#pragma unroll
      for (int r = 0; r < kEntries; ++r) s[r] = row.w[r];
#pragma unroll
      for (int h = kEntries / 2; h >= 1; h >>= 1)
#pragma unroll
        for (int r = 0; r < h; ++r) s[r] = s[r] + s[r + h];
      tw = s[0];
    }
    if (is_long) {
#pragma unroll
      for (int o = kLongLanes / 2; o >= 1; o >>= 1) tw = tw + __shfl_xor_sync(0xffffffffu, tw, o);
    }
    if (mine) {
      row.total = tw;
      row.recip = label_recip(tw, fast);
    }
  }
  __syncthreads();
  if (c.overflow) return false;
  row.open = false;
  if (row.slot != kIdle) {
#pragma unroll
    for (int r = 0; r < kEntries; ++r)
      if ((c.meta[(row.at[r] - lab0) / 4] & (kMarkable | kOwned)) == kMarkable) row.open = true;
  }
  return true;
}

constexpr unsigned kPlane = sizeof(float) * (kSlots + 4);  // lab[0], lab[1], mark[0], mark[1] in a row

// Shared-memory accesses of a pass, with the plane as an immediate and in
// program order: the loads of a pass have to be in flight together, and an
// address addition per access would be a fifth of the pass's instructions.
template <unsigned PLANE>
__device__ __forceinline__ float ld(unsigned a) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(x) : "r"(a), "n"(PLANE * kPlane));
  return x;
}
__device__ __forceinline__ int4 ld4(unsigned a) {
  int4 x;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(a));
  return x;
}

// Stint pass j of parity P by a warp that holds rows; false, with nothing done,
// when the pass must not run. Eager: all lanes gather at once, whether or not
// their row is marked, so that the mark, the labels and the control words are
// one shared-memory latency and nothing branches; the other form reads the marks
// first, which costs a latency and saves the gathers of warps without a marked
// row. Stores are predicated, not branched around: with one or two warps per
// scheduler a branch costs as much as four dependent additions.
template <int P, bool EAGER>
__device__ __forceinline__ bool pass(Row &row, unsigned control, bool is_long, int last, float delta, bool fast,
                                     int j) {
  const int4 ctl = ld4(control);
  const float mark = ld<2 + P>(row.own);
  float x[kEntries], old = 0.0f;
  if (EAGER) {
    old = ld<P>(row.own);
#pragma unroll
    for (int r = 0; r < kEntries; ++r) x[r] = ld<P>(row.at[r]);
  }
  const bool go = goes_on(ctl, j) & !needs_rows(ctl, j) & (j < last);
  const bool act = go & (__float_as_int(mark) == j + 1);
  if (!EAGER) {
    if (!__any_sync(0xffffffffu, act)) return go;
#pragma unroll
    for (int r = 0; r < kEntries; ++r) x[r] = 0.0f;
    if (act) {
      old = ld<P>(row.own);
#pragma unroll
      for (int r = 0; r < kEntries; ++r) x[r] = ld<P>(row.at[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < kEntries; ++r) x[r] = __fmaf_rn(row.w[r], x[r], 0.0f);
#pragma unroll
  for (int h = kEntries / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int r = 0; r < h; ++r) x[r] = x[r] + x[r + h];
  float tl = x[0];
  if (is_long) {
    // the sum of four lanes: every lane gets the tree's value, because
    // floating-point addition commutes
#pragma unroll
    for (int o = kLongLanes / 2; o >= 1; o >>= 1) tl = tl + __shfl_xor_sync(0xffffffffu, tl, o);
  }
  float nl = label_by_recip(row.total, row.recip, tl);
  if (act & !recip_serves(row.recip, tl)) nl = updated_label(row.total, tl, old, fast);
  const bool moved = act & (fabsf(nl - old) > delta);
  row.visits += act ? 1u : 0u;
  row.last = act ? j : row.last;
  // The label; and where it moved, marks of pass j + 1 for the row and its
  // neighbours (ground-truth neighbours and empty entries too: nothing owns
  // them, and a load or the end of the stint leaves them out) and the control
  // words.
  asm volatile(
      "{\n\t"
      ".reg .pred pa, pm, po;\n\t"
      "setp.ne.s32 pa, %0, 0;\n\t"
      "setp.ne.s32 pm, %1, 0;\n\t"
      "setp.ne.and.s32 po, %2, 0, pm;\n\t"
      "@pa st.shared.f32 [%3+%15], %4;\n\t"
      "@pm st.shared.b32 [%6+%14], %5;\n\t"
      "@pm st.shared.b32 [%7+%14], %5;\n\t"
      "@pm st.shared.b32 [%8+%14], %5;\n\t"
      "@pm st.shared.b32 [%9+%14], %5;\n\t"
      "@pm st.shared.b32 [%10+%14], %5;\n\t"
      "@pm st.shared.b32 [%11+%14], %5;\n\t"
      "@pm st.shared.b32 [%12+%14], %5;\n\t"
      "@pm st.shared.b32 [%13+%14], %5;\n\t"
      "@pm st.shared.b32 [%3+%14], %5;\n\t"
      "@pm st.shared.b32 [%16], %5;\n\t"
      "@po st.shared.b32 [%16+4], %5;\n\t"
      "}" ::"r"(static_cast<int>(act)),
      "r"(static_cast<int>(moved)), "r"(static_cast<int>(row.open)), "r"(row.own), "f"(nl), "r"(j + 2),
      "r"(row.at[0]), "r"(row.at[1]), "r"(row.at[2]), "r"(row.at[3]), "r"(row.at[4]), "r"(row.at[5]),
      "r"(row.at[6]), "r"(row.at[7]), "n"((2 + (P ^ 1)) * kPlane), "n"((P ^ 1) * kPlane), "r"(control)
      : "memory");
  return go;
}

// Stint passes from j to last - 1 at most, by the warps that hold rows; returns
// the first one not run. Every exit reads words written before the last
// barrier, so all warps leave together. tick() is called by the leader every 64
// passes and returns whether the stint has to end; record(j, row), when RECORD,
// by every thread in every pass.
//
// Not inlined, on a copy of the row: the loop then has the thread's registers
// to itself (inlined, it spilled).
template <bool EAGER, bool RECORD, class Tick, class Record>
__device__ __noinline__ int run_as(Cache &c, Row &kept, int j, int last, float delta, bool fast, int warps,
                                   bool is_long, bool leader, Tick tick, Record record) {
  Row row = kept;
  const unsigned control = shared_address(&c.ctl);
  auto step = [&](auto parity) {
    constexpr int P = decltype(parity)::value;
    if (RECORD) record(j, row);
    if (!pass<P, EAGER>(row, control, is_long, last, delta, fast, j)) return false;
    if (P == 1 && (j & 63) == 63) {
      const int at = j & (kRepack - 1);
      if (leader) {
        // lanes in use during the kRepack passes up to 64 passes ago
        const bool repack = at == 63 && j > kRepack && 2 * (c.recent / 32 + 2) <= warps;
        if (at == 63) c.recent = 0;
        if (tick() || repack) asm volatile("st.shared.b32 [%0+8], %1;" ::"r"(control), "r"(j + 2) : "memory");
      }
      if (at == kRepack - 1) {
        const int used = __popc(__ballot_sync(0xffffffffu, row.slot != kIdle && row.last > j - kRepack));
        if ((threadIdx.x & 31) == 0 && used) atomicAdd(&c.recent, used);
      }
    }
    asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
    ++j;
    return true;
  };
  using Even = std::integral_constant<int, 0>;
  using Odd = std::integral_constant<int, 1>;
  if (!(j & 1) || step(Odd{}))
    while (step(Even{}) && step(Odd{})) {
    }
  kept.visits = row.visits;
  kept.last = row.last;
  return j;
}

template <class Tick, class Record>
__device__ __forceinline__ int run(Cache &c, Row &row, int j, int last, float delta, bool fast, int warps,
                                   bool is_long, bool leader, Tick tick, bool recorded, Record record) {
  if (row.slot == kIdle) {  // a lane without a row gathers from the pad and is never marked
    const unsigned lab0 = shared_address(c.lab[0]);
    row.own = lab0 + kIdle * 4;
#pragma unroll
    for (int r = 0; r < kEntries; ++r) {
      row.at[r] = lab0 + kPad * 4;
      row.w[r] = 0.0f;
    }
  }
  if (recorded) return run_as<false, true>(c, row, j, last, delta, fast, warps, is_long, leader, tick, record);
  if (warps <= kEager) return run_as<true, false>(c, row, j, last, delta, fast, warps, is_long, leader, tick, record);
  return run_as<false, false>(c, row, j, last, delta, fast, warps, is_long, leader, tick, record);
}

}  // namespace stint
}  // namespace dlp
