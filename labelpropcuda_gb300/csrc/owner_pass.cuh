// Full-grid propagation passes over owned rows.
//
// Every block but the first owns a share of the launch's vertices (tiles of 32,
// dealt out in turn, all graphs one after the other) and keeps their live rows
// in shared memory for the whole launch. A frontier is a word per vertex in
// global memory, one plane per pass parity. A pass is: read and clear the own
// words, list the set ones in shared memory, run their rows with one
// lane per row of at most 8 entries, four lanes up to 32 and a warp beyond,
// store a word for every neighbour that a moved label marks, barrier. The first
// block owns nothing: it runs the one-block passes and the clock.
//
// What bounds a pass: four trips to L2 in a row (own words, neighbour labels,
// acknowledged stores, barrier). A pass over frontier lists takes twice as
// many (counts, list entry, row start, row, labels, mark atomic, reservation,
// list store, barrier). Static ownership is what saves them: a row needs no
// lookup, a mark no answer, and the list of a block no global counter. On large
// frontiers the scattered stores bound a pass: the GPU takes 173 G a second of
// 4-byte ones over 690,000 vertices and 83 G over 50,000, but 107 G and 47 G of
// single bytes (and 298 G loads), hence words.
//
// Measured, microseconds a pass, owned rows against lists: 5,000 vertices of
// degree 5 3.15 against 5.1, 20,000 of degree 7 3.2 against 6.2, 50,000 of degree
// 5 3.2 against 7.5 to 8.0, 500,000 of degree 7 5.0 against 16.2. A scheduler issues in
// a fifth of its cycles, and warps stand at the pass's barriers for three quarters of
// their time.
//
// Shared memory ends at 24,576 vertices per block (3.7 million on 151). Most rows
// then stay in global memory and a scan reads all words of the graph. The engine
// uses frontier lists beyond 20,320 (engine_kernel.cu), the launchers, whose list
// passes are the slower ones, beyond 24,544.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace dlp {
namespace owner {

constexpr int kTile = 32;                       // vertices of a warp's scan step
constexpr int kMaxVertices = 24576;             // per block
constexpr int kLaneEntries = 8;
constexpr int kLongLanes = 4;
constexpr int kMaxRow = kLaneEntries * kLongLanes;
constexpr unsigned kNoPool = (1u << 15) - 1;    // the row did not fit the pool: read from global memory
constexpr unsigned kUnmarkable = 0x80000000u;   // pool entry: a neighbour that is never marked
constexpr unsigned kNoEntry = 0xffffffffu;      // pool entry: soft-deleted
constexpr int kWideLen = 63, kNoRowLen = 62;    // length codes: longer than 32, not active
constexpr int kMaxStint = 32000;                // passes between two clears of visits (15 bits)
constexpr unsigned short kWideRow = 0x8000;

struct Local {           // a graph of the launch
  float *lab[2];         // [k & 1] is read by launch pass k
  unsigned flat;         // its first vertex among the launch's
  int limit;             // first launch pass its pass limit forbids
  int last;              // last launch pass the block ran a row of it in, -1 none
  unsigned long long edges, visits;  // of the stint
};

struct Head {
  int pool_used;
  int first_limit;       // the smallest limit of the graphs
  int count;             // rows of the pass: short | long << 16
  int wide;              // its rows of more than 32 entries
  int wide_at;           // of them in the list
  int moved;
  int steps;             // the most steps that a tile's rows take a warp (tile_steps)
  // what every pass reads
  unsigned *marks;
  unsigned plane;
  float delta;
  int fast;
  int budget, solo_from, stint_end;
  unsigned solo_entry;
  SumBarrier *bar;
  int *err;
  unsigned long long timeout_ns;
};

// The block's dynamic shared memory: Head, then graph[graphs], kinds[tiles], and
// with V = 32 tiles meta[V], visits[V], list[V], pool[cap]. Named by 32-bit offsets
// from its start, so that a pass keeps no pointers in registers: a register
// spilled there is a trip to L2 in every pass, because the barrier's acquire
// empties L1.
extern __shared__ __align__(16) unsigned char g_smem[];
constexpr int kHeadBytes = (sizeof(Head) + 15) & ~15;
static_assert(sizeof(Local) % 16 == 0, "what follows the graphs stays aligned");

// The active vertices of a tile by the kind of their row, a bit per vertex.
struct alignas(16) Kinds {
  unsigned shorts, longs, wides;
};

struct Store {
  int tiles;     // owned
  int meta_at;   // byte offset of meta[]
  int pool_cap;
  __device__ int n() const { return tiles * kTile; }  // owned vertices
  __device__ Head &head() const { return *reinterpret_cast<Head *>(g_smem); }
  __device__ Local &graph(int i) const { return reinterpret_cast<Local *>(g_smem + kHeadBytes)[i]; }
  __device__ Kinds &kinds(int tile) const {
    return reinterpret_cast<Kinds *>(g_smem + meta_at - static_cast<int>(sizeof(Kinds)) * tiles)[tile];
  }
  // pool offset (15 bits) | length (6 bits: kWideLen, kNoRowLen) | graph (10 bits)
  __device__ unsigned &meta(int i) const { return reinterpret_cast<unsigned *>(g_smem + meta_at)[i]; }
  // passes that updated the row (Graph::kCounts); kWideRow: the pass has listed it
  // as a wide row
  __device__ unsigned short &visits(int i) const {
    return reinterpret_cast<unsigned short *>(g_smem + meta_at + 4 * kTile * tiles)[i];
  }
  // rows of the pass: short from the front, long from the back
  __device__ unsigned short &list(int i) const {
    return reinterpret_cast<unsigned short *>(g_smem + meta_at + 6 * kTile * tiles)[i];
  }
  // {neighbour | kUnmarkable, weight}
  __device__ int2 &pool(int i) const { return reinterpret_cast<int2 *>(g_smem + meta_at + 8 * kTile * tiles)[i]; }
};

__device__ __forceinline__ Store store(int bytes, int graphs, int tiles) {
  const int at = kHeadBytes + graphs * static_cast<int>(sizeof(Local)) + tiles * static_cast<int>(sizeof(Kinds));
  const int room = (bytes - at - 8 * kTile * tiles) / static_cast<int>(sizeof(int2));
  return Store{tiles, at, min(room, static_cast<int>(kNoPool) - kMaxRow)};
}

// Shared memory of a block that owns `tiles` of a launch of `graphs` graphs, less
// the pool.
constexpr size_t bytes_of(size_t graphs, size_t tiles) {
  return kHeadBytes + graphs * sizeof(Local) + tiles * (sizeof(Kinds) + 8 * kTile);
}

// Dynamic shared memory of a block that needs `need` bytes (bytes_of) and in any
// case `least`, beside `fixed` bytes of static shared memory and 1 KB that the
// system keeps; at most `most`. What shared memory takes is taken from L1, in
// steps, and the phases and passes around the rows in shared memory live on
// gathers that L1 has to have lines for: with all of it shared, 28 KB are left. So
// a pool of 16 KB is asked for, the step that holds it is filled, and the last
// step is taken only by what does not fit the one before. Measured, milliseconds,
// all shared against this: 12 batches of 500,000 vertices (degree 7, 300 passes at
// most) 6.65 and 5.62, of a million 9.47 and 8.2, of 2 million 14.5 and 13.0, of
// 2.6 million 16.4 and 15.7; 10 of 2 million with 2 passes 3.34 and 2.8; a
// recompute of 3.5 million (30 passes) 12.7 and 7.5.
constexpr size_t kPoolBytes = 16 << 10, kSystemBytes = 1 << 10;
constexpr size_t kSteps[] = {100 << 10, 132 << 10, 164 << 10, 196 << 10};
constexpr bool leaves_l1(size_t need, size_t fixed) { return need + fixed + kSystemBytes <= kSteps[3]; }
inline size_t smem_of(size_t need, size_t least, size_t fixed, size_t most) {
  const size_t asked = std::max(need + kPoolBytes, least), bound = std::max(need, least);
  size_t bytes = most;
  if (leaves_l1(bound, fixed))
    for (const size_t step : kSteps) {
      bytes = step - fixed - kSystemBytes;
      if (asked <= bytes) break;
    }
  return std::min(bytes, most) & ~static_cast<size_t>(15);
}

__device__ __forceinline__ unsigned pack(unsigned off, int len, int g) {
  return off | (static_cast<unsigned>(len) << 15) | (static_cast<unsigned>(g) << 21);
}
__device__ __forceinline__ unsigned pool_of(unsigned m) { return m & kNoPool; }
__device__ __forceinline__ int len_of(unsigned m) { return static_cast<int>((m >> 15) & 63u); }
__device__ __forceinline__ int graph_of(unsigned m) { return static_cast<int>(m >> 21); }

// Steps of a warp that runs all rows of a tile (tile_rows): 32 short rows, 8 long
// ones or a wide one each. Beyond kTileSteps a block's rows are listed and dealt out to
// all its warps, also where it owns at most 32 vertices per warp: 2,000 vertices of
// degree 100 are a tile a block, whose warp ran 32 rows one after the other while 31
// waited. Measured, 8 batches in milliseconds over lists, always by tiles, and so:
// 2,000 vertices of degree 100 5.3, 10.5 and 2.8; 20,000 of degree 100 5.9, 8.6 and 3.6;
// 5,000 of degree 20 6.9, 3.9 and 3.5; 20,000 of degree 12 13.7, 6.6 and 6.5. (With 4
// steps the last two take 4.1 and 7.1.)
constexpr int kTileSteps = 2;
__device__ __forceinline__ int tile_steps(const Kinds &c) {
  return (c.shorts != 0) + (__popc(c.longs) + 32 / kLongLanes - 1) / (32 / kLongLanes) + __popc(c.wides);
}

// The tiles of the launch are dealt out to the blocks but the first in turn. A
// contiguous range per block would follow the graphs and the vertex ids, and so
// do frontiers: some graphs have converged while others have a quarter of
// their vertices in the frontier, and the first frontier of a batch is at low
// ids. The slowest blocks then ran 1,800 rows a pass where others ran none.
__device__ __forceinline__ int owned_tiles(int tiles) {
  const int b = static_cast<int>(blockIdx.x) - 1, blocks = static_cast<int>(gridDim.x) - 1;
  return b < 0 || b >= tiles ? 0 : (tiles - b - 1) / blocks + 1;
}
// Owned vertex i among the launch's vertices.
__device__ __forceinline__ unsigned flat_of(int i) {
  return (blockIdx.x - 1u + static_cast<unsigned>(i / kTile) * (gridDim.x - 1u)) * kTile +
         static_cast<unsigned>(i % kTile);
}

// Rows of the block's vertices into shared memory (head and graphs filled by
// the caller).
// Graph: kCounts, whether visits and last passes of the rows are kept (their
// reader has to clear them every kMaxStint passes); graphs(); nodes(g); row(g, v) {start, length}; active(g, v): v can be in
// a frontier; markable(g, v): v is marked as a neighbour (every active vertex
// is); entry(g, at, v, w), v = -1 for an entry that does not count; entries<N>(g,
// start, e, step, len, v, w), N of them from start + e on, v = -1 also for those from
// start + len on, and markables<N>(g, v), a bit for each that is markable, both with
// the loads of all N in flight together.
template <class Graph>
__device__ void load(const Store &s, const Graph &gr) {
  const int tid = threadIdx.x, lane = tid & 31;
  Head &h = s.head();
  for (int i = tid; i < s.n(); i += blockDim.x) {
    const unsigned flat = flat_of(i);
    int g = 0;  // the last graph that starts at or before the vertex
    for (int hi = gr.graphs() - 1; g < hi;) {
      const int mid = (g + hi + 1) >> 1;
      if (s.graph(mid).flat <= flat) g = mid;
      else hi = mid - 1;
    }
    const int v = static_cast<int>(flat - s.graph(g).flat);
    int2 ri = make_int2(0, 0);
    const bool active = v < gr.nodes(g) && gr.active(g, v);
    if (active) ri = gr.row(g, v);
    const int len = ri.y;
    // pool room for the warp's rows, one reservation
    const int want = len <= kMaxRow ? len : 0;
    int incl = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    int base = 0;
    if (lane == 31 && incl) base = atomicAdd(&h.pool_used, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    const int off = base + incl - want;
    const bool fits = off + want <= s.pool_cap;
    s.meta(i) = pack(fits ? static_cast<unsigned>(off) : kNoPool, active ? (len > kMaxRow ? kWideLen : len) : kNoRowLen, g);
    s.visits(i) = 0;
    Kinds kinds;
    kinds.shorts = __ballot_sync(0xffffffffu, active && len <= kLaneEntries);
    kinds.longs = __ballot_sync(0xffffffffu, active && len > kLaneEntries && len <= kMaxRow);
    kinds.wides = __ballot_sync(0xffffffffu, active && len > kMaxRow);
    if (lane == 0) {
      s.kinds(i / kTile) = kinds;
      atomicMax(&h.steps, tile_steps(kinds));
    }
    if (!fits) continue;  // lanes of the next round reconverge at its first shuffle
    for (int b = 0; b < want; b += kLaneEntries) {
      int u[kLaneEntries];
      float w[kLaneEntries];
#pragma unroll
      for (int r = 0; r < kLaneEntries; ++r) {
        u[r] = -1;
        w[r] = 0.0f;
        if (b + r < want) gr.entry(g, ri.x + b + r, u[r], w[r]);
      }
      unsigned mk = 0;
#pragma unroll
      for (int r = 0; r < kLaneEntries; ++r)
        if (u[r] >= 0 && gr.markable(g, u[r])) mk |= 1u << r;
#pragma unroll
      for (int r = 0; r < kLaneEntries; ++r)
        if (b + r < want) {
          const bool live = u[r] >= 0;
          const unsigned x = static_cast<unsigned>(u[r]) | ((mk >> r) & 1u ? 0u : kUnmarkable);
          s.pool(off + b + r) = make_int2(static_cast<int>(live ? x : kNoEntry), __float_as_int(live ? w[r] : 0.0f));
        }
    }
  }
}

// The accesses of a row step are predicated, not branched around: a load in a
// branch is waited for before the next one is issued. (A stand-in address that
// all idle lanes share is no way out: its L2 slice cost 3,000 cycles a pass.)
// Pool entry at byte address `at` + OFF of shared memory, kNoEntry with weight 0
// unless `e` < `len`.
template <int OFF>
__device__ __forceinline__ void pool_entry(unsigned at, int e, int len, unsigned &u, float &w) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.lt.s32 p, %3, %4;\n\t"
      "mov.b32 %0, -1;\n\t"
      "mov.f32 %1, 0f00000000;\n\t"
      "@p ld.shared.v2.b32 {%0, %1}, [%2+%5];\n\t"
      "}" : "=&r"(u), "=&f"(w) : "r"(at), "r"(e), "r"(len), "n"(OFF));
}
// The label of entry u from L2, 0 for kNoEntry.
__device__ __forceinline__ float gather(const float *src, unsigned u) {
  float x;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.u32 p, %2, -1;\n\t"
      "mov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.cg.f32 %0, [%1];\n\t"
      "}" : "=&f"(x) : "l"(src + (u & ~kUnmarkable)), "r"(u));
  return x;
}
// Marks entry u if it can be and `moved`.
__device__ __forceinline__ void mark(unsigned *marks, unsigned u, int moved) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.s32 q, %2, 0;\n\t"
      "setp.ge.and.s32 p, %1, 0, q;\n\t"
      "@p st.global.u32 [%0], %3;\n\t"
      "}" ::"l"(marks + (u & ~kUnmarkable)), "r"(u), "r"(moved), "r"(1) : "memory");
}

template <int LANES, int R = 0>
__device__ __forceinline__ void pool_row(unsigned at, int sub, int len, unsigned (&u)[kLaneEntries],
                                         float (&w)[kLaneEntries]) {
  if constexpr (R < kLaneEntries) {
    pool_entry<8 * LANES * R>(at, sub + LANES * R, len, u[R], w[R]);
    pool_row<LANES, R + 1>(at, sub, len, u, w);
  }
}

// The row of owned vertex i by LANES lanes (1: up to 8 entries, 4: up to 32).
// All lanes of the warp call; returns whether the label moved (on every lane of
// the row). MARK: a moved label marks, and (Graph::kCounts) the row's visits are
// counted.
template <int LANES, bool MARK = true, class Graph>
__device__ __forceinline__ bool row(const Store &s, const Graph &gr, bool valid, int i, int k, float delta, bool fast,
                                    unsigned *next) {
  const int sub = threadIdx.x & (LANES - 1);
  const unsigned m = s.meta(i);
  const int len = valid ? len_of(m) : 0, g = graph_of(m);
  const unsigned off = pool_of(m);
  const Local &l = s.graph(g);
  const float *src = l.lab[k & 1];
  const unsigned first = l.flat;
  const unsigned v = flat_of(i) - first;
  const float old = gather(src, valid ? v : kNoEntry);
  unsigned u[kLaneEntries];
  float w[kLaneEntries], x[kLaneEntries];
  pool_row<LANES>(static_cast<unsigned>(__cvta_generic_to_shared(&s.pool(0))) + 8 * (off + sub), sub,
                  off != kNoPool ? len : 0, u, w);
  // Lanes without a row have none to look up either: their vertex may lie after
  // the graph's last one.
  if (valid && off == kNoPool) {
    const int start = gr.row(g, static_cast<int>(v)).x;
#pragma unroll
    for (int r = 0; r < kLaneEntries; ++r) {
      const int e = sub + LANES * r;
      int c = -1;
      if (e < len) gr.entry(g, start + e, c, w[r]);
      if (c < 0) w[r] = 0.0f;
      u[r] = c < 0 ? kNoEntry : static_cast<unsigned>(c);
    }
#pragma unroll
    for (int r = 0; r < kLaneEntries; ++r)
      if (!(u[r] & kUnmarkable) && !gr.markable(g, static_cast<int>(u[r]))) u[r] |= kUnmarkable;
  }
#pragma unroll
  for (int r = 0; r < kLaneEntries; ++r) x[r] = gather(src, u[r]);
#pragma unroll
  for (int r = 0; r < kLaneEntries; ++r) x[r] = __fmaf_rn(w[r], x[r], 0.0f);  // an empty slot: 0 * 0 + 0
  // the reference's tree (row_sums.cuh): strides 16 to 4 within a lane of a
  // long row, 2 and 1 across its lanes; strides 4 to 1 within that of a short
#pragma unroll
  for (int h = kLaneEntries / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int r = 0; r < h; ++r) {
      x[r] = x[r] + x[r + h];
      w[r] = w[r] + w[r + h];
    }
  float tl = x[0], tw = w[0];
#pragma unroll
  for (int o = LANES / 2; o >= 1; o >>= 1) {
    tl = tl + __shfl_xor_sync(0xffffffffu, tl, o);
    tw = tw + __shfl_xor_sync(0xffffffffu, tw, o);
  }
  const float recip = label_recip(tw, fast);
  float nl = label_by_recip(tw, recip, tl);
  if (valid & !recip_serves(recip, tl)) nl = updated_label(tw, tl, old, fast);
  const bool moved = valid & (fabsf(nl - old) > delta);
  unsigned *const marks = next + first;
  if (MARK) {
#pragma unroll
    for (int r = 0; r < kLaneEntries; ++r) mark(marks, u[r], moved);
  }
  if (valid && sub == 0) {
    l.lab[(k & 1) ^ 1][v] = nl;
    if (MARK) {
      if constexpr (Graph::kCounts) {
        ++s.visits(i);
        s.graph(g).last = k;
      }
      mark(marks, v, moved);
    }
  }
  return moved;
}

// A row of more than 32 entries by a warp, from global memory: slots lane + 32 j
// of 256, then the tree. AHEAD entries a lane in flight: with four, a step is three
// trips to L2 (entries, what the caller knows of the neighbours, labels) for 128
// entries; passes over tiles, which have few such rows, have no registers for that.
// The neighbours' marks are set by a reduction: where rows are wide a vertex is
// marked by many of them in one pass, and stores of one word from many SMs took
// longer. 45 passes of a propagation over 20,000 vertices of degree 100 take 1.8 ms
// and 2.4 with stores, 37 over 100,000 of degree 64 4.1 and 4.5; over 2,000 of degree
// 100, one warp's rows at a time, 0.75 and 0.68; a million of degree 40 the same.
template <bool MARK, int AHEAD, class Graph>
__device__ __forceinline__ bool wide_row(const Store &s, const Graph &gr, int i, int k, float delta, bool fast,
                                         unsigned *next) {
  const int lane = threadIdx.x & 31;
  const int lg = graph_of(s.meta(i)), g = lg;
  const Local &l = s.graph(lg);
  const float *src = l.lab[k & 1];
  const int v = static_cast<int>(flat_of(i) - l.flat);
  const int2 ri = gr.row(g, v);
  float sw[8], sl[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sw[j] = sl[j] = 0.0f;
  for (int p = 0; p < ri.y; p += 256) {
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += AHEAD) {
      const int e = p + j0 * 32 + lane;
      if (e - lane >= ri.y) break;
      int u[AHEAD];
      float w[AHEAD], x[AHEAD];
      gr.template entries<AHEAD>(g, ri.x, e, 32, ri.y, u, w);
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) x[j] = gather(src, static_cast<unsigned>(u[j]));
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) {
        sw[j0 + j] = u[j] >= 0 ? sw[j0 + j] + w[j] : sw[j0 + j];
        sl[j0 + j] = u[j] >= 0 ? __fmaf_rn(w[j], x[j], sl[j0 + j]) : sl[j0 + j];
      }
    }
  }
#pragma unroll
  for (int half = 4; half >= 1; half >>= 1)
#pragma unroll
    for (int j = 0; j < half; ++j) {
      sw[j] = sw[j] + sw[j + half];
      sl[j] = sl[j] + sl[j + half];
    }
  float tw = sw[0], tl = sl[0];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    tw = tw + __shfl_xor_sync(0xffffffffu, tw, o);
    tl = tl + __shfl_xor_sync(0xffffffffu, tl, o);
  }
  const float old = __ldcg(src + v);
  const float nl = updated_label(tw, tl, old, fast);
  if (lane == 0) {
    l.lab[(k & 1) ^ 1][v] = nl;
    if constexpr (MARK && Graph::kCounts) {
      ++s.visits(i);
      s.graph(lg).last = k;
    }
  }
  if (!(fabsf(nl - old) > delta)) return false;
  if constexpr (MARK) {
    for (int e = lane; e - lane < ri.y; e += AHEAD * 32) {
      int u[AHEAD];
      float w[AHEAD];
      gr.template entries<AHEAD>(g, ri.x, e, 32, ri.y, u, w);
      const unsigned can = gr.template markables<AHEAD>(g, u);
#pragma unroll
      for (int j = 0; j < AHEAD; ++j)
        if ((can >> j) & 1u) atomicOr(next + l.flat + u[j], 1u);
    }
    if (lane == 0) next[l.flat + v] = 1;
  }
  return true;
}

// Kind of the row of marked vertex i in pass k: 0 short, 1 long, 2 wide, 3 none
// (not active, or past its graph's pass limit).
__device__ __forceinline__ int kind_of(const Store &s, int i, int k) {
  const unsigned m = s.meta(i);
  const int len = len_of(m);
  if (len == kNoRowLen || (k >= s.head().first_limit && k >= s.graph(graph_of(m)).limit)) return 3;
  return len <= kLaneEntries ? 0 : len <= kMaxRow ? 1 : 2;
}

// The rows that a warp's tile runs in pass k of its marked vertices (a bit
// each): all but those past their graph's pass limit. All lanes call.
__device__ __forceinline__ Kinds kinds_of(const Store &s, int tile, unsigned marked, int k) {
  if (k >= s.head().first_limit) {
    const bool past = k >= s.graph(graph_of(s.meta(tile * kTile + (threadIdx.x & 31)))).limit;
    marked &= ~__ballot_sync(0xffffffffu, past);
  }
  Kinds c = s.kinds(tile);
  c.shorts &= marked;
  c.longs &= marked;
  c.wides &= marked;
  return c;
}

// The rows of a warp's tile, vertices first .. first + 31, each lane with the
// kind of its own. Returns whether a label moved, on all lanes.
template <class Graph>
__device__ __forceinline__ bool tile_rows(const Store &s, const Graph &gr, int first, int kind, int k, float delta,
                                          bool fast, unsigned *next) {
  const int lane = threadIdx.x & 31;
  bool moved = false;
  if (__any_sync(0xffffffffu, kind == 0))
    moved = row<1>(s, gr, kind == 0, first + lane, k, delta, fast, next);
  unsigned longs = __ballot_sync(0xffffffffu, kind == 1), wides = __ballot_sync(0xffffffffu, kind == 2);
  while (longs) {  // 8 at a time, the q-th remaining one to the q-th lanes
    unsigned m = longs;
    for (int q = lane / kLongLanes; q > 0 && m; --q) m &= m - 1;
    moved |= row<kLongLanes>(s, gr, m != 0, first + __ffs(m ? m : longs) - 1, k, delta, fast, next);
    for (int q = 32 / kLongLanes; q > 0 && longs; --q) longs &= longs - 1;
  }
  for (; wides; wides &= wides - 1)
    moved |= wide_row<true, 1>(s, gr, first + __ffs(wides) - 1, k, delta, fast, next);
  return __any_sync(0xffffffffu, moved);
}

// A pass of a block that owns at most 32 vertices per warp: every warp runs the
// marked rows of its own tile, without a list and without waiting for the
// others.
template <class Graph, class Each>
__device__ __forceinline__ void tile_pass(const Store &s, const Graph &gr, unsigned *own, unsigned *next, int k,
                                          float delta, bool fast, Each each) {
  const int lane = threadIdx.x & 31, i = threadIdx.x;
  const bool marked = i < s.n() && __ldcg(own + flat_of(i)) != 0;
  if (!__any_sync(0xffffffffu, marked)) return;
  int kind = 3;
  if (marked) {
    own[flat_of(i)] = 0;
    kind = kind_of(s, i, k);
    if (kind != 3) each(i);
  }
  const bool moved = tile_rows(s, gr, i - lane, kind, k, delta, fast, next);
  const int rows = __popc(__ballot_sync(0xffffffffu, kind != 3));
  if (lane == 0 && rows) {
    atomicAdd(&s.head().count, rows);
    if (moved) s.head().moved = 1;
  }
}

// The listed rows, dealt out evenly: ns short ones from the first warp up, 32 to
// a warp, nl long ones from the last down, 8 to a warp. A step is some 300
// instructions however many rows it holds, and few full warps issue them sooner
// than many with a row each. Returns whether one of the lane's labels moved.
template <bool MARK, class Graph>
__device__ __forceinline__ bool listed_rows(const Store &s, const Graph &gr, int ns, int nl, int k, float delta,
                                            bool fast, unsigned *next) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  constexpr int kPer = 32 / kLongLanes;
  const int n = s.n(), sub = lane / kLongLanes;
  bool moved = false;
  for (int b = warp * 32; b < ns; b += nwarps * 32) {
    const bool valid = b + lane < ns;
    moved |= row<1, MARK>(s, gr, valid, s.list(valid ? b + lane : b), k, delta, fast, next);
  }
  for (int b = (nwarps - 1 - warp) * kPer; b < nl; b += nwarps * kPer) {
    const bool valid = b + sub < nl;
    moved |= row<kLongLanes, MARK>(s, gr, valid, s.list(n - 1 - (valid ? b + sub : b)), k, delta, fast, next);
  }
  return moved;
}

// Pass k of the block's vertices, up to the barrier. own: this pass's plane;
// next: the plane of the next pass. The rows are
// listed for the whole block and dealt out evenly: with every warp on its own
// part of them, the warps with the most marked rows took two to four
// steps where most took one, and every block waits for the slowest.
template <class Graph, class Each>
__device__ __forceinline__ void pass(const Store &s, const Graph &gr, unsigned *own, unsigned *next, int k,
                                     float delta, bool fast, Each each) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  Head &h = s.head();
  const int n = s.n();
  // A word per lane, four loads in flight; the set ones are listed with one
  // reservation per warp.
  constexpr int kAhead = 4;
  for (int base = warp * 32; base < n; base += kAhead * nwarps * 32) {
    unsigned b[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int i = base + j * nwarps * 32 + lane;
      b[j] = i < n ? __ldcg(own + flat_of(i)) : 0;
    }
    unsigned shorts[kAhead], longs[kAhead];
    int add = 0;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      shorts[j] = longs[j] = 0;
      const unsigned marked = __ballot_sync(0xffffffffu, b[j] != 0);
      if (!marked) continue;
      const int i = base + j * nwarps * 32 + lane;
      if (b[j]) own[flat_of(i)] = 0;
      const Kinds c = kinds_of(s, i / kTile, marked, k);
      if (((c.shorts | c.longs | c.wides) >> lane) & 1u) each(i);
      shorts[j] = c.shorts;
      longs[j] = c.longs;
      add += __popc(c.shorts) + (__popc(c.longs) << 16);
      if ((c.wides >> lane) & 1u) {  // listed below
        atomicAdd(&h.wide, 1);
        s.visits(i) |= kWideRow;
      }
    }
    if (add == 0) continue;
    int at = 0;
    if (lane == 0) at = atomicAdd(&h.count, add);
    at = __shfl_sync(0xffffffffu, at, 0);
    int at_short = at & 0xffff, at_long = n - 1 - (at >> 16);
    const unsigned bit = 1u << lane, below = bit - 1u;
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const unsigned short i = static_cast<unsigned short>(base + j * nwarps * 32 + lane);
      if (shorts[j] & bit) s.list(at_short + __popc(shorts[j] & below)) = i;
      if (longs[j] & bit) s.list(at_long - __popc(longs[j] & below)) = i;
      at_short += __popc(shorts[j]);
      at_long -= __popc(longs[j]);
    }
  }
  __syncthreads();
  const int nw = h.wide, ns = h.count & 0xffff, nl = h.count >> 16;
  bool moved = listed_rows<true>(s, gr, ns, nl, k, delta, fast, next);
  if (nw) {  // the room between the short and the long rows holds them
    for (int i = tid; i < n; i += blockDim.x)
      if (s.visits(i) & kWideRow) {
        s.visits(i) &= static_cast<unsigned short>(~kWideRow);
        s.list(ns + atomicAdd(&h.wide_at, 1)) = static_cast<unsigned short>(i);
      }
    __syncthreads();
    for (int q = warp; q < nw; q += nwarps) moved |= wide_row<true, 4>(s, gr, s.list(ns + q), k, delta, fast, next);
  }
  if (__any_sync(0xffffffffu, moved) && lane == 0) h.moved = 1;
}

// All active rows of the block into the list, once (the wide ones behind the short
// ones); then dense_pass runs them (no marks): every active vertex takes the average
// of its neighbours.
__device__ __forceinline__ void list_all(const Store &s) {
  const int lane = threadIdx.x & 31, n = s.n();
  Head &h = s.head();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const Kinds c = s.kinds(i / kTile);
    const int add = __popc(c.shorts) + (__popc(c.longs) << 16);
    int at = 0;
    if (lane == 0 && add) at = atomicAdd(&h.count, add);
    at = __shfl_sync(0xffffffffu, at, 0);
    const unsigned bit = 1u << lane, below = bit - 1u;
    if (c.shorts & bit) s.list((at & 0xffff) + __popc(c.shorts & below)) = static_cast<unsigned short>(i);
    if (c.longs & bit) s.list(n - 1 - (at >> 16) - __popc(c.longs & below)) = static_cast<unsigned short>(i);
  }
  __syncthreads();
  const int ns = h.count & 0xffff;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    if ((s.kinds(i / kTile).wides >> lane) & 1u) s.list(ns + atomicAdd(&h.wide, 1)) = static_cast<unsigned short>(i);
  __syncthreads();
}

template <class Graph>
__device__ __forceinline__ void dense_pass(const Store &s, const Graph &gr, int k, float delta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  Head &h = s.head();
  const int ns = h.count & 0xffff;
  bool moved = listed_rows<false>(s, gr, ns, h.count >> 16, k, delta, false, nullptr);
  for (int q = warp; q < h.wide; q += nwarps)
    moved |= wide_row<false, 4>(s, gr, s.list(ns + q), k, delta, false, nullptr);
  if (__any_sync(0xffffffffu, moved) && lane == 0) h.moved = 1;
}

}  // namespace owner
}  // namespace dlp
