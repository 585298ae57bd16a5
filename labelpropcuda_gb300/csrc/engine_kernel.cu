// The multi-graph batch engine kernel (see engine.cuh). One cooperative
// persistent launch applies one batch to each listed graph; the phases and
// their arithmetic are the single-graph ones (session_kernel.cuh), each walking
// a work list flattened over all graphs.
//
// Arithmetic that must agree bit for bit with the CPU oracle:
//   * a row's weighted average follows the reference's summation order (slot
//     t of a 256-slot block accumulates entries t, t+256, ...; weight by add,
//     weighted label by FMA; tree with strides 128..1,
//     src/iterativePropagation.cu:126-150). A row of at most 32 entries only
//     adds +0 at strides 128..32, so a group of G lanes holding slots lane+G*r
//     reproduces it exactly; longer rows take a warp holding lane+32*j.
//   * division is IEEE round-to-nearest (__fdiv_rn; or, with
//     dlp_config.arithmetic = 1, the reference's fast-math division);
//     built with -fmad=false.
//   * supernode weights are exact 32.32 fixed-point sums (order independent).
#include "engine.cuh"
#include "owner_pass.cuh"
#include "row_stint.cuh"

namespace dlp {
namespace engine {
namespace {

using session::BatchArgs;
using session::BatchCounters;
using session::DevState;
using session::kBlock;
using session::kMaxHookRounds;
using session::kNarrowMax;
using session::kRecordIters;
using session::kRowGroup;

struct Ctx {
  int gtid, nthreads, lane, gwarp, nwarps;
};

__device__ __forceinline__ Ctx make_ctx() {
  Ctx c;
  c.gtid = blockIdx.x * blockDim.x + threadIdx.x;
  c.nthreads = gridDim.x * blockDim.x;
  c.lane = threadIdx.x & 31;
  c.gwarp = c.gtid >> 5;
  c.nwarps = c.nthreads >> 5;
  return c;
}

__device__ __forceinline__ bool in_range(int v, int n) {
  return static_cast<unsigned>(v) < static_cast<unsigned>(n);
}

// One graph's state and batch as a phase sees them.
struct GV {
  const DevState &s;
  const BatchArgs &a;
  unsigned cur;  // this batch's stamp for deleted / GT / dirty marks
  unsigned g0;   // this batch's first frontier stamp

  __device__ bool inserted_now(int v) const {
    const int p = s.local[v];
    return p >= 0 && p < a.I && a.ins[p] == v;
  }
  // ref: a vertex inserted and deleted in one batch is DELETED for that batch
  __device__ bool dev_deleted(int v) const { return !a.spec && s.del_stamp[v] == cur; }
  // live in the host rebuild of this batch (src/dynLP.cu:143-157)
  __device__ bool live(int v) const {
    if (s.status[v] == kDeleted) return false;
    if (s.batch_map) {
      const int m = s.batch_map[v];
      if (m < 0 || m > a.batch) return false;
    }
    return true;
  }
  __device__ bool comp_path() const { return a.spec ? (a.I > 0) : (a.I > 0 && a.E > 0); }
};

__device__ __forceinline__ GV view(const EngineArgs &e, int g) {
  const GraphRec &r = e.recs[g];
  return GV{r.st, r.ba, static_cast<unsigned>(r.ba.seq) + 1u, r.st.ctl->stamp_base + 1u};
}

// ------------------------------------------------------- launch barrier ----
__shared__ SumState s_bar;
__shared__ int s_bad;  // this block found invalid input

// All blocks of the launch; false when the launch has to end.
__device__ __forceinline__ bool launch_sync(const EngineArgs &e) {
  unsigned long long sum;
  return sum_sync(&e.ectl->bar, s_bar, &e.ectl->err, e.timeout_ns, [] { return s_bad ? kSumError : 0ull; }, sum);
}

// ----------------------------------------------------------- warp helpers --
// Reserves one slot per predicated lane in the list whose counter is `count`;
// lanes of one warp may target different counters (different graphs).
// Called by all 32 lanes. Returns the slot, or -1 for lanes without pred.
__device__ __forceinline__ int reserve_keyed(bool pred, int *count) {
  const unsigned act = __ballot_sync(0xffffffffu, pred);
  if (!pred) return -1;
  const unsigned peers = __match_any_sync(act, reinterpret_cast<unsigned long long>(count));
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

__device__ __forceinline__ void append_keyed(bool pred, int value, int *list, int *count) {
  const int slot = reserve_keyed(pred, count);
  if (slot >= 0) list[slot] = value;
}

__device__ __forceinline__ void append_back_keyed(bool pred, int value, int *list, int cap, int *count) {
  const int slot = reserve_keyed(pred, count);
  if (slot >= 0) list[cap - 1 - slot] = value;
}

// Adds v into *dst once per group of lanes sharing dst (all 32 lanes call).
__device__ __forceinline__ void add_keyed(bool pred, unsigned v, unsigned long long *dst) {
  const unsigned act = __ballot_sync(0xffffffffu, pred && v != 0);
  if (!(pred && v != 0)) return;
  const unsigned peers = __match_any_sync(act, reinterpret_cast<unsigned long long>(dst));
  const unsigned sum = __reduce_add_sync(peers, v);
  if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(dst, static_cast<unsigned long long>(sum));
}

// ------------------------------------------------------ flattened lists ----
// Exclusive prefix of per-graph counts in shared memory (all block threads
// call; the counts must read the same global values in every block).
template <class F>
__device__ int flat_build(int *pref, int ng, F count) {
  __shared__ int s_warp[kBlock / 32];
  __syncthreads();
  if (ng == 1) {
    if (threadIdx.x == 0) {
      pref[0] = 0;
      pref[1] = count(0);
    }
    __syncthreads();
    return pref[1];
  }
  constexpr int kPer = (kMaxGraphs + kBlock - 1) / kBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int vals[kPer];
  int local = 0;
  const int start = threadIdx.x * kPer;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int g = start + j;
    vals[j] = g < ng ? count(g) : 0;
    local += vals[j];
  }
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int x = lane < kBlock / 32 ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < kBlock / 32) s_warp[lane] = x;
  }
  __syncthreads();
  int run = incl - local + (warp > 0 ? s_warp[warp - 1] : 0);
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int g = start + j;
    if (g < ng) pref[g] = run;
    run += vals[j];
  }
  if (threadIdx.x == kBlock - 1) pref[ng] = run;
  __syncthreads();
  return pref[ng];
}

// Largest g with pref[g] <= item: the graph that owns work item `item`.
__device__ __forceinline__ int locate(const int *pref, int ng, int item) {
  int lo = 0, hi = ng - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pref[mid] <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Group-of-kRowGroup items over a flattened list; every lane of a warp runs
// the same number of iterations so warp collectives stay legal.
template <class F>
__device__ __forceinline__ void flat_groups(const Ctx &c, const int *pref, int ng, int total, F fn) {
  constexpr int GPW = 32 / kRowGroup;
  const int grp = c.lane / kRowGroup, gl = c.lane & (kRowGroup - 1);
  for (int base = c.gwarp * GPW; base < total; base += c.nwarps * GPW) {
    const int item = base + grp;
    const bool valid = item < total;
    const int g = valid ? locate(pref, ng, item) : 0;
    fn(g, valid ? item - pref[g] : 0, valid, gl, grp);
  }
}

// Per-thread items over a flattened list, warp-uniform trip count.
template <class F>
__device__ __forceinline__ void flat_threads(const Ctx &c, const int *pref, int ng, int total, F fn) {
  for (int base = c.gwarp * 32; base < total; base += c.nwarps * 32) {
    const int item = base + c.lane;
    const bool valid = item < total;
    const int g = valid ? locate(pref, ng, item) : 0;
    fn(g, valid ? item - pref[g] : 0, valid);
  }
}

// Seed mark: the batch's first stamp; the first mark appends to the seed list.
__device__ __forceinline__ void seed_mark(const GV &w, bool cand, int v) {
  bool first = false;
  if (cand) first = atomicMax(&w.s.front_stamp[v], w.g0) < w.g0;
  append_keyed(first, v, w.s.seed_list, &w.s.bc->num_seeds);
}

// Frontier append into set `set` (narrow rows from the front, wide from the
// back) and, the first time in this batch, into the touched list.
__device__ __forceinline__ void frontier_append(const GV &w, bool pred, bool first, int v, int set) {
  const DevState &s = w.s;
  bool wide = false;
  if (pred) wide = s.act_len[v] > kNarrowMax;
  int *list = s.flist + static_cast<size_t>(set) * s.n;
  append_keyed(pred && !wide, v, list, &s.bc->front_count[set][0]);
  append_back_keyed(pred && wide, v, list, s.n, &s.bc->front_count[set][1]);
  append_keyed(first, v, s.touched + static_cast<size_t>(w.a.seq & 1) * s.n, &s.ctl->touched_count[w.a.seq & 1]);
}

// ---------------------------------------------------------------- phase A ---
// Position map, stamps, input validation, label-buffer re-sync at the vertices
// the previous batch's propagation wrote (both buffers start a batch equal,
// src/dynLP.cu:519 and src/iterativePropagation.cu:268-270).
__device__ void phase_a(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  auto prev_touched = [&](int g) {
    const GraphRec &r = e.recs[g];
    return r.ba.seq > 0 ? r.st.ctl->touched_count[(r.ba.seq - 1) & 1] : 0;
  };
  const int total = flat_build(pref, ng, [&](int g) {
    const BatchArgs &a = e.recs[g].ba;
    return a.I + a.D + a.G + a.E + prev_touched(g);
  });
  int bad = 0;
  for (int item = c.gtid; item < total; item += c.nthreads) {
    const int g = locate(pref, ng, item);
    int i = item - pref[g];
    const GV w = view(e, g);
    const DevState &s = w.s;
    const BatchArgs &a = w.a;
    const int n = s.n;
    if (i < a.I) {
      const int v = a.ins[i];
      if (!in_range(v, n)) { bad = 1; continue; }
      s.local[v] = i;
      s.par[i] = i;
      s.acc[2 * i] = 0;
      s.acc[2 * i + 1] = 0;
      if (a.record) s.rec_minid[i] = 0x7fffffff;
      continue;
    }
    i -= a.I;
    if (i < a.D) {
      const int v = a.del[i];
      if (!in_range(v, n)) { bad = 1; continue; }
      if (a.spec) s.del_pre[i] = s.status[v];
      s.del_stamp[v] = w.cur;
      continue;
    }
    i -= a.D;
    if (i < a.G) {
      const int v = a.gt_ids[i];
      if (!in_range(v, n)) { bad = 1; continue; }
      s.gt_stamp[v] = w.cur;
      continue;
    }
    i -= a.G;
    if (i < a.E) {
      if (!in_range(a.es[i], n) || !in_range(a.ed[i], n)) bad = 1;
      continue;
    }
    i -= a.E;
    const int cb = s.ctl->cur_buf;
    const int v = s.touched[static_cast<size_t>((a.seq - 1) & 1) * n + i];
    (cb ? s.lab0 : s.lab1)[v] = (cb ? s.lab1 : s.lab0)[v];
  }
  for (int g = c.gtid; g < ng; g += c.nthreads) {
    const GraphRec &r = e.recs[g];
    r.st.ctl->touched_count[r.ba.seq & 1] = 0;
  }
  if (bad) {
    atomicCAS(&e.ectl->err, 0, DLP_ERR_INVALID_ARGUMENT);
    s_bad = 1;
  }
}

// ---------------------------------------------------------------- phase B ---
// Host-status update (ref: delete, insert, then ground truth,
// src/dynLP.cu:117-130; spec: deletions win) and dirty-row marking.
__device__ void phase_b(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  int total = flat_build(pref, ng, [&](int g) {
    const BatchArgs &a = e.recs[g].ba;
    return a.D + a.I + a.G;
  });
  for (int item = c.gtid; item < total; item += c.nthreads) {
    const int g = locate(pref, ng, item);
    int i = item - pref[g];
    const GV w = view(e, g);
    const DevState &s = w.s;
    const BatchArgs &a = w.a;
    if (i < a.D) {
      const int v = a.del[i];
      if (a.spec || (!w.inserted_now(v) && s.gt_stamp[v] != w.cur)) s.status[v] = kDeleted;
      continue;
    }
    i -= a.D;
    if (i < a.I) {
      const int v = a.ins[i];
      if (s.gt_stamp[v] == w.cur) continue;
      if (a.spec && s.del_stamp[v] == w.cur) continue;
      s.status[v] = kActive;
      continue;
    }
    i -= a.I;
    const int v = a.gt_ids[i];
    const float l = a.gt_lab[i];
    s.gt[v] = l < 0.5f ? 0 : 1;
    s.nmeta[v] = s.act_len[v] > kNarrowMax ? 2 : 0;  // not markable any more
    s.lab0[v] = l;
    s.lab1[v] = l;
    if (!(a.spec && s.del_stamp[v] == w.cur)) s.status[v] = kGroundTruth;
  }
  // Rows whose live content can change: every changed vertex and its
  // full-graph neighbours; the previous batch's deletions give a same-batch
  // insert+delete (ref) its row back.
  total = flat_build(pref, ng, [&](int g) {
    const BatchArgs &a = e.recs[g].ba;
    return a.D + a.I + a.PD + a.G;
  });
  flat_groups(c, pref, ng, total, [&](int g, int k, bool valid, int gl, int) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    const BatchArgs &a = w.a;
    int x = -1;
    if (valid) {
      if (k < a.D) x = a.del[k];
      else if ((k -= a.D) < a.I) x = a.ins[k];
      else if ((k -= a.I) < a.PD) x = a.prev_del[k];
      else x = a.gt_ids[k - a.PD];
    }
    const int rs = valid ? s.full_row[x] : 0;
    const int len = valid ? s.full_row[x + 1] - rs : 0;
    const int maxlen = __reduce_max_sync(0xffffffffu, len + 1);  // +1: the vertex itself
    for (int off = 0; off < maxlen; off += kRowGroup) {
      const int ee = off + gl - 1;  // -1: x itself
      int v = -1;
      if (valid && ee < len) v = ee < 0 ? x : s.full_adj[rs + ee].x;
      bool first = false;
      if (v >= 0) first = atomicMax(&s.dirty_stamp[v], w.cur) < w.cur;
      append_keyed(first, v, s.dirty_list, &s.bc->num_dirty);
    }
  });
}

// ---------------------------------------------------------------- phase C ---
// Live-row compaction, deletion marks and the tau filter.
__device__ void phase_c(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  int total = flat_build(pref, ng, [&](int g) { return e.recs[g].st.bc->num_dirty; });
  flat_groups(c, pref, ng, total, [&](int g, int item, bool valid, int gl, int grp) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    int u = 0, rs = 0, len = 0;
    bool keep_row = false, del_row = false;
    if (valid) {
      u = s.dirty_list[item];
      keep_row = w.live(u);
      rs = s.full_row[u];
      len = keep_row ? s.full_row[u + 1] - rs : 0;
      del_row = keep_row && w.dev_deleted(u);
    }
    add_keyed(valid && gl == 0, static_cast<unsigned>(len), &s.bc->dirty_entries);
    const int maxlen = __reduce_max_sync(0xffffffffu, len);
    const unsigned gmask = ((1u << kRowGroup) - 1u) << (grp * kRowGroup);
    int pos = 0;
    for (int off = 0; off < maxlen; off += kRowGroup) {
      const int ee = off + gl;
      bool keep = false;
      int2 ent = make_int2(-1, 0);
      if (ee < len) {
        ent = s.full_adj[rs + ee];
        keep = ent.x >= 0 && w.live(ent.x);
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep) & gmask;
      if (keep) {
        const int rank = __popc(m & ((1u << c.lane) - 1u));
        int col = ent.x;
        // soft delete (src/sparsifySubgraph.cu:78,108): entries of a row deleted
        // this batch and entries pointing at such a vertex
        if (del_row || w.dev_deleted(col)) col = -1;
        s.act_adj[rs + pos + rank] = make_int2(col, ent.y);
      }
      // neighbours of a deleted vertex's live row are affected
      // (src/sparsifySubgraph.cu:71-76; empty unless inserted this batch)
      seed_mark(w, keep && del_row, ent.x);
      pos += __popc(m);
    }
    if (valid && gl == 0) {
      const int len = keep_row ? pos : 0;
      s.act_len[u] = len;
      s.rowinfo[u] = make_int2(rs, len);
      s.nmeta[u] = static_cast<uint8_t>((s.gt[u] < 0 ? 1 : 0) | (len > kNarrowMax ? 2 : 0));
    }
  });

  // spec: neighbours of every deleted vertex that was live before this batch's
  // deletions, in the adjacency before the deletion
  total = flat_build(pref, ng, [&](int g) {
    const BatchArgs &a = e.recs[g].ba;
    return a.spec ? a.D : 0;
  });
  if (total > 0)
    flat_groups(c, pref, ng, total, [&](int g, int item, bool valid, int gl, int) {
      const GV w = view(e, g);
      const DevState &s = w.s;
      int x = 0;
      bool was = false;
      if (valid) {
        x = w.a.del[item];
        was = s.del_pre[item] != kDeleted || w.inserted_now(x) || s.gt_stamp[x] == w.cur;
        if (was && s.batch_map) {
          const int m = s.batch_map[x];
          was = m >= 0 && m <= w.a.batch;
        }
      }
      const int rs = was ? s.full_row[x] : 0;
      const int len = was ? s.full_row[x + 1] - rs : 0;
      const int maxlen = __reduce_max_sync(0xffffffffu, len);
      for (int off = 0; off < maxlen; off += kRowGroup) {
        const int ee = off + gl;
        const int v = ee < len ? s.full_adj[rs + ee].x : -1;
        seed_mark(w, v >= 0 && w.live(v), v);
      }
    });

  // Tau filter over each batch's raw edges, four per lane (int4/float4 loads
  // when the arrays are 16-byte aligned): positions for the components step,
  // the kept new-new edges, and the endpoint marks.
  total = flat_build(pref, ng, [&](int g) {
    const GV w = view(e, g);
    return w.comp_path() ? (w.a.E + 3) >> 2 : 0;
  });
  flat_threads(c, pref, ng, total, [&](int g, int q, bool valid) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    const BatchArgs &a = w.a;
    int sv[4] = {0, 0, 0, 0}, dv[4] = {0, 0, 0, 0};
    float wv[4] = {0.f, 0.f, 0.f, 0.f};
    int nv = 0;
    if (valid) {
      const int base = q * 4;
      nv = min(4, a.E - base);
      const bool vec = nv == 4 && ((reinterpret_cast<uintptr_t>(a.es) | reinterpret_cast<uintptr_t>(a.ed) |
                                    reinterpret_cast<uintptr_t>(a.ew)) & 15u) == 0;
      if (vec) {
        const int4 s4 = reinterpret_cast<const int4 *>(a.es)[q];
        const int4 d4 = reinterpret_cast<const int4 *>(a.ed)[q];
        const float4 w4 = reinterpret_cast<const float4 *>(a.ew)[q];
        sv[0] = s4.x; sv[1] = s4.y; sv[2] = s4.z; sv[3] = s4.w;
        dv[0] = d4.x; dv[1] = d4.y; dv[2] = d4.z; dv[3] = d4.w;
        wv[0] = w4.x; wv[1] = w4.y; wv[2] = w4.z; wv[3] = w4.w;
      } else {
        for (int j = 0; j < nv; ++j) {
          sv[j] = a.es[base + j];
          dv[j] = a.ed[base + j];
          wv[j] = a.ew[base + j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = valid && j < nv;
      int ls = -1, ld = -1;
      bool kept = false;
      if (ok) {
        ls = w.inserted_now(sv[j]) ? s.local[sv[j]] : -1;
        ld = w.inserted_now(dv[j]) ? s.local[dv[j]] : -1;
        kept = wv[j] > a.tau && ls >= 0 && ld >= 0;
        s.lsrc[q * 4 + j] = ls;
        s.ldst[q * 4 + j] = ld;
      }
      // kept new-new edge (src/sparsifySubgraph.cu:133,165-174)
      const int k = reserve_keyed(kept, &s.bc->num_kept);
      if (k >= 0) {
        s.sub_pairs[2 * k] = sv[j];
        s.sub_pairs[2 * k + 1] = dv[j];
        s.sub_local[2 * k] = ls;
        s.sub_local[2 * k + 1] = ld;
      }
      if (!a.spec) {
        // ref: endpoints of edges with w > tau, clipped to ids below the
        // inserted count (src/sparsifySubgraph.cu:259-263 with :177-178)
        const bool heavy = ok && wv[j] > a.tau;
        seed_mark(w, heavy && sv[j] < a.I, sv[j]);
        seed_mark(w, heavy && dv[j] < a.I, dv[j]);
      } else {
        seed_mark(w, ok && w.live(sv[j]), sv[j]);
        seed_mark(w, ok && w.live(dv[j]), dv[j]);
      }
    }
  });

  // spec: every new non-ground-truth vertex is affected
  total = flat_build(pref, ng, [&](int g) {
    const BatchArgs &a = e.recs[g].ba;
    return a.spec ? a.I : 0;
  });
  if (total > 0)
    flat_threads(c, pref, ng, total, [&](int g, int i, bool valid) {
      const GV w = view(e, g);
      const int v = valid ? w.a.ins[i] : 0;
      seed_mark(w, valid && w.s.gt[v] < 0 && w.live(v), v);
    });
}

// ---------------------------------------------------------------- phase D ---
__device__ void phase_d_frontier(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  const int total = flat_build(pref, ng, [&](int g) { return e.recs[g].st.bc->num_seeds; });
  flat_threads(c, pref, ng, total, [&](int g, int i, bool valid) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    int v = 0;
    bool ok = false;
    if (valid) {
      v = s.seed_list[i];
      // collect filter (src/iterativePropagation.cu:73-75)
      ok = s.status[v] == kActive && !w.dev_deleted(v) && s.gt[v] < 0;
    }
    frontier_append(w, ok, ok, v, 0);
    const int slot = reserve_keyed(ok, &s.bc->seed_frontier);
    if (slot >= 0 && w.a.record) s.rec_front0[slot] = v;
  });
}

// Edges the components step hooks: ref, the first min(numSubEdges, E) raw
// edges (src/dynLP.cu:437-440); spec, the kept new-new edges.
__device__ __forceinline__ int hook_count(const GV &w) {
  if (!w.comp_path()) return 0;
  const int kept = w.s.bc->num_kept;
  if (w.a.spec) return kept;
  return kept > 0 ? min(2 * kept, w.a.E) : 0;
}

// Shiloach-Vishkin rounds for every graph with edges to hook: hook (larger
// root under the smaller with atomicMin, src/connectedComponents.cu:79-100),
// then pointer jumping to the root (:108-121), until a hook pass of that
// graph changes nothing. -1 stands for a vertex that is not new this batch.
__device__ bool phase_d_sv(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  for (int r = 0; r < kMaxHookRounds; ++r) {
    auto active = [&](int g) {
      const BatchCounters *bc = e.recs[g].st.bc;
      return r == 0 || ld_relaxed_i32(&bc->hook_flag[r - 1]) != 0;
    };
    int total = flat_build(pref, ng, [&](int g) { return active(g) ? hook_count(view(e, g)) : 0; });
    if (total == 0) break;
    flat_threads(c, pref, ng, total, [&](int g, int i, bool valid) {
      bool changed = false;
      int *flag = nullptr;
      if (valid) {
        const GV w = view(e, g);
        const DevState &s = w.s;
        const int *A = w.a.spec ? s.sub_local : s.lsrc;
        const int *B = w.a.spec ? s.sub_local + 1 : s.ldst;
        const size_t stride = w.a.spec ? 2 : 1;
        const int x = A[i * stride], y = B[i * stride];
        const int rx = x < 0 ? -1 : s.par[x];
        const int ry = y < 0 ? -1 : s.par[y];
        if (rx != ry) {
          const int hi = max(rx, ry), lo = min(rx, ry);
          if (atomicMin(&s.par[hi], lo) != lo) changed = true;
        }
        flag = &s.bc->hook_flag[r];
      }
      if (changed) *flag = 1;
    });
    if (!launch_sync(e)) return false;
    total = flat_build(pref, ng, [&](int g) { return active(g) && hook_count(view(e, g)) > 0 ? e.recs[g].ba.I : 0; });
    for (int item = c.gtid; item < total; item += c.nthreads) {
      const int g = locate(pref, ng, item);
      const DevState &s = e.recs[g].st;
      const int i = item - pref[g];
      int p = s.par[i];
      while (p >= 0) {
        const int q = s.par[p];
        if (q == p) break;
        p = q;
      }
      s.par[i] = p;
    }
    if (!launch_sync(e)) return false;
  }
  return true;
}

// ---------------------------------------------------------------- phase E ---
// Component count and fixed-point supernode weights per component root
// (src/labelInitialization.cu:59-88).
__device__ void phase_e(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  auto count = [&](int g) {
    const GV w = view(e, g);
    return w.comp_path() ? w.a.I : 0;
  };
  int total = flat_build(pref, ng, count);
  flat_threads(c, pref, ng, total, [&](int g, int i, bool valid) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    bool root = false;
    if (valid) {
      const int p = s.par[i];
      root = p == i;
      if (w.a.record && p >= 0) atomicMin(&s.rec_minid[p], w.a.ins[i]);
    }
    const int slot = reserve_keyed(root, &s.bc->num_comp);
    (void)slot;
  });
  flat_groups(c, pref, ng, total, [&](int g, int item, bool valid, int gl, int) {
    const GV w = view(e, g);
    const DevState &s = w.s;
    int rs = 0, len = 0, root = -1;
    if (valid) {
      root = s.par[item];
      const int u = w.a.ins[item];
      if (root >= 0) {
        rs = s.full_row[u];
        len = s.act_len[u];
      }
    }
    const int maxlen = __reduce_max_sync(0xffffffffu, len);
    long long q0 = 0, q1 = 0;
    for (int off = 0; off < maxlen; off += kRowGroup) {
      const int ee = off + gl;
      if (ee < len) {
        const int2 ent = s.act_adj[rs + ee];
        if (ent.x >= 0) {
          const int gc = s.gt[ent.x];
          const long long q = to_fixed(__int_as_float(ent.y));
          if (gc == 0) q0 += q;
          else if (gc == 1) q1 += q;
        }
      }
    }
#pragma unroll
    for (int o = kRowGroup / 2; o > 0; o >>= 1) {
      q0 += __shfl_down_sync(0xffffffffu, q0, o, kRowGroup);
      q1 += __shfl_down_sync(0xffffffffu, q1, o, kRowGroup);
    }
    if (valid && gl == 0 && root >= 0) {
      if (q0) atomicAdd(reinterpret_cast<unsigned long long *>(&s.acc[2 * root]), static_cast<unsigned long long>(q0));
      if (q1)
        atomicAdd(reinterpret_cast<unsigned long long *>(&s.acc[2 * root + 1]), static_cast<unsigned long long>(q1));
    }
  });
}

// ---------------------------------------------------------------- phase F ---
__device__ void phase_f(const EngineArgs &e, const Ctx &c, int *pref) {
  const int ng = e.ng_new;
  const int total = flat_build(pref, ng, [&](int g) { return e.recs[g].ba.I; });
  for (int item = c.gtid; item < total; item += c.nthreads) {
    const int g = locate(pref, ng, item);
    const int i = item - pref[g];
    const GV w = view(e, g);
    const DevState &s = w.s;
    const BatchArgs &a = w.a;
    const int u = a.ins[i];
    const bool comp = w.comp_path();
    float l;
    if (comp) {
      // src/labelInitialization.cu:99-142
      const int gc = s.gt[u];
      const int root = s.par[i];
      if (gc == 0) l = 0.0f;
      else if (gc == 1) l = 1.0f;
      else if (root < 0) l = 0.5f;
      else {
        const float w0 = from_fixed(s.acc[2 * root]);
        const float w1 = from_fixed(s.acc[2 * root + 1]);
        const float den = w0 + w1;
        l = den > 1e-10f ? quotient(w1, den, e.fast_div) : 0.5f;
      }
      s.lab0[u] = l;
      s.lab1[u] = l;
    } else if (s.gt_stamp[u] == w.cur && s.gt[u] >= 0) {
      // new vertices without new edges (src/dynLP.cu:482-504): this batch's
      // ground truth keeps the label set in phase B, everything else 0.5
      l = s.lab0[u];
    } else {
      l = 0.5f;
      s.lab0[u] = l;
      s.lab1[u] = l;
    }
    if (a.record) {
      s.rec_init[i] = l;
      const int root = comp ? s.par[i] : -1;
      s.rec_root[i] = root < 0 ? -1 : s.rec_minid[root];
    }
  }
}

// ---------------------------------------------------------------- phase G ---
// One row of at most 32 live entries by a group of G lanes; calls
// mark(cand, v) for each slot and for u itself, on every lane.
// cand[] receives what a changed row marks (src/iterativePropagation.cu:200-216):
// its non-deleted, non-ground-truth neighbours (cand[0..R)) and the vertex
// itself (cand[R]), -1 where nothing is marked; bit r of wide_bits is set when
// cand[r]'s live row is longer than 32 entries. Every load that depends only
// on the row (own label, neighbour labels, classes and row lengths) is issued
// before the row's sum is formed, so a row costs three dependent memory round
// trips (list entry, row, neighbours) before its marks.
template <int G>
__device__ __forceinline__ void narrow_row(const DevState &s, const float *src, float *dst, float delta, bool fast,
                                           int u, bool valid, int gl, int &len_out, int (&cand)[32 / G + 1],
                                           unsigned &wide_bits) {
  constexpr int R = 32 / G;
  int rs = 0, len = 0;
  float old = 0.0f;
  if (valid) {
    const int2 ri = s.rowinfo[u];
    rs = ri.x;
    len = ri.y;
    if (gl == 0) old = src[u];
  }
  float sw[R], sl[R];
  int vv[R];
  unsigned wb = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int ee = gl + G * r;
    sw[r] = 0.0f;
    sl[r] = 0.0f;
    vv[r] = -1;
    if (ee < len) {
      const int2 ent = s.act_adj[rs + ee];
      if (ent.x >= 0) {
        const float wt = __int_as_float(ent.y);
        sw[r] = wt;                               // 0 + w
        sl[r] = __fmaf_rn(wt, src[ent.x], 0.0f);  // fma(w, F_v, 0)
        const unsigned meta = s.nmeta[ent.x];
        if (meta & 1u) vv[r] = ent.x;
        if (meta & 2u) wb |= 1u << r;
      }
    }
  }
#pragma unroll
  for (int half = R / 2; half >= 1; half >>= 1)
#pragma unroll
    for (int r = 0; r < half; ++r) {
      sw[r] = sw[r] + sw[r + half];
      sl[r] = sl[r] + sl[r + half];
    }
  float tw = sw[0], tl = sl[0];
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) {
    tw = tw + __shfl_down_sync(0xffffffffu, tw, o, G);
    tl = tl + __shfl_down_sync(0xffffffffu, tl, o, G);
  }
  int changed = 0;
  if (valid && gl == 0) {
    const float nl = updated_label(tw, tl, old, fast);
    dst[u] = nl;
    changed = fabsf(nl - old) > delta;
  }
  changed = __shfl_sync(0xffffffffu, changed, 0, G);
  len_out = len;
#pragma unroll
  for (int r = 0; r < R; ++r) cand[r] = changed ? vv[r] : -1;
  cand[R] = (changed && gl == 0) ? u : -1;
  if (len > kNarrowMax) wb |= 1u << R;
  wide_bits = changed ? wb : 0u;
}

// Marks of one G-lane group (one row, one graph): every stamp atomic is
// issued before any result is used, then each of the three lists (narrow
// rows from the front of set `set`, wide rows from its back, the batch's
// touched list) gets one reservation for the whole group. The marked set is
// the same as marking one candidate at a time; only the order of the list
// entries differs, and nothing depends on that order.
template <int G>
__device__ __forceinline__ void group_mark(const GV &w, const int (&cand)[32 / G + 1], unsigned wide_bits,
                                           unsigned stamp, int set, int gl) {
  constexpr int C = 32 / G + 1;
  const DevState &s = w.s;
  unsigned old[C];
#pragma unroll
  for (int r = 0; r < C; ++r) old[r] = cand[r] >= 0 ? atomicMax(&s.front_stamp[cand[r]], stamp) : stamp;
  int nn = 0, nw = 0, nf = 0;
#pragma unroll
  for (int r = 0; r < C; ++r) {
    if (old[r] < stamp) {
      if ((wide_bits >> r) & 1u) ++nw;
      else ++nn;
    }
    if (old[r] < w.g0) ++nf;
  }
  // counts packed 10 bits each (a group marks at most 64 vertices)
  const int mine = nn | (nw << 10) | (nf << 20);
  int incl = mine;
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o, G);
    if (gl >= o) incl += t;
  }
  const int tot = __shfl_sync(0xffffffffu, incl, G - 1, G);
  int bn = 0, bw = 0, bf = 0;
  if (gl == G - 1 && tot != 0) {
    const int tn = tot & 1023, tw = (tot >> 10) & 1023, tf = tot >> 20;
    if (tn) bn = atomicAdd(&s.bc->front_count[set][0], tn);
    if (tw) bw = atomicAdd(&s.bc->front_count[set][1], tw);
    if (tf) bf = atomicAdd(&s.ctl->touched_count[w.a.seq & 1], tf);
  }
  bn = __shfl_sync(0xffffffffu, bn, G - 1, G);
  bw = __shfl_sync(0xffffffffu, bw, G - 1, G);
  bf = __shfl_sync(0xffffffffu, bf, G - 1, G);
  if (mine == 0) return;
  const int excl = incl - mine;
  int on = bn + (excl & 1023), ow = bw + ((excl >> 10) & 1023), of = bf + (excl >> 20);
  int *list = s.flist + static_cast<size_t>(set) * s.n;
  int *touched = s.touched + static_cast<size_t>(w.a.seq & 1) * s.n;
#pragma unroll
  for (int r = 0; r < C; ++r) {
    if (old[r] < stamp) {
      if ((wide_bits >> r) & 1u) list[s.n - 1 - ow++] = cand[r];
      else list[on++] = cand[r];
    }
    if (old[r] < w.g0) touched[of++] = cand[r];
  }
}

// One row of any length by a whole warp: 256 slots held as lane + 32*j.
template <class Mark>
__device__ __forceinline__ void wide_row(const DevState &s, const float *src, float *dst, float delta, bool fast,
                                         int u, int lane, Mark mark) {
  const int2 ri = s.rowinfo[u];
  const int rs = ri.x;
  const int len = ri.y;
  float sw[8], sl[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sw[j] = sl[j] = 0.0f;
  for (int p = 0; p < len; p += 256) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int ee = p + j * 32 + lane;
      if (ee < len) {
        const int2 ent = s.act_adj[rs + ee];
        if (ent.x >= 0) {
          const float wt = __int_as_float(ent.y);
          sw[j] = sw[j] + wt;
          sl[j] = __fmaf_rn(wt, src[ent.x], sl[j]);
        }
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
    tw = tw + __shfl_down_sync(0xffffffffu, tw, o);
    tl = tl + __shfl_down_sync(0xffffffffu, tl, o);
  }
  int changed = 0;
  if (lane == 0) {
    const float old = src[u];
    const float nl = updated_label(tw, tl, old, fast);
    dst[u] = nl;
    changed = fabsf(nl - old) > delta;
  }
  changed = __shfl_sync(0xffffffffu, changed, 0);
  if (changed) {
    for (int e0 = 0; e0 < len; e0 += 32) {
      const int ee = e0 + lane;
      const int v = ee < len ? s.act_adj[rs + ee].x : -1;
      mark(v >= 0 && s.gt[v] < 0, v);
    }
    mark(lane == 0, u);
  }
}

// A graph takes part in the launch's pass k (its own pass k + pass0) while its
// frontier is not empty and its pass is below max_iter; passes counts the
// passes it ran.
__device__ __forceinline__ bool graph_in_pass(const GraphRec &r, int k, int &nn, int &nw) {
  const BatchCounters *bc = r.st.bc;
  const int kg = k + r.ba.pass0;
  nn = ld_relaxed_i32(&bc->front_count[kg % 3][0]);
  nw = ld_relaxed_i32(&bc->front_count[kg % 3][1]);
  return nn + nw > 0 && kg < r.ba.max_iter;
}

// True once the launch's time slice has run out (checked by thread 0 of block
// 0 only, which recorded the launch's start).
__device__ __forceinline__ bool slice_over(const EngineArgs &e) {
  return e.slice_ns != 0 && global_timer_ns() - e.ectl->t_launch > e.slice_ns;
}

// A stop request for pass k of this launch (EngineCtl::slice_stop).
__device__ __forceinline__ unsigned long long stop_code(const EngineArgs &e, int k) {
  return (static_cast<unsigned long long>(static_cast<unsigned>(e.tag)) << 32) | static_cast<unsigned>(k);
}

// Solo mode: when all graphs' frontiers together are small, block 0 runs the
// passes alone, rows in registers and labels in shared memory
// (row_stint.cuh), while the other blocks wait at the next grid barrier. A row
// is loaded from HBM the first time its vertex is in the frontier; afterwards a
// pass touches only the block's own registers and shared memory. Labels of
// vertices outside the frontier cannot change during the stint, so loading
// them once is exact; every label written goes back to HBM when the stint
// ends. Passes and arithmetic are those of the grid path.
//
// Measured on the default workload (50,000 vertices, frontiers of 9 to 300
// rows): 0.22 to 0.27 us a pass, against 1.2 to 1.7 us for passes that walked a frontier
// list in shared memory with 8, 4 or 2 lanes per row and rebuilt the list with
// mark atomics and a reservation.
static_assert(kBlock == stint::kThreads, "block 0 runs a stint with all its threads");
static_assert(kSoloEntryMax <= stint::kSlotsUse, "a stint starts by putting the whole frontier into the vertex table");
static_assert(kOwnedTile == owner::kTile && kMaxGraphs <= 1024, "what owner_pass.cuh packs");
static_assert(kNarrowMax == stint::kMaxRow, "rows the frontier calls narrow are rows a stint can hold");
constexpr unsigned long long kSoloBudgetNs = 100000000ull;
constexpr int kTeamWarps = 16;  // a pass by at most this many warps counts as a team pass

struct SoloCache {
  stint::Cache c;
  int lastpass[kMaxGraphs];  // last launch pass each graph took part in during the stint
  int stop_slice;            // the request to stop was the launch's time slice
  int last;                  // the first pass a pass limit forbids
  int record;                // some graph records its frontier sizes
  int full;                  // the stint ended for lack of room
  unsigned long long start, launch;  // global timer at the start of the stint and of the launch
  unsigned long long team;   // passes of the stint by at most kTeamWarps warps
};

// The engine's graphs as a stint reads them: pass k0 + pass0 of each graph is
// stint pass 0.
struct SoloGraphs {
  const EngineArgs &e;
  int k0;
  __device__ void vertex(int g, int v, float &a, float &b, unsigned &meta) const {
    const GraphRec &r = e.recs[g];
    const DevState &s = r.st;
    const bool swapped = ((s.ctl->cur_buf ^ r.ba.pass0 ^ k0) & 1) != 0;
    const float l0 = s.lab0[v], l1 = s.lab1[v];
    a = swapped ? l1 : l0;
    b = swapped ? l0 : l1;
    // nmeta: bit 0 no ground truth, bit 1 row longer than 32 (kMarkable, kWide)
    meta = s.nmeta[v] | (swapped ? stint::kSwapped : 0u);
  }
  __device__ int2 row(int g, int v) const { return e.recs[g].st.rowinfo[v]; }
  __device__ void entry(int g, int at, int &v, float &w) const {
    const int2 ent = e.recs[g].st.act_adj[at];
    v = ent.x;
    w = __int_as_float(ent.y);
  }
};

// Not inlined: the row registers of a stint would otherwise be spilled around
// the other phases' code.
__device__ __noinline__ void solo_passes(const EngineArgs &e, int k0, int slot) {
  extern __shared__ __align__(16) unsigned char dsmem[];
  SoloCache &sc = *reinterpret_cast<SoloCache *>(dsmem);
  stint::Cache &c = sc.c;
  const int ng = e.ng;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SoloGraphs gr{e, k0};
  stint::clear(c);
  for (int g = tid; g < ng; g += kBlock) sc.lastpass[g] = -1;
  if (tid == 0) {
    sc.stop_slice = 0;
    sc.last = e.pass_budget > 0 ? e.pass_budget : 0x7fffffff;
    sc.record = 0;
    sc.full = 0;
    sc.team = 0;
    sc.start = global_timer_ns();
    sc.launch = e.slice_ns ? ld_relaxed_u64(&e.ectl->t_launch) : 0;
  }
  __syncthreads();
  // F_k0 of every graph into the table
  for (int g = warp; g < ng; g += stint::kWarps) {
    const GraphRec &r = e.recs[g];
    int nn, nw;
    if (!graph_in_pass(r, k0, nn, nw)) continue;
    if (lane == 0) {
      atomicMin(&sc.last, r.ba.max_iter - r.ba.pass0);
      if (r.ba.record) sc.record = 1;
    }
    const int *list = r.st.flist + static_cast<size_t>((k0 + r.ba.pass0) % 3) * r.st.n;
    for (int i = lane; i < nn + nw; i += 32) stint::seed(c, gr, g, i < nn ? list[i] : list[r.st.n - 1 - (i - nn)]);
  }
  // recorded sizes are counted up by the passes
  auto clear_record = [&](int k, int first, int step) {
    for (int g = first; g < ng; g += step) {
      const GraphRec &r = e.recs[g];
      const int kg = k + r.ba.pass0;
      if (r.ba.record && kg < kRecordIters) r.st.rec_fsizes[kg] = 0;
    }
  };
  __syncthreads();
  const int last = sc.last;
  const bool rec_any = sc.record != 0;
  if (rec_any) {
    clear_record(k0, tid, kBlock);
    __syncthreads();
  }
  stint::Row row;
  int j = 0;  // stint pass: launch pass k0 + j
  for (;;) {
    const int4 ctl = c.ctl;
    if (!stint::goes_on(ctl, j) || j >= last - k0) break;
    if (stint::needs_rows(ctl, j) && !stint::load_rows(c, gr, row, j, e.fast_div)) {
      if (tid == 0) sc.full = 1;
      break;
    }
    const int ns = stint::short_warps(c), nl = stint::long_warps(c);
    const bool is_long = warp >= stint::kWarps - nl;
    const int warps = (e.solo & 4) ? ns + nl : stint::kWarps;
    if (!(e.solo & 4) || warp < ns || is_long) {
      const bool leader = tid == (ns > 0 || !(e.solo & 4) ? 0 : kBlock - 32);
      auto tick = [&] {  // time budgets
        const uint64_t now = global_timer_ns();
        const bool slice = e.slice_ns != 0 && now - sc.launch > e.slice_ns;
        if (slice) sc.stop_slice = 1;
        return slice || now - sc.start > kSoloBudgetNs;
      };
      auto record = [&](int jj, const stint::Row &r) {
        const int4 now = c.ctl;
        if (!stint::goes_on(now, jj) || stint::needs_rows(now, jj) || jj >= last - k0) return;  // it will not run
        if (r.lead && stint::marked(c, r.slot, jj)) {
          const GraphRec &gr2 = e.recs[c.key[r.slot] >> 32];
          const int kg = k0 + jj + gr2.ba.pass0;
          if (gr2.ba.record && kg < kRecordIters) atomicAdd(&gr2.st.rec_fsizes[kg], 1);
        }
        if (leader) clear_record(k0 + jj + 1, 0, 1);
      };
      const int end =
          stint::run(c, row, j, last - k0, e.delta, e.fast_div, warps, is_long, leader, tick, rec_any, record);
      if (leader) c.end = end;
    }
    __syncthreads();  // the warps without rows wait here
    if (tid == 0 && warps <= kTeamWarps) sc.team += c.end - j;
    j = c.end;
  }
  const int k = k0 + j;
  __syncthreads();
  if (tid == 0 && sc.stop_slice) e.ectl->slice_stop = stop_code(e, k);  // the grid resumes at pass k and stops
  // rows that took part: their visit counts and the last pass of their graph
  {
    const bool own = row.visits != 0 && row.lead;
    const int g = own ? static_cast<int>(c.key[row.slot] >> 32) : 0;
    BatchCounters *bc = e.recs[g].st.bc;
    if (own) {
      c.meta[row.slot] |= stint::kVisited;
      atomicMax(&sc.lastpass[g], k0 + row.last);
    }
    add_keyed(own, row.visits * static_cast<unsigned>(row.len), &bc->aff_edges);
    add_keyed(own, row.visits, &bc->front_visits);
  }
  __syncthreads();
  // per-graph pass counts; the sets of the graph's pass k + pass0 and the next
  // one start empty
  for (int g = tid; g < ng; g += kBlock) {
    BatchCounters *bc = e.recs[g].st.bc;
    const int kg = k + e.recs[g].ba.pass0;
    if (sc.lastpass[g] >= 0) bc->passes = sc.lastpass[g] + e.recs[g].ba.pass0 + 1;
    bc->front_count[kg % 3][0] = bc->front_count[kg % 3][1] = 0;
    bc->front_count[(kg + 1) % 3][0] = bc->front_count[(kg + 1) % 3][1] = 0;
  }
  __syncthreads();
  // Labels written during the stint go back to HBM; the marks of pass k are
  // the frontier; vertices that were or are in a frontier join the touched
  // list the first time in this batch, with the batch's first stamp.
  for (int i = tid; i < stint::kSlots; i += kBlock) {
    const unsigned long long key = c.key[i];
    if (key == stint::kEmptyKey) continue;
    const unsigned meta = c.meta[i];
    const bool visited = (meta & stint::kVisited) != 0;
    const bool front = stint::marked(c, i, j) && (meta & stint::kMarkable) != 0;
    if (!visited && !front) continue;
    const GraphRec &r = e.recs[key >> 32];
    const DevState &s = r.st;
    const int v = static_cast<int>(key);
    if (visited) {
      const int first = (meta & stint::kSwapped) ? 1 : 0;
      s.lab0[v] = c.lab[first][i];
      s.lab1[v] = c.lab[first ^ 1][i];
    }
    if (front) {
      const int set = (k + r.ba.pass0) % 3;
      int *list = s.flist + static_cast<size_t>(set) * s.n;
      if (meta & stint::kWide) list[s.n - 1 - atomicAdd(&s.bc->front_count[set][1], 1)] = v;
      else list[atomicAdd(&s.bc->front_count[set][0], 1)] = v;
    }
    const unsigned g0 = s.ctl->stamp_base + 1u;
    if (atomicMax(&s.front_stamp[v], g0) < g0) {
      const int t = r.ba.seq & 1;
      s.touched[static_cast<size_t>(t) * s.n + atomicAdd(&s.ctl->touched_count[t], 1)] = v;
    }
  }
  if (tid == 0) {
    e.ectl->solo_k[slot] = k;
    e.ectl->solo_passes[slot] = k - k0;
    e.ectl->solo_full[slot] = sc.full;
    e.ectl->mode_passes[1] += sc.team;  // their time is part of the one-block stint's
  }
}

// One row of at most kLaneRow live entries by one lane, its 8-slot tree in
// registers (slot t = entry t). For such a row the reference's tree over 256
// slots adds only +0 at strides 128..8, so strides 4, 2, 1 give exactly its
// sum — the same as narrow_row<G>. cand[] and wide_bits as in narrow_row.
constexpr int kLaneRow = 8;

__device__ __forceinline__ void lane_row(const DevState &s, const float *src, float *dst, float delta, bool fast,
                                         int u, int rs, int len, bool valid, int (&cand)[kLaneRow + 1],
                                         unsigned &wide_bits) {
  float sw[kLaneRow], sl[kLaneRow];
  int vv[kLaneRow];
  unsigned wb = 0;
  const float old = valid ? src[u] : 0.0f;
#pragma unroll
  for (int t = 0; t < kLaneRow; ++t) {
    sw[t] = 0.0f;
    sl[t] = 0.0f;
    vv[t] = -1;
    if (valid && t < len) {
      const int2 ent = s.act_adj[rs + t];
      if (ent.x >= 0) {
        const float wt = __int_as_float(ent.y);
        sw[t] = wt;                               // 0 + w
        sl[t] = __fmaf_rn(wt, src[ent.x], 0.0f);  // fma(w, F_v, 0)
        const unsigned meta = s.nmeta[ent.x];
        if (meta & 1u) vv[t] = ent.x;
        if (meta & 2u) wb |= 1u << t;
      }
    }
  }
#pragma unroll
  for (int h = kLaneRow / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int t = 0; t < h; ++t) {
      sw[t] = sw[t] + sw[t + h];
      sl[t] = sl[t] + sl[t + h];
    }
  bool changed = false;
  if (valid) {
    const float nl = updated_label(sw[0], sl[0], old, fast);
    dst[u] = nl;
    changed = fabsf(nl - old) > delta;
  }
#pragma unroll
  for (int t = 0; t < kLaneRow; ++t) cand[t] = changed ? vv[t] : -1;
  cand[kLaneRow] = changed ? u : -1;
  wide_bits = changed ? wb : 0u;
}

// Marks of one-lane rows: every stamp atomic is issued before any result is
// used; then the lanes of one graph (a contiguous run: the work list is
// sorted by graph, invalid lanes last) reserve their next-frontier and
// touched-list entries with one atomic per list per run.
__device__ __forceinline__ void lane_mark(const GV &w, bool valid, int key, const int (&cand)[kLaneRow + 1],
                                          unsigned wide_bits, unsigned stamp, int set, int lane) {
  constexpr int C = kLaneRow + 1;
  const DevState &s = w.s;
  unsigned old[C];
#pragma unroll
  for (int r = 0; r < C; ++r) old[r] = cand[r] >= 0 ? atomicMax(&s.front_stamp[cand[r]], stamp) : stamp;
  int nn = 0, nw = 0, nf = 0;
#pragma unroll
  for (int r = 0; r < C; ++r) {
    if (old[r] < stamp) {
      if ((wide_bits >> r) & 1u) ++nw;
      else ++nn;
    }
    if (old[r] < w.g0) ++nf;
  }
  // counts packed 10 bits each (a run of 32 lanes marks at most 288)
  const int mine = nn | (nw << 10) | (nf << 20);
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    const int kp = __shfl_up_sync(0xffffffffu, key, o);
    if (lane >= o && kp == key) incl += t;
  }
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  const int tail = 31 - __clz(peers);
  const int tot = __shfl_sync(0xffffffffu, incl, tail);
  int bn = 0, bw = 0, bf = 0;
  // the run's last lane reserves for the whole run, whether or not it marked
  // anything itself (its own row may be one for the 4-lane groups)
  if (lane == tail && tot != 0) {
    const int tn = tot & 1023, tw = (tot >> 10) & 1023, tf = tot >> 20;
    if (tn) bn = atomicAdd(&s.bc->front_count[set][0], tn);
    if (tw) bw = atomicAdd(&s.bc->front_count[set][1], tw);
    if (tf) bf = atomicAdd(&s.ctl->touched_count[w.a.seq & 1], tf);
  }
  bn = __shfl_sync(0xffffffffu, bn, tail);
  bw = __shfl_sync(0xffffffffu, bw, tail);
  bf = __shfl_sync(0xffffffffu, bf, tail);
  if (!valid || mine == 0) return;
  const int excl = incl - mine;
  int on = bn + (excl & 1023), ow = bw + ((excl >> 10) & 1023), of = bf + (excl >> 20);
  int *list = s.flist + static_cast<size_t>(set) * s.n;
  int *touched = s.touched + static_cast<size_t>(w.a.seq & 1) * s.n;
#pragma unroll
  for (int r = 0; r < C; ++r) {
    if (old[r] < stamp) {
      if ((wide_bits >> r) & 1u) list[s.n - 1 - ow++] = cand[r];
      else list[on++] = cand[r];
    }
    if (old[r] < w.g0) touched[of++] = cand[r];
  }
}

// One propagation pass k over the flattened frontier, by the warps
// [warp0, warp0 + nwarps) and threads [t0, t0 + nthreads) of the launch.
template <int G>
__device__ void run_pass(const EngineArgs &e, int k, const int *pref, int tn, const int *pref2, int tw, int lane,
                         int warp0, int nwarps, int t0, int nthreads) {
  const int ng = e.ng;
  constexpr int GPW = 32 / G;
  const int grp = lane / G, gl = lane & (G - 1);
  // per graph: the set filled two passes from now was last read one pass ago
  for (int g = t0; g < ng; g += nthreads) {
    const GraphRec &r = e.recs[g];
    const int kg = k + r.ba.pass0;
    int nn, nw;
    const bool in = graph_in_pass(r, k, nn, nw);
    r.st.bc->front_count[(kg + 2) % 3][0] = 0;
    r.st.bc->front_count[(kg + 2) % 3][1] = 0;
    if (in) {
      r.st.bc->passes = kg + 1;
      if (r.ba.record && kg < kRecordIters) r.st.rec_fsizes[kg] = nn + nw;
    }
  }
  // A frontier large enough to give every warp two or more rounds of G-lane
  // groups runs with one lane per short row instead: 32 rows in flight per
  // warp rather than 32 / G, so a warp's dependent memory round trips overlap
  // across four to eight times more rows. Smaller frontiers keep the groups,
  // which spread one row's entries over G lanes. Same results either way.
  const bool lane_rows = G == 1 || tn >= 2 * nwarps * GPW;
  if (lane_rows) {
    // rows of at most 32 entries: one lane per row of at most 8 entries, 32
    // rows in flight per warp; rows of 9 to 32 entries of the same 32 go to
    // 4-lane groups afterwards
    // A lane's row of the next round is looked up while this round's rows
    // are in flight: its frontier entry is loaded at the top of the round,
    // its row start and length once this round's gathers are done. The
    // frontier list and the row table do not change during a pass.
    const int stride = nwarps * 32;
    auto entry_of = [&](int item, int &g, int &u) {
      g = 0;
      u = 0;
      if (item < tn) {
        g = locate(pref, ng, item);
        const GraphRec &r = e.recs[g];
        u = r.st.flist[static_cast<size_t>((k + r.ba.pass0) % 3) * r.st.n + (item - pref[g])];
      }
    };
    int g, u, rs = 0, len = 0;
    entry_of(warp0 * 32 + lane, g, u);
    if (warp0 * 32 + lane < tn) {
      const int2 ri = e.recs[g].st.rowinfo[u];
      rs = ri.x;
      len = ri.y;
    }
    for (int base = warp0 * 32; base < tn; base += stride) {
      const int item = base + lane;
      const bool valid = item < tn;
      int g1, u1, rs1 = 0, len1 = 0;
      entry_of(item + stride, g1, u1);
      {
        const GV w = view(e, g);
        const DevState &s = w.s;
        const int kg = k + w.a.pass0;
        const int cb = s.ctl->cur_buf;
        const float *src = ((cb ^ kg) & 1) ? s.lab1 : s.lab0;
        float *dst = ((cb ^ kg) & 1) ? s.lab0 : s.lab1;
        const bool mine = valid && len <= kLaneRow;
        int cand[kLaneRow + 1];
        unsigned wide_bits = 0;
        lane_row(s, src, dst, w.a.delta, e.fast_div, u, rs, len, mine, cand, wide_bits);
        if (item + stride < tn) {
          const int2 ri = e.recs[g1].st.rowinfo[u1];
          rs1 = ri.x;
          len1 = ri.y;
        }
        lane_mark(w, mine, valid ? g : -1, cand, wide_bits, w.g0 + static_cast<unsigned>(kg) + 1u, (kg + 1) % 3,
                  lane);
        add_keyed(mine, static_cast<unsigned>(len), &s.bc->aff_edges);
        add_keyed(mine, 1u, &s.bc->front_visits);
        // the 4-lane groups below take this round's long rows
        const int gc = g, uc = u, lc = len;
        g = g1;
        u = u1;
        rs = rs1;
        len = len1;
        g1 = gc;
        u1 = uc;
        len1 = lc;
      }
      unsigned longm = __ballot_sync(0xffffffffu, valid && len1 > kLaneRow);
      const int q = lane >> 2, ql = lane & 3;
      while (longm) {  // up to 8 rows a round, the q-th remaining one to 4-lane group q
        unsigned m = longm;
        for (int i = 0; i < q && m; ++i) m &= m - 1;
        const bool have = m != 0;
        const int from = have ? __ffs(m) - 1 : 0;
        const int gq = __shfl_sync(0xffffffffu, g1, from);
        const int uq = __shfl_sync(0xffffffffu, u1, from);
        for (int i = 0; i < 8 && longm; ++i) longm &= longm - 1;
        const GV w = view(e, gq);
        const DevState &s = w.s;
        const int kg = k + w.a.pass0;
        const int cb = s.ctl->cur_buf;
        const float *src = ((cb ^ kg) & 1) ? s.lab1 : s.lab0;
        float *dst = ((cb ^ kg) & 1) ? s.lab0 : s.lab1;
        int lq = 0;
        int cand[32 / 4 + 1];
        unsigned wide_bits = 0;
        narrow_row<4>(s, src, dst, w.a.delta, e.fast_div, uq, have, ql, lq, cand, wide_bits);
        group_mark<4>(w, cand, wide_bits, w.g0 + static_cast<unsigned>(kg) + 1u, (kg + 1) % 3, ql);
        add_keyed(have && ql == 0, static_cast<unsigned>(lq), &s.bc->aff_edges);
        add_keyed(have && ql == 0, 1u, &s.bc->front_visits);
      }
    }
  } else
  // rows of at most 32 entries: groups of G lanes
  for (int base = warp0 * GPW; base < tn; base += nwarps * GPW) {
    const int item = base + grp;
    const bool valid = item < tn;
    const int g = valid ? locate(pref, ng, item) : 0;
    const GV w = view(e, g);
    const DevState &s = w.s;
    const int kg = k + w.a.pass0;
    const int nset = (kg + 1) % 3;
    const int cb = s.ctl->cur_buf;
    const float *src = ((cb ^ kg) & 1) ? s.lab1 : s.lab0;
    float *dst = ((cb ^ kg) & 1) ? s.lab0 : s.lab1;
    const unsigned stamp = w.g0 + static_cast<unsigned>(kg) + 1u;
    const int u = valid ? s.flist[static_cast<size_t>(kg % 3) * s.n + (item - pref[g])] : 0;
    int len = 0;
    int cand[32 / G + 1];
    unsigned wide_bits = 0;
    narrow_row<G>(s, src, dst, w.a.delta, e.fast_div, u, valid, gl, len, cand, wide_bits);
    group_mark<G>(w, cand, wide_bits, stamp, nset, gl);
    add_keyed(valid && gl == 0, static_cast<unsigned>(len), &s.bc->aff_edges);
    add_keyed(valid && gl == 0, 1u, &s.bc->front_visits);
  }
  // longer rows: one warp each
  for (int wi = warp0; wi < tw; wi += nwarps) {
    const int g = locate(pref2, ng, wi);
    const GV w = view(e, g);
    const DevState &s = w.s;
    const int kg = k + w.a.pass0;
    const int nset = (kg + 1) % 3;
    const int cb = s.ctl->cur_buf;
    const float *src = ((cb ^ kg) & 1) ? s.lab1 : s.lab0;
    float *dst = ((cb ^ kg) & 1) ? s.lab0 : s.lab1;
    const unsigned stamp = w.g0 + static_cast<unsigned>(kg) + 1u;
    const int u = s.flist[static_cast<size_t>(kg % 3) * s.n + (s.n - 1 - (wi - pref2[g]))];
    auto mark = [&](bool cand, int v) {
      bool fresh = false, first = false;
      if (cand) {
        const unsigned old = atomicMax(&s.front_stamp[v], stamp);
        fresh = old < stamp;
        first = old < w.g0;
      }
      frontier_append(w, fresh, first, v, nset);
    };
    wide_row(s, src, dst, w.a.delta, e.fast_div, u, lane, mark);
    if (lane == 0) {
      atomicAdd(&s.bc->aff_edges, static_cast<unsigned long long>(s.act_len[u]));
      atomicAdd(&s.bc->front_visits, 1ull);
    }
  }
}

// Frontier sizes of pass k: narrow rows into pref, wide rows into pref2. Both
// prefixes come from one scan: a graph's two counts are read once and summed
// as the halves of one 64-bit value (a frontier never reaches 2^32 rows).
__device__ __forceinline__ void pass_sizes(const EngineArgs &e, int k, int *pref, int *pref2, int &tn, int &tw) {
  __shared__ unsigned long long s_warp2[kBlock / 32];
  const int ng = e.ng;
  __syncthreads();
  constexpr int kPer = (kMaxGraphs + kBlock - 1) / kBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long vals[kPer];
  unsigned long long local = 0;
  const int start = threadIdx.x * kPer;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int g = start + j;
    int nn = 0, nw = 0;
    if (g < ng && !graph_in_pass(e.recs[g], k, nn, nw)) nn = nw = 0;
    vals[j] = (static_cast<unsigned long long>(nw) << 32) | static_cast<unsigned>(nn);
    local += vals[j];
  }
  unsigned long long incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp2[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    unsigned long long x = lane < kBlock / 32 ? s_warp2[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < kBlock / 32) s_warp2[lane] = x;
  }
  __syncthreads();
  unsigned long long run = incl - local + (warp > 0 ? s_warp2[warp - 1] : 0);
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int g = start + j;
    if (g < ng) {
      pref[g] = static_cast<int>(run & 0xffffffffu);
      pref2[g] = static_cast<int>(run >> 32);
    }
    run += vals[j];
  }
  if (threadIdx.x == kBlock - 1) {
    pref[ng] = static_cast<int>(run & 0xffffffffu);
    pref2[ng] = static_cast<int>(run >> 32);
  }
  __syncthreads();
  tn = pref[ng];
  tw = pref2[ng];
}

// The engine's graphs as owned passes read them.
struct OwnedGraphs {
  static constexpr bool kCounts = true;
  const EngineArgs &e;
  __device__ int graphs() const { return e.ng; }
  __device__ int nodes(int g) const { return e.recs[g].st.n; }
  __device__ int2 row(int g, int v) const { return e.recs[g].st.rowinfo[v]; }
  __device__ bool active(int g, int v) const { return markable(g, v); }
  __device__ bool markable(int g, int v) const { return (e.recs[g].st.nmeta[v] & 1u) != 0; }
  __device__ void entry(int g, int at, int &v, float &w) const {
    const int2 ent = e.recs[g].st.act_adj[at];
    v = ent.x;
    w = __int_as_float(ent.y);
  }
  template <int N>
  __device__ void entries(int g, int start, int first, int step, int len, int (&v)[N], float (&w)[N]) const {
    const int2 *adj = e.recs[g].st.act_adj + start;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int2 ent = load_if(first + j * step < len, adj + first + j * step, -1);
      v[j] = ent.x;
      w[j] = __int_as_float(ent.y);
    }
  }
  template <int N>
  __device__ unsigned markables(int g, const int (&v)[N]) const {
    const uint8_t *meta = e.recs[g].st.nmeta;
    unsigned can = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) can |= (load_if(v[j] >= 0, meta + v[j], 0) & 1u) << j;
    return can;
  }
};

// Recorded frontier sizes of pass k back to zero, by one block.
__device__ __forceinline__ void clear_record(const EngineArgs &e, int k) {
  for (int g = threadIdx.x; g < e.ng; g += kBlock) {
    const GraphRec &r = e.recs[g];
    const int kg = k + r.ba.pass0;
    if (r.ba.record && kg < kRecordIters && kg < r.ba.max_iter) r.st.rec_fsizes[kg] = 0;
  }
}

// The passes of a stint on owned rows, from k on; returns the first pass not
// run, or -1 when the launch has to end. TILES: the block's passes are tile_pass (up to
// 1,024 owned vertices, 151 x 1,024 in the launch, in tiles of few steps).
template <bool TILES>
__device__ __forceinline__ int owned_loop_as(const EngineArgs &e, int k, owner::Store s, bool rec_any) {
  const OwnedGraphs gr{e};
  owner::Head &h = s.head();
  unsigned before = 0xffffffffu;  // rows of the pass before the last
  for (;;) {
    if (s.tiles > 0) {
      unsigned *own = h.marks + (k & 1 ? h.plane : 0u);
      unsigned *next = h.marks + (k & 1 ? 0u : h.plane);
      auto each = [&](int i) {
        if (!rec_any) return;
        const GraphRec &r = e.recs[owner::graph_of(s.meta(i))];
        const int kg = k + r.ba.pass0;
        if (r.ba.record && kg < kRecordIters) atomicAdd(&r.st.rec_fsizes[kg], 1);
      };
      if (TILES) owner::tile_pass(s, gr, own, next, k, h.delta, h.fast != 0, each);
      else owner::pass(s, gr, own, next, k, h.delta, h.fast != 0, each);
    } else if (rec_any && blockIdx.x == 0) {
      clear_record(e, k + 1);
    }
    unsigned long long sum;
    const bool ok = sum_sync(&e.ectl->bar, s_bar, &e.ectl->err, e.timeout_ns, [&]() -> unsigned long long {
      if (s.tiles == 0) {
        if (blockIdx.x != 0 || !slice_over(e)) return 0ull;
        e.ectl->slice_stop = stop_code(e, k + 1);
        return kSumStop;
      }
      const unsigned long long mine =
          static_cast<unsigned>((h.count & 0xffff) + (h.count >> 16) + h.wide) | (h.moved ? kSumMoved : 0ull);
      h.count = h.wide = h.wide_at = 0;
      h.moved = 0;
      return mine;
    }, sum);
    if (!ok) return -1;
    ++k;
    const unsigned rows = static_cast<unsigned>(sum);
    const bool moved = (sum & (0xffull * kSumMoved)) != 0, stop = (sum & (0xffull * kSumStop)) != 0;
    if (!moved || stop || k >= h.budget || k >= h.stint_end) return k;
    // small in two passes running: the next one is small too, as a rule
    if (max(rows, before) <= h.solo_entry && k >= h.solo_from) return k;
    before = rows;
  }
}

// Not inlined, so that its registers are its own; one function for both loops: as two,
// or as one loop, the kernel's other functions get other registers (one-block passes of
// 5,000 vertices 227 instead of 217 ns, full-grid ones 3.24 instead of 3.15 us).
__device__ __noinline__ int owned_loop(const EngineArgs &e, int k, owner::Store s, bool rec_any, bool tiles) {
  return tiles ? owned_loop_as<true>(e, k, s, rec_any) : owned_loop_as<false>(e, k, s, rec_any);
}

// Passes from k0 on by the blocks that own the rows (owner_pass.cuh). The
// frontier of pass k0 is in the lists (pref, pref2: its sizes), that of the
// pass returned in k_out is in them again. Ends when the frontier empties,
// fits the one-block mode, at a pass or time limit. `loaded`: this block holds
// its rows already.
__device__ __noinline__ bool owned_passes(const EngineArgs &e, int k0, int solo_from, const int *pref,
                                          const int *pref2, int tn, int tw, bool loaded, int *k_out) {
  const int ng = e.ng, tid = threadIdx.x;
  const OwnedGraphs gr{e};
  auto marks = [&](int k) { return e.marks + (k & 1 ? e.mark_plane : 0u); };
  // frontier lists -> marks
  for (int item = blockIdx.x * kBlock + tid; item < tn + tw; item += gridDim.x * kBlock) {
    const bool wide = item >= tn;
    const int at = wide ? item - tn : item;
    const int g = locate(wide ? pref2 : pref, ng, at);
    const GraphRec &r = e.recs[g];
    const int i = at - (wide ? pref2 : pref)[g];
    const int v = r.st.flist[static_cast<size_t>((k0 + r.ba.pass0) % 3) * r.st.n + (wide ? r.st.n - 1 - i : i)];
    marks(k0)[r.ba.flat + v] = 1;
  }
  const owner::Store s = owner::store(e.smem_bytes, ng, owner::owned_tiles(e.tiles));
  owner::Head &h = s.head();
  const bool owns = s.tiles > 0;
  if (owns && !loaded) {
    if (tid == 0) {
      h.pool_used = 0;
      h.first_limit = 0x7fffffff;
      h.count = h.wide = h.wide_at = 0;
      h.moved = h.steps = 0;
    }
    __syncthreads();
    for (int g = tid; g < ng; g += kBlock) {
      const GraphRec &r = e.recs[g];
      const bool swapped = ((r.st.ctl->cur_buf ^ r.ba.pass0) & 1) != 0;
      owner::Local &l = s.graph(g);
      l.lab[0] = swapped ? r.st.lab1 : r.st.lab0;
      l.lab[1] = swapped ? r.st.lab0 : r.st.lab1;
      l.flat = r.ba.flat;
      l.limit = r.ba.max_iter - r.ba.pass0;
      atomicMin(&h.first_limit, l.limit);
    }
    __syncthreads();
    owner::load(s, gr);
  }
  if (tid == 0) {
    h.marks = e.marks;
    h.plane = e.mark_plane;
    h.delta = e.delta;
    h.fast = e.fast_div;
    h.budget = e.pass_budget > 0 ? e.pass_budget : 0x7fffffff;
    h.solo_entry = (e.solo & 1) ? static_cast<unsigned>(e.solo_entry) : 0u;
    h.solo_from = solo_from;
    h.stint_end = k0 + owner::kMaxStint;
  }
  if (owns)
    for (int g = tid; g < ng; g += kBlock) {
      s.graph(g).last = -1;
      s.graph(g).edges = s.graph(g).visits = 0;
    }
  bool rec_any = false;
  for (int g = tid; g < ng; g += kBlock) rec_any |= e.recs[g].ba.record != 0;
  rec_any = __syncthreads_or(rec_any) != 0;
  if (rec_any && blockIdx.x == 0) clear_record(e, k0);
  if (!launch_sync(e)) return false;
  if (blockIdx.x == 0)  // the lists are filled again at the end
    for (int i = tid; i < 6 * ng; i += kBlock) (&e.recs[i / 6].st.bc->front_count[0][0])[i % 6] = 0;
  const bool tiles = !owns || (s.n() <= kBlock && h.steps <= owner::kTileSteps);
  const int k = owned_loop(e, k0, s, rec_any, tiles);
  if (k < 0) return false;
  // marks -> frontier lists; visits -> counters; vertices that were or are in a
  // frontier join the touched list the first time in this batch
  if (owns) {
    for (int i = tid; i < s.n(); i += kBlock) {
      const unsigned vis = s.visits(i);
      const int lg = owner::graph_of(s.meta(i));
      const GraphRec &r = e.recs[lg];
      const DevState &d = r.st;
      const int v = static_cast<int>(owner::flat_of(i) - s.graph(lg).flat);
      unsigned *mark = marks(k) + owner::flat_of(i);
      const bool marked = __ldcg(mark) != 0;
      if (marked) *mark = 0;
      s.visits(i) = 0;
      const bool front = marked && k < s.graph(lg).limit;
      const int len = vis || front ? d.act_len[v] : 0;
      const int set = (k + r.ba.pass0) % 3;
      int *list = d.flist + static_cast<size_t>(set) * d.n;
      append_keyed(front && len <= kNarrowMax, v, list, &d.bc->front_count[set][0]);
      append_back_keyed(front && len > kNarrowMax, v, list, d.n, &d.bc->front_count[set][1]);
      if (vis) {
        atomicAdd(&s.graph(lg).edges, static_cast<unsigned long long>(vis) * len);
        atomicAdd(&s.graph(lg).visits, static_cast<unsigned long long>(vis));
      }
      const unsigned g0 = d.ctl->stamp_base + 1u;
      const bool fresh = (vis || front) && atomicMax(&d.front_stamp[v], g0) < g0;
      append_keyed(fresh, v, d.touched + static_cast<size_t>(r.ba.seq & 1) * d.n,
                   &d.ctl->touched_count[r.ba.seq & 1]);
    }
    __syncthreads();
    for (int g = tid; g < ng; g += kBlock) {
      const owner::Local &l = s.graph(g);
      if (l.last < 0) continue;
      const GraphRec &r = e.recs[g];
      atomicAdd(&r.st.bc->aff_edges, l.edges);
      atomicAdd(&r.st.bc->front_visits, l.visits);
      atomicMax(&r.st.bc->passes, l.last + r.ba.pass0 + 1);
    }
  }
  *k_out = k;
  return launch_sync(e);
}

// The propagation passes of the launch; k_end is the first pass not run (the
// graphs whose frontier is live at k_end continue in a later launch). OWNED:
// passes run on owned rows after the first e.list_passes, otherwise over lists, in a
// kernel of its own.
template <int G, bool OWNED>
__device__ bool phase_g(const EngineArgs &e, int *pref, int *pref2, int &k_end) {
  auto place = [] {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
  };
  auto lead = [&] { return blockIdx.x == 0 && place() == 0; };
  int solo_from = 0;     // the one-block mode declined: not tried again before this pass
  bool owned = false;    // the block holds its rows (owned_passes)
  int stint_no = 0;
  int listed = 0;        // full-grid passes run over lists
  int k = 0;
  // passes and device time per mode in this launch (one block, full grid), by
  // thread 0 of block 0; in shared memory, because in registers they cost the
  // list passes (launches beyond owned rows) 104 bytes of spills and 3%: 62.8
  // against 60.7 ms for 14 batches of 4.2 million vertices
  __shared__ unsigned long long mp[2], mns[2], t_mode;
  if (lead()) mp[0] = mp[1] = mns[0] = mns[1] = 0;
  for (;; ++k) {
    int tn, tw;
    pass_sizes(e, k, pref, pref2, tn, tw);
    if (tn + tw == 0) break;
    if (e.pass_budget > 0 && k >= e.pass_budget) break;
    if (ld_relaxed_u64(&e.ectl->slice_stop) == stop_code(e, k)) break;
    if (lead()) e.ectl->where_pass = k;
    const bool solo_ok = (e.solo & 1) && tn + tw <= e.solo_entry && k >= solo_from;
    if (solo_ok) {
      if (lead()) t_mode = global_timer_ns();
      if (blockIdx.x == 0) solo_passes(e, k, stint_no & 1);
      if (!launch_sync(e)) return false;
      const int done = ld_relaxed_i32(&e.ectl->solo_passes[stint_no & 1]);
      const int kk = ld_relaxed_i32(&e.ectl->solo_k[stint_no & 1]);
      ++stint_no;
      if (lead()) {
        mp[0] += done;
        mns[0] += global_timer_ns() - t_mode;
      }
      if (done == 0) solo_from = k + 1;  // declined: the full grid's
      // A stint that ran out of room soon would run out again: a load costs
      // several passes, so the frontier stays with the grid for a while.
      if (done < 256 && ld_relaxed_i32(&e.ectl->solo_full[(stint_no - 1) & 1])) solo_from = kk + 256;
      k = kk - 1;  // the loop increment resumes at pass kk
      continue;
    }
    if (lead()) t_mode = global_timer_ns();
    if (OWNED && listed >= e.list_passes) {
      int kk = k;
      if (!owned_passes(e, k, solo_from, pref, pref2, tn, tw, owned, &kk)) return false;
      owned = true;
      if (lead()) {
        mp[1] += kk - k;
        mns[1] += global_timer_ns() - t_mode;
      }
      k = kk - 1;  // the loop increment resumes at pass kk
      continue;
    }
    ++listed;
    // Nothing of the thread's place is kept over the loop: the call of the one-block
    // mode leaves few registers for it (4 and 16 bytes of spill stores and loads
    // instead of 40 and 88, with the owned passes in the same kernel). 4.2 million
    // vertices, frontiers of 210,000 and 340,000 rows: 46 -> 44 and 67 -> 64 us.
    const int tid = place();
    const int gtid = blockIdx.x * kBlock + tid, nthreads = gridDim.x * kBlock;
    run_pass<G>(e, k, pref, tn, pref2, tw, tid & 31, gtid >> 5, nthreads >> 5, gtid, nthreads);
    if (lead() && slice_over(e)) e.ectl->slice_stop = stop_code(e, k + 1);
    if (!launch_sync(e)) return false;
    if (lead()) {
      ++mp[1];
      mns[1] += global_timer_ns() - t_mode;
    }
  }
  k_end = k;
  if (lead()) {
    e.ectl->mode_passes[0] += mp[0];
    e.ectl->mode_ns[0] += mns[0];
    e.ectl->mode_passes[3] += mp[1];
    e.ectl->mode_ns[3] += mns[1];
  }
  return true;
}

// A graph's batch ends in this launch when it takes no part in pass k_end.
__device__ __forceinline__ bool batch_done(const GraphRec &r, int k_end) {
  int nn, nw;
  return !graph_in_pass(r, k_end, nn, nw);
}

// ---------------------------------------------------------------- phase H ---
// Ground truth of this batch back to exactly 0/1 in both buffers
// (src/iterativePropagation.cu:224-235; earlier ground truth already is), and
// the accuracy counters (src/dynLP.cu:65-85) updated at every vertex whose
// status or label may have changed.
__device__ void phase_h(const EngineArgs &e, const Ctx &c, int *pref, int k_end) {
  const int ng = e.ng;
  const int total = flat_build(pref, ng, [&](int g) {
    const GraphRec &r = e.recs[g];
    if (!batch_done(r, k_end)) return 0;
    return r.ba.G + r.ba.D + r.st.ctl->touched_count[r.ba.seq & 1] + r.ba.I + r.ba.D + r.ba.G;
  });
  flat_threads(c, pref, ng, total, [&](int g, int i, bool valid) {
    const GraphRec &r = e.recs[g];
    const DevState &s = r.st;
    const BatchArgs &a = r.ba;
    int dc = 0, dt = 0;
    if (valid) {
      if (i < a.G) {
        const int v = a.gt_ids[i];
        const float l = s.gt[v] == 0 ? 0.0f : 1.0f;
        s.lab0[v] = l;
        s.lab1[v] = l;
      } else if ((i -= a.G) < a.D) {
        s.del_keep[i] = a.del[i];  // the next batch restores these rows (ref)
      } else {
        i -= a.D;
        const int tc = s.ctl->touched_count[a.seq & 1];
        int v;
        if (i < tc) v = s.touched[static_cast<size_t>(a.seq & 1) * s.n + i];
        else if ((i -= tc) < a.I) v = a.ins[i];
        else if ((i -= a.I) < a.D) v = a.del[i];
        else v = a.gt_ids[i - a.D];
        const int st = s.status[v];
        int now = -1;
        if (st != kDeleted && st != kGroundTruth) {
          const int passes = s.bc->passes;
          const float *lab = ((s.ctl->cur_buf ^ passes) & 1) ? s.lab1 : s.lab0;
          const int pred = lab[v] >= 0.5f ? 1 : 0;
          const int truth = s.truth ? s.truth[v] : 0;
          now = pred == truth ? 1 : 0;
        }
        const int before = atomicExch(&s.contrib[v], now);
        dc = (now == 1) - (before == 1);
        dt = (now >= 0) - (before >= 0);
      }
    }
    const unsigned act = __ballot_sync(0xffffffffu, valid && (dc != 0 || dt != 0));
    if (valid && (dc != 0 || dt != 0)) {
      const unsigned peers = __match_any_sync(act, reinterpret_cast<unsigned long long>(s.ctl));
      const int sc = __reduce_add_sync(peers, dc);
      const int st2 = __reduce_add_sync(peers, dt);
      if ((threadIdx.x & 31) == __ffs(peers) - 1) {
        if (sc) atomicAdd(reinterpret_cast<unsigned long long *>(&s.ctl->correct), static_cast<unsigned long long>(static_cast<long long>(sc)));
        if (st2) atomicAdd(reinterpret_cast<unsigned long long *>(&s.ctl->total), static_cast<unsigned long long>(static_cast<long long>(st2)));
      }
    }
  });
}

}  // namespace

template <int G, bool OWNED>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) engine_kernel(const __grid_constant__ EngineArgs e) {
  const Ctx c = make_ctx();
  __shared__ int pref[kMaxGraphs + 1];
  __shared__ int pref2[kMaxGraphs + 1];
  if (ld_relaxed_i32(&e.ectl->err) != 0) return;
  if (threadIdx.x == 0) {
    s_bar.gen = 0;
    s_bad = 0;
  }
  __syncthreads();

  // block 0 records the last phase it reached (read back after a timeout)
  auto at = [&](int phase) {
    if (blockIdx.x == 0 && threadIdx.x == 0) e.ectl->where = phase;
  };
  if (c.gtid == 0) e.ectl->t_launch = global_timer_ns();
  if (e.ng_new > 0) {  // a launch that only continues batches starts at phase G
    at(1);
    phase_a(e, c, pref);
    if (!launch_sync(e)) return;
    at(2);
    phase_b(e, c, pref);
    if (!launch_sync(e)) return;
    at(3);
    phase_c(e, c, pref);
    if (!launch_sync(e)) return;
    at(4);
    phase_d_frontier(e, c, pref);
    if (!phase_d_sv(e, c, pref)) return;
    at(5);
    if (!launch_sync(e)) return;
    at(6);
    phase_e(e, c, pref);
    if (!launch_sync(e)) return;
    at(7);
    phase_f(e, c, pref);
    if (!launch_sync(e)) return;
  }
  at(8);
  int k_end = 0;
  if (!phase_g<G, OWNED>(e, pref, pref2, k_end)) return;
  at(9);
  phase_h(e, c, pref, k_end);
  if (!launch_sync(e)) return;
  at(10);

  // per-graph statistics and the state the next batch starts from
  for (int g = c.gtid; g < e.ng; g += c.nthreads) {
    const GraphRec &r = e.recs[g];
    const DevState &s = r.st;
    const BatchArgs &a = r.ba;
    const BatchCounters *bc = s.bc;
    if (!batch_done(r, k_end)) {  // continues in a later launch
      if (e.progress) e.progress[g] = make_int2(0, k_end + a.pass0);
      continue;
    }
    if (e.progress) e.progress[g] = make_int2(1, bc->passes);
    const GV w = view(e, g);
    const bool comp = w.comp_path();
    const int passes = bc->passes;
    const int hc = hook_count(w);
    int rounds = 0;
    if (hc > 0) {
      rounds = kMaxHookRounds;
      for (int q = 0; q < kMaxHookRounds; ++q)
        if (bc->hook_flag[q] == 0) {
          rounds = q + 1;
          break;
        }
    }
    dlp_batch_stats st;
    memset(&st, 0, sizeof(st));
    st.batch = a.batch;
    st.iterations = passes;
    st.num_components = comp ? bc->num_comp : 0;
    st.num_sub_edges = comp ? 2 * bc->num_kept : 0;
    st.hook_edges = a.spec ? 2 * hc : hc;
    st.hook_rounds = rounds;
    st.seed_frontier = bc->seed_frontier;
    st.seed_marks = bc->num_seeds;
    st.affected_edges = static_cast<int64_t>(bc->aff_edges);
    st.frontier_visits = static_cast<int64_t>(bc->front_visits);
    st.correct = s.ctl->correct;
    st.total = s.ctl->total;
    st.accuracy = st.total > 0 ? static_cast<float>(st.correct) / static_cast<float>(st.total) : 1.0f;
    st.status = DLP_OK;
    st.init_branch = comp ? 1 : (a.I > 0 ? 2 : 0);
    st.hook_truncated = (!a.spec && comp && 2 * bc->num_kept > a.E) ? 1 : 0;
    st.dirty_rows = bc->num_dirty;
    st.dirty_entries = static_cast<int64_t>(bc->dirty_entries);
    *s.stats_slot = st;
    s.ctl->cur_buf ^= (passes & 1);
    s.ctl->stamp_base = w.g0 + static_cast<unsigned>(passes) + 1u;
  }
}

template __global__ void engine_kernel<1, false>(const __grid_constant__ EngineArgs);
template __global__ void engine_kernel<4, false>(const __grid_constant__ EngineArgs);
template __global__ void engine_kernel<8, false>(const __grid_constant__ EngineArgs);
template __global__ void engine_kernel<16, false>(const __grid_constant__ EngineArgs);
template __global__ void engine_kernel<32, false>(const __grid_constant__ EngineArgs);
template __global__ void engine_kernel<8, true>(const __grid_constant__ EngineArgs);

// One block per graph that starts a batch: its counters back to zero; block 0
// also clears the launch's barrier.
__global__ void zero_counters_kernel(const GraphRec *recs, int ng_new, EngineCtl *ectl) {
  if (blockIdx.x == 0) {
    if (threadIdx.x < 4) ectl->bar.word[threadIdx.x].v = 0;
  }
  if (blockIdx.x >= ng_new) return;
  int *p = reinterpret_cast<int *>(recs[blockIdx.x].st.bc);
  constexpr int kWords = static_cast<int>(sizeof(BatchCounters) / sizeof(int));
  for (int i = threadIdx.x; i < kWords; i += blockDim.x) p[i] = 0;
}

void launch_zero_counters(const GraphRec *recs, int ng_new, EngineCtl *ectl, cudaStream_t stream) {
  zero_counters_kernel<<<ng_new > 0 ? ng_new : 1, 128, 0, stream>>>(recs, ng_new, ectl);
}

size_t engine_dynamic_smem() { return sizeof(SoloCache); }

namespace {
size_t owned_need(int grid, int graphs, size_t tiles) {
  const size_t blocks = static_cast<size_t>(grid - 1);
  return owner::bytes_of(graphs, (tiles + blocks - 1) / blocks);
}
}  // namespace

// As many as leave L1 more than its last 28 KB (smem_of, owner_pass.cuh). With
// that little, lists are faster: 14 batches of 300 passes at most, milliseconds
// over lists and on owned rows: 3.0 million vertices of degree 7 35.2 and 29.8, 3.3
// million of degree 5 9.6 and 11.6, 3.5 million of degree 5 9.8 and 14.8, 3.6 million of
// degree 7 43.4 and 46.2.
constexpr int kOwnedVertices = 20320;
static_assert(owner::leaves_l1(owner::bytes_of(1, kOwnedVertices / owner::kTile) + owner::kPoolBytes, 10240));

unsigned owned_limit(int grid) { return grid > 1 ? static_cast<unsigned>(grid - 1) * kOwnedVertices : 0u; }

// Rows are loaded for the passes that follow: some 20 us for a million vertices, 60 for
// 2 and 75 for 3. A launch that may run 3 full-grid passes at most (pass limits, pass
// budget) runs them over lists: 100 steps of 2 passes over 32 graphs (560,000 vertices)
// 9.7 and 9.0 ms. From 1.75 million vertices on, a launch starts with 8 passes over
// lists, which a batch that goes on makes up for. 10 batches of 2, 8, 20 and 60 passes,
// milliseconds, rows loaded at once and after 8: 1.5 million vertices 2.2, 2.7, 3.3, 5.0
// and 1.9, 2.4, 3.4, 5.1; 2 million 2.8, 3.3, 4.0, 6.3 and 2.4, 2.8, 4.1, 6.2; 2.6 million
// 3.5, 4.1, 5.0, 7.7 and 3.0, 3.5, 5.0, 7.5; with 300 passes they differ by less than 1%.
int list_passes(size_t vertices) { return vertices < 1750000 ? 0 : 8; }

// Nor does a time slice that is hardly longer than the load. Four batches each over
// several graphs from a queue, milliseconds over lists and on owned rows: 80,000 vertices
// in all, slices of 20 us 19.7 and 15.8; 640,000, 30 us 26.8 and 39.3, 60 us 22.9 and
// 19.3; 1.6 million, 60 us 40.2 and 46.8, 120 us 35.4 and 30.4; 2.4 million, 200 us 49.1
// and 52.8, 400 us 46.5 and 48.5.
unsigned long long least_slice_ns(size_t vertices) {
  return vertices < 1750000 ? 15000 + vertices * 40 / 1000 : 1000000;
}

size_t owned_smem(int grid, int graphs, size_t vertices, size_t fixed, size_t most) {
  if (vertices > owned_limit(grid)) return 0;
  // the graphs' own records count as well
  const size_t need = owned_need(grid, graphs, vertices / owner::kTile);
  return owner::leaves_l1(need + owner::kPoolBytes, fixed) ? owner::smem_of(need, sizeof(SoloCache), fixed, most) : 0;
}

const void *owned_kernel_ptr() { return reinterpret_cast<const void *>(&engine_kernel<8, true>); }

const void *engine_kernel_ptr(int lanes) {
  switch (lanes) {
    case 1: return reinterpret_cast<const void *>(&engine_kernel<1, false>);
    case 4: return reinterpret_cast<const void *>(&engine_kernel<4, false>);
    case 8: return reinterpret_cast<const void *>(&engine_kernel<8, false>);
    case 16: return reinterpret_cast<const void *>(&engine_kernel<16, false>);
    case 32: return reinterpret_cast<const void *>(&engine_kernel<32, false>);
    default: return nullptr;
  }
}

}  // namespace engine
}  // namespace dlp
