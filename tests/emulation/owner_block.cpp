// One block's owned passes (csrc/owner_pass.cuh) on the CPU, over a graph that
// checks every vertex and entry it is asked for.
//   owner_block remainder   a partial last tile whose rows do not fit the pool
//   owner_block counter     rows at the end of their visit counters beside a wide row
//   owner_block mixed       passes over short, long and wide rows, listed and by tiles,
//                           marked and dense, with and without room in the pool
//   owner_block shared      the shared memory of a launch, over all sizes
#include "owner_pass.cuh"

#include <cstdio>
#include <string>

alignas(16) unsigned char dlp::owner::g_smem[1 << 17];

using namespace dlp::owner;

struct Checked {
  static constexpr bool kCounts = false;
  int n;
  std::vector<int> start, col;
  std::vector<float> val;
  mutable int bad = 0;  // lookups outside the graph
  int graphs() const { return 1; }
  int nodes(int) const { return n; }
  bool vertex(int v) const {
    const bool ok = v >= 0 && v < n;
    if (!ok) __atomic_fetch_add(&bad, 1, __ATOMIC_SEQ_CST);
    return ok;
  }
  int2 row(int, int v) const { return vertex(v) ? make_int2(start[v], start[v + 1] - start[v]) : make_int2(0, 0); }
  bool active(int, int v) const { return vertex(v); }
  bool markable(int, int v) const { return vertex(v); }
  void entry(int, int at, int &v, float &w) const {
    if (at < 0 || at >= start[n]) {
      __atomic_fetch_add(&bad, 1, __ATOMIC_SEQ_CST);
      return;
    }
    v = col[at];
    w = val[at];
  }
  template <int N>
  void entries(int g, int first, int e, int step, int len, int (&v)[N], float (&w)[N]) const {
    for (int j = 0; j < N; ++j) {
      v[j] = -1;
      if (e + j * step < len) entry(g, first + e + j * step, v[j], w[j]);
    }
  }
  template <int N>
  unsigned markables(int g, const int (&v)[N]) const {
    unsigned can = 0;
    for (int j = 0; j < N; ++j) can |= (v[j] >= 0 && markable(g, v[j]) ? 1u : 0u) << j;
    return can;
  }
};

// Rows of `len(v)` entries at the vertices after v, weights by position.
template <class Len>
Checked graph(int n, Len len) {
  Checked g;
  g.n = n;
  g.start.assign(1, 0);
  for (int v = 0; v < n; ++v) {
    for (int e = 0; e < len(v); ++e) {
      g.col.push_back((v + 1 + e) % n);
      g.val.push_back(0.25f + 0.5f * static_cast<float>((v + e) % 7));
    }
    g.start.push_back(static_cast<int>(g.col.size()));
  }
  return g;
}

struct Run {
  Checked g;
  Store s;
  std::vector<float> lab[2];
  std::vector<unsigned> marks[2];

  Run(Checked graph_, int pool) : g(std::move(graph_)) {
    gridDim.x = 2;
    const int tiles = (g.n + kTile - 1) / kTile;
    s = store(static_cast<int>(bytes_of(1, tiles) + 8 * pool), 1, tiles);
    for (int p = 0; p < 2; ++p) {
      marks[p].assign(tiles * kTile, 0);
      for (int v = 0; v < g.n; ++v) lab[p].push_back(static_cast<float>(v % 5) / 4.0f);
    }
    Head &h = s.head();
    std::memset(&h, 0, sizeof h);
    h.first_limit = 0x7fffffff;
    Local &l = s.graph(0);
    l.lab[0] = lab[0].data();
    l.lab[1] = lab[1].data();
    l.flat = 0;
    l.limit = 0x7fffffff;
  }
  // The average that the pass has to give vertex v from buffer `src`.
  float average(int src, int v) const {
    double w = 0, l = 0;
    for (int e = g.start[v]; e < g.start[v + 1]; ++e) {
      w += g.val[e];
      l += static_cast<double>(g.val[e]) * lab[src][g.col[e]];
    }
    return static_cast<float>(l / w);
  }
};

// What a pass over the marked vertices has to leave: labels, marks, and whether a label
// moved.
struct Expected {
  std::vector<float> lab;
  std::vector<unsigned> marks;
  int rows = 0;
  bool moved = false;
};
Expected expected(const Run &r, int k, float delta, bool dense) {
  Expected x{r.lab[(k & 1) ^ 1], std::vector<unsigned>(r.marks[0].size(), 0)};
  for (int v = 0; v < r.g.n; ++v) {
    if (!dense && !r.marks[k & 1][v]) continue;
    ++x.rows;
    x.lab[v] = r.g.start[v] == r.g.start[v + 1] ? r.lab[k & 1][v] : r.average(k & 1, v);
    if (std::fabs(x.lab[v] - r.lab[k & 1][v]) <= delta) continue;
    x.moved = true;
    x.marks[v] = 1;
    for (int e = r.g.start[v]; e < r.g.start[v + 1]; ++e) x.marks[r.g.col[e]] = 1;
  }
  return x;
}

// Passes over 300 vertices (ten tiles, the last partial) of a block of `threads`.
void mixed(unsigned threads, int pool, bool dense, int &outside, int &wrong) {
  const auto len = [](int v) { return v % 97 == 5 ? 290 : v % 9 == 0 ? 33 + v % 40 : v % 5 == 0 ? 9 + v % 24 : v % 9; };
  Run r(graph(300, len), pool);
  Head &h = r.s.head();
  const float delta = 1e-3f;
  for (int v = 0; v < r.g.n; ++v) r.marks[0][v] = v % 3 == 0;
  run_block(1, threads, [&] {
    load(r.s, r.g);
    __syncthreads();
    if (dense) list_all(r.s);
  });
  for (int k = 0; k < 4; ++k) {
    const Expected x = expected(r, k, delta, dense);
    unsigned *const own = r.marks[k & 1].data(), *const next = r.marks[(k & 1) ^ 1].data();
    const bool tiles = threads >= 320;
    run_block(1, threads, [&] {
      auto each = [](int) {};
      if (dense) dense_pass(r.s, r.g, k, delta);
      else if (tiles) tile_pass(r.s, r.g, own, next, k, delta, false, each);
      else pass(r.s, r.g, own, next, k, delta, false, each);
    });
    for (int v = 0; v < r.g.n; ++v) {
      wrong += std::fabs(r.lab[(k & 1) ^ 1][v] - x.lab[v]) > 1e-6f;
      if (!dense) wrong += r.marks[(k & 1) ^ 1][v] != x.marks[v] || own[v] != 0;
    }
    for (size_t i = r.g.n; i < r.marks[0].size(); ++i) wrong += r.marks[0][i] != 0 || r.marks[1][i] != 0;
    wrong += (h.moved != 0) != x.moved;
    if (!dense) {
      wrong += (h.count & 0xffff) + (h.count >> 16) + h.wide != x.rows;
      h.count = h.wide = h.wide_at = 0;
    }
    h.moved = 0;
  }
  outside += r.g.bad;
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  int wrong = 0;
  if (what == "remainder") {
    Run r(graph(40, [](int v) { return v % 4 ? 30 : 5; }), 100);
    for (int v = 0; v < r.g.n; ++v) r.marks[0][v] = 1;
    run_block(1, 64, [&] {
      load(r.s, r.g);
      __syncthreads();
      tile_pass(r.s, r.g, r.marks[0].data(), r.marks[1].data(), 0, 1e-4f, false, [](int) {});
    });
    for (int v = 0; v < r.g.n; ++v) wrong += std::fabs(r.lab[1][v] - r.average(0, v)) > 1e-5f;
    for (int v = r.g.n; v < 64; ++v) wrong += r.marks[1][v] != 0;
    std::printf("outside %d wrong %d\n", r.g.bad, wrong);
  } else if (what == "counter") {
    // Vertex 3 runs in pass 0, vertex 0 (40 entries) in pass 1. A reader of the
    // counters that has not cleared them for 32,767 passes would see this:
    Run r(graph(96, [](int v) { return v == 0 ? 40 : 5; }), 1000);
    r.marks[0][3] = 1;
    run_block(1, 32, [&] {
      load(r.s, r.g);
      __syncthreads();
      if (threadIdx.x == 0) r.s.visits(3) = 0x7fff;
      __syncthreads();
      auto each = [](int) {};
      pass(r.s, r.g, r.marks[0].data(), r.marks[1].data(), 0, 2.0f, false, each);
      __syncthreads();
      if (threadIdx.x == 0) {
        r.s.head().count = r.s.head().wide = r.s.head().wide_at = 0;
        r.marks[1][0] = 1;
        r.lab[0][3] = 7.0f;  // what pass 1 must not touch
      }
      __syncthreads();
      pass(r.s, r.g, r.marks[1].data(), r.marks[0].data(), 1, 2.0f, false, each);
    });
    wrong += std::fabs(r.lab[0][0] - r.average(1, 0)) > 1e-5f;
    std::printf("outside %d wrong %d label %.1f\n", r.g.bad, wrong, r.lab[0][3]);
  } else if (what == "mixed") {
    int outside = 0;
    for (int pool : {20, 2000, 12000})
      for (unsigned threads : {64u, 320u}) {
        mixed(threads, pool, false, outside, wrong);
        mixed(threads, pool, true, outside, wrong);
      }
    std::printf("outside %d wrong %d\n", outside, wrong);
  } else if (what == "shared") {
    constexpr size_t kFixed = 10192, kMost = 222240, kLeast = 110768;
    for (size_t need = 0; need <= kMost; need += 16) {
      const size_t bytes = smem_of(need, kLeast, kFixed, kMost);
      wrong += bytes > kMost || bytes % 16 != 0 || bytes < need || bytes < kLeast;
      // L1 keeps more than its last 28 KB whenever that can be, and no step is taken
      // that the vertices and their pool do not ask for
      wrong += leaves_l1(need, kFixed) && bytes + kFixed + kSystemBytes > kSteps[3];
      for (size_t step : kSteps)
        wrong += std::max(need + kPoolBytes, kLeast) + kFixed + kSystemBytes <= step &&
                 bytes + kFixed + kSystemBytes > step;
    }
    std::printf("wrong %d\n", wrong);
  } else {
    return 2;
  }
  return 0;
}
