// One block's owned passes (csrc/owner_pass.cuh) on the CPU, over a graph that
// checks every vertex and entry it is asked for.
//   owner_block remainder   a partial last tile whose rows do not fit the pool
//   owner_block counter     rows at the end of their visit counters beside a wide row
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
  } else {
    return 2;
  }
  return 0;
}
