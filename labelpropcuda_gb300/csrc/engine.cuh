// Multi-graph batch engine: one cooperative persistent kernel applies one
// batch to each of up to kMaxGraphs resident graphs at once.
//
// Every phase of the per-batch update (see session_kernel.cuh for the phase
// map against the reference) walks a flattened work list: the per-graph item
// counts are prefix-summed in shared memory after each grid barrier and a
// work item is mapped back to (graph, local index) by binary search. Graphs
// converge independently: a graph whose frontier is empty (or that reached
// max_iter) contributes no items to later passes and its pass count is
// recorded; the launch ends when every graph has finished. A resident single
// graph (dlp_session) is the one-graph case of the same kernel.
//
// Continuous batching: a launch may be sliced (a pass budget or a time budget
// for its propagation). Graphs whose frontier is still live when the slice
// ends keep their whole propagation state in device memory (frontier sets,
// counters, both label buffers) and are continued by a later launch, which
// lists them after the graphs that start a new batch: phases A-F run over the
// new graphs only, the propagation passes over all of them, each graph at its
// own pass number (BatchArgs::pass0 + the launch's pass). A graph's batch ends
// (phase H, statistics) in the launch where its frontier empties.
#pragma once

#include "session_kernel.cuh"

namespace dlp {
namespace engine {

constexpr int kMaxGraphs = 1024;
// Frontier size below which propagation passes leave the full grid for one
// block (default 512, at most kSoloEntryMax). Tunable per engine. There is no
// mode on fewer blocks than all of them in between: with SumBarrier a pass over
// 600 to 2,000 rows takes 5.1 to 6.2 us on 152 blocks (3.2 on owned rows)
// and 7 to 8 us on 16.
constexpr int kSoloEntryDefault = 512;
constexpr int kSoloEntryMax = 1024;
constexpr int kSubEntryMax = 4096;  // dlp_config.subgrid_entry, accepted and without effect

constexpr int kOwnedTile = 32;  // a graph's vertices count in whole tiles (owner_pass.cuh)

struct GraphRec {
  session::DevState st;
  session::BatchArgs ba;
};

struct EngineCtl {
  SumBarrier bar;       // all blocks of the launch; zeroed before each launch
  int err;
  // Hand-back of a one-block stint: the pass at which it stopped and the
  // passes it ran, in slot (stint number & 1), so that the next stint cannot
  // overwrite a value a slow block has yet to read.
  int solo_k[2];
  int solo_passes[2];
  int solo_full[2];     // a one-block stint ended for lack of room
  int where;            // last phase block 0 reached (1..10)
  int where_pass;       // last propagation pass block 0 started
  // The launch's time slice ran out: a request to stop, written by thread 0 of
  // block 0 and read by every block at the top of a pass, (launch tag << 32) | the
  // pass at which to stop. A read at the top of pass k takes only a request naming
  // pass k, so a request written during pass k (for pass k + 1) is never seen early
  // by a block that is slow to start pass k.
  unsigned long long slice_stop;
  unsigned long long t_launch;  // global timer at the start of the launch (thread 0 of block 0)
  // Propagation passes run so far by mode, and the device time they took
  // (global timer): 0 one block, 1 of which by at most 16 warps, 2 unused,
  // 3 full grid. Written by thread 0 of block 0 only, once per launch.
  unsigned long long mode_passes[4];
  unsigned long long mode_ns[4];
};

struct EngineArgs {
  GraphRec *recs;
  int ng;       // graphs in the launch
  int ng_new;   // the first ng_new of them start a batch; the rest continue one
  EngineCtl *ectl;
  unsigned long long timeout_ns;
  int solo;  // bit 0: one-block passes; bit 2: one-block passes by the warps that hold rows only
  int fast_div;    // 1: the reference's fast-math division (dlp_config.arithmetic), else IEEE
  int solo_entry;  // total frontier at most this: one-block passes (<= kSoloEntryMax)
  int pass_budget;                // propagation passes this launch runs at most (0: no limit)
  unsigned long long slice_ns;    // propagation time after which the launch stops (0: no limit)
  int tag;                        // unique per launch (stop requests)
  float delta;                    // convergence threshold (the engine's, the same for every graph)
  // Owned passes (owner_pass.cuh): tiles of kOwnedTile vertices of all graphs of the
  // launch (0: passes over frontier lists), and the two mark planes, all zero
  // between stints.
  int tiles;
  int smem_bytes;                 // dynamic shared memory of the launch
  unsigned *marks;
  unsigned mark_plane;            // words of a plane
  int list_passes;                // full-grid passes over lists before rows are loaded
  int2 *progress;                 // per graph: {1 batch finished / 0 continues, passes so far}
};

// Zeroes the batch counters of the graphs that start a batch (recs[0..ng_new))
// and the launch's barrier.
void launch_zero_counters(const GraphRec *recs, int ng_new, EngineCtl *ectl, cudaStream_t stream);

// Launches over frontier lists only, by lanes per short row, and launches with
// owned passes.
const void *engine_kernel_ptr(int lanes);
const void *owned_kernel_ptr();
// Dynamic shared memory per block that every launch of the engine kernel needs
// (the one-block mode's).
size_t engine_dynamic_smem();
// Frees the engine's mark planes, for good, when they take more than `room` bytes:
// what a server's budget leaves beside graphs, staging and scratch. Passes then run
// over frontier lists.
void fit_marks(dlp_engine *e, size_t room);
// Vertices (in whole tiles) of a launch up to which a grid can own them.
unsigned owned_limit(int grid);
// Full-grid passes over lists before a launch of that many vertices loads rows; the
// most passes that a launch may run over lists only, and the shortest time slice of a
// launch that loads rows.
int list_passes(size_t vertices);
constexpr int kListOnly = 3;
unsigned long long least_slice_ns(size_t vertices);
// Dynamic shared memory of a launch with owned passes over that many graphs and
// vertices (in whole tiles), beside `fixed` bytes of static shared memory and at
// most `most`; 0 when they do not fit.
size_t owned_smem(int grid, int graphs, size_t vertices, size_t fixed, size_t most);

}  // namespace engine
}  // namespace dlp
