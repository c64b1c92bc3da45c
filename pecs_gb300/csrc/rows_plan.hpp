// Tile plan of the few-right-hand-side solve sweeps (rows.cuh).  Host only.
#pragma once
#include <cstddef>
#include <vector>

#include "mf.hpp"

namespace pecs {

constexpr int kRowsThreads = 256;  // threads of a CTA
constexpr int kRowsMaxSets = 4;
constexpr int kRowsSlots = 7;      // child update slots in a record

constexpr int kRowsSms = 152;      // multiprocessors of a GB300

// The blocks hold triangular inverses (L11^-1 P, U11^-1): a tile leaves out the
// columns that are zero in all of its rows.  Forward, a node's columns are taken
// in the order of their first nonzero row, and a tile of the first s rows covers
// those that start above its end; backward, a tile covers the columns from the
// first one that reaches its rows or later ones.
struct NodeSpans {
  std::vector<int> order, start, reach;
  // columns [k0, k0 + K) of rows [r0, r1) of a node of s own and m update rows (forward:
  // places in `order`)
  void columns(bool fwd, int s, int m, int r0, int r1, int& k0, int& K) const;
};
NodeSpans node_spans(const MfFactor& F, int j);

// Where a front position's value comes from (forward): the right-hand side of
// dof src (update rows: their own slot) and up to kRowsSlots child update slots (-1: no more); with
// more of them the last entry is -2 - i, and more[i] holds their number, then them.
struct alignas(16) RowRec {
  int src;
  int slot[kRowsSlots];
};

// A tile: rows x cols values from value `off` on, [column][padded row], applied
// by one team of threads.  A batch (ts = 0): `pad` whole nodes of equal shape one
// after another, [node][column][row], a thread per output.
struct alignas(16) RowItem {
  int rows, pad, cols;  // rows, rows padded to the vector width (batch: nodes), columns
  int set;
  int src, dst;         // first column in the source list / records, first row in the destination list
  int pt, npt;          // forward: first record and number of the pass-through rows (the last npt rows)
  long long off;
  int magic;            // ceil(2^16 / (pad / values per vector))
  int node, row0;       // bank-wide node (batch: the first), first row
  int d, leaf;          // forward: first column in the set's assembled columns; node without children
  int kc;               // columns whose values are staged at a time
};

// Sizes of a launch's shared memory: the largest of its tiles.
struct RowShape {
  int cols = 0;  // columns
  int npt = 0;   // pass-through rows of nodes with children
  int vals = 0;  // values of one chunk of columns
  int chunks = 0;  // chunks of columns
};

// Shared memory of one team, in bytes from its slice: two barriers, then one or two
// buffers of tile values, the source values (overlaid by the partial sums) and the
// pass-through sums (forward).
struct RowsSmem {
  int kc = 1;                // staged columns per chunk
  unsigned buf = 0;          // bytes of one value buffer
  unsigned ds = 0, cu = 0;   // offsets
  unsigned team_bytes = 0;
};

constexpr size_t kRowsSmem = 220 * 1024;  // most of a CTA

// The layout for tiles of these sizes, teams of ts threads and chunks of rb right-hand
// sides; the teams of a CTA take kRowsSmem at most.
RowsSmem rows_smem(const RowShape& P, int vr, int rb, int ts);

// One tree level: its tiles (teams of ts threads), then its batches.
struct RowLevel {
  int first = 0, n_tile = 0, n_batch = 0, ts = kRowsThreads;
  int n_node = 0;  // nodes of the tiles
  bool leaf = true;  // no tile node has children
  RowShape shape;
  // forward, per set: the tile nodes' column and update records, and their
  // columns' first place among the set's assembled columns
  int col[kRowsMaxSets] = {}, n_col[kRowsMaxSets] = {}, d[kRowsMaxSets] = {}, upd[kRowsMaxSets] = {},
      n_upd[kRowsMaxSets] = {};
};

// Flow sweep: an entry is `count` tiles from item `first` on (a team of ts threads
// each), or a batch (ts = 0) of `count` nodes, in topological order.  Each tile, or
// node of a batch, has a RowSync (from `sync` on): the counter it waits for (-1:
// none) with its target, and the counter it adds one to (-1: none).
struct alignas(16) RowEntry {
  int ts, first, count, sync;
};
struct alignas(16) RowSync {
  int wait, target, signal, unused;
};

// A record with these child update slots (more than it holds: in `more`).
RowRec make_rec(int src, const std::vector<int>& slots, std::vector<int>& more);

struct RowsPlan {
  struct Node {
    int set, j, s, m, level[2], parent, w_off;
    bool leaf;
  };
  struct Dir {
    std::vector<RowItem> items;
    std::vector<RowLevel> levels;
    RowShape flow_shape[4];  // teams of 32, 64, 128, 256 threads
    std::vector<RowEntry> entries;
    std::vector<RowSync> sync;
    // sources: forward the columns' own dofs, backward own dofs, then ~update
    // dofs; destinations: own dofs, forward then update slots; nodes in level order
    std::vector<int> src, dst;
    std::vector<int> src0, dst0;  // first entry of each node
    std::vector<int> at, pos;     // nodes in level order, and each node's place there
    long long n_values = 0;
  };
  Dir dir[2];  // forward, backward
  std::vector<Node> nodes;
  std::vector<int> wtotal;           // update slots per set
  std::vector<RowRec> rec, upd;      // forward: columns (as dir[0].src), update rows
  std::vector<int> more;
  std::vector<NodeSpans> spans;      // per node
  long long entries = 0;             // stored values of the factors, zeros included
};

// vr: values per 16 bytes; max_nrhs: right-hand sides per set (0: unknown).
RowsPlan plan_rows(const std::vector<const MfFactor*>& factors, int vr, int max_nrhs);

// The values of direction d in the items' order (n_values of them).
void pack_rows(const RowsPlan& P, const std::vector<const MfFactor*>& factors, int d, double* out);
void pack_rows(const RowsPlan& P, const std::vector<const MfFactor*>& factors, int d, float* out);

}  // namespace pecs
