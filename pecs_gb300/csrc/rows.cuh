// Solve sweeps for few right-hand sides per set (fewer than kPanelMinRhs): the
// plain single-instance path, small instance groups and the drop-in solver.
//
// Every tree node applies a dense block (Gf forward, Hb backward; mf.hpp) to a
// short vector per right-hand side.  A block is cut into row tiles; a tile's
// values are stored one after another in the order the kernel reads them
// ([column][row], rows padded to a 16-byte vector), so every load of a factor
// value is a coalesced 16-byte load whatever the node's size.  A team of 32 to
// 256 threads applies a tile to a chunk of right-hand sides: its threads split
// the tile's columns, keep a few rows x all right-hand sides of the chunk in
// registers, and add their partial sums in shared memory in a fixed order.
// Small leaves of FP64 factors go in batches, a thread per output.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.hpp"
#include "mf.hpp"
#include "rows_plan.hpp"

namespace pecs {

// Right-hand sides and solutions of one set: element (dof d, rhs r) at
// d * sd + r * sr, so interleaved buffers (sd = nrhs, sr = 1) and one vector
// after another (sd = 1, sr = n) are both read in place.  y and w are the
// sweep's own scratch, interleaved ([dof][rhs]).
struct RowSet {
  int nrhs = 0;
  int n = 0;  // dofs
  int sd = 0;
  long long sr = 0;
  const double* b = nullptr;
  double* x = nullptr;  // solutions (written)
  // scratch, interleaved: forward results (n x nrhs doubles of room), update
  // vectors (set_wtotal x nrhs) and, optional, assembled columns (n x nrhs; may be
  // x where x is interleaved).  FP32 factors keep y in single precision -- their
  // products' own -- with a copy of x behind it.
  double* y = nullptr;
  double* w = nullptr;
  double* d = nullptr;
};

struct RowSets {
  RowSet set[kRowsMaxSets];
};

struct RowsDirView {
  const void* val;
  const RowItem* items;
  const int* src;
  const int* dst;
  const RowRec* rec;
  const RowRec* upd;
  const int* more;
};

class RowsSweep {
 public:
  void build(const std::vector<const MfFactor*>& factors, int precision, int max_nrhs);
  // y = forward(b), x = backward(y) for every set
  void solve(const RowSets& sets, int max_nrhs, cudaStream_t st) const;
  // Loads the kernels of every solve of 1 to most_rhs right-hand sides without
  // assembled columns, so that those solves load nothing themselves.
  void load_kernels(int most_rhs) const;
  int set_wtotal(int set) const { return wtotal_[set]; }
  int dofs(int set) const { return dofs_[set]; }
  long long entries() const { return entries_; }
  long long bytes() const { return bytes_; }
  // launches of one solve whose sets have room for assembled columns
  int launches_per_solve(int max_nrhs) const;
  int n_levels() const { return (int)dir_[0].levels.size(); }
  // The flow sweep (one persistent launch per direction instead of one per
  // level): on when it times faster (mode 0), wherever it applies (1), never
  // (-1).  It applies when one chunk holds all right-hand sides of a set.
  void tune_flow(const RowSets& sets, int max_nrhs, cudaStream_t st, int mode, int reps);
  bool flow_on() const { return flow_on_; }
  double tuned_ms() const { return tuned_ms_; }
  int flow_error(bool clear) const;
  void debug_arm_flow_stall() const;

 private:
  template <typename T, int RB>
  void solve_flow(const RowSets& sets, cudaStream_t st) const;
  template <typename T, int RB>
  void ready() const;
  int prec_ = PECS_PREC_FP64;
  int n_sets_ = 0;
  int wtotal_[kRowsMaxSets] = {0, 0, 0, 0}, dofs_[kRowsMaxSets] = {0, 0, 0, 0};
  long long entries_ = 0, bytes_ = 0;
  struct Dir {
    DBuf<double> v64;
    DBuf<float> v32;
    DBuf<RowItem> items;
    DBuf<int> src, dst;
    std::vector<RowLevel> levels;
    DBuf<RowEntry> entries;  // flow sweep
    DBuf<RowSync> sync;
    RowShape flow_shape[4];
    int n_entries = 0;
  };
  RowsDirView view(int d) const {
    const Dir& D = dir_[d];
    return RowsDirView{D.v64.p ? (const void*)D.v64.p : (const void*)D.v32.p, D.items.p, D.src.p, D.dst.p,
                       rec_.p, upd_.p, more_.p};
  }
  DBuf<RowRec> rec_, upd_;
  DBuf<int> more_;
  Dir dir_[2];
  DBuf<int> flow_state_;       // [2][nodes] counters, 2 tickets, error flag
  int n_nodes_ = 0, stall_node_ = -1;
  bool flow_on_ = false;
  // launch state of the chunk width last used (0: none yet)
  struct FlowLaunch {
    int rb = 0, grid[2] = {0, 0};
    size_t bytes[2] = {0, 0};
  };
  mutable FlowLaunch flow_;
  mutable int ready_rb_ = 0;
  double tuned_ms_ = 0.0;
};

}  // namespace pecs
