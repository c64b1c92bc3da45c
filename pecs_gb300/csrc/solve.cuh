// Application of multifrontal LU factors on the GPU, level by level or as a
// dataflow sweep (flow plans below).
//
// A FactorBank holds one or more factors (mf.hpp) concatenated node-wise.  Each
// factor is bound to a "RHS set": a list of right-hand sides that share the
// factor (e.g. electrons and holes of every instance when their mobilities
// are equal), so that every stored factor entry read from HBM is applied to
// all of them.  One or two kernel launches process one tree level of every factor in
// the bank.  Few right-hand sides per set: rows.cuh.  Many: each node's block is a
// small dense GEMM: forward, a level's columns -- right-hand side minus the children's
// updates -- are assembled once per node, then every tile of rows takes its packed
// values by one bulk copy and the vectors' rows (interleaved layout: a dof's values
// are contiguous) and multiplies them in register tiles.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.hpp"
#include "mf.hpp"
#include "panel_plan.hpp"
#include "rows.cuh"

namespace pecs {

constexpr int kMaxSets = 4;
constexpr int kTargetCtas = 152; // SMs of a GB300: FP32 levels with fewer tiles take shorter ones
constexpr int kSolveThreads = 256;
constexpr int kPanelMinRhs = 32;  // right-hand sides per set from which banks use the panel kernels

// Flow sweeps and leaf warps: device pointers, passed by value to kernels.
struct BankView {
  const int* own_idx;
  const int* upd_idx;
  const int* cmap_ptr;
  const int* cmap_idx;
  const void* G;
  const void* H;
};

// Interleaved layout: all right-hand sides of a set in one buffer, element
// (dof d, rhs r) at d * nrhs + r, so a dof's values are contiguous.
struct IlSetView {
  int nrhs;
  const double* b;
  double* y;
  double* w;  // update vectors, set_wtotal(set) x nrhs
  double* x;
};

struct IlSetsView {
  IlSetView set[kMaxSets];
};

// Interleaved layout with single-precision sweep vectors (FP32 factors on the
// panel path): b, y, update vectors and x are float -- they carry the FP32
// factors' results; refinement forms residuals in double-float and adds the
// correction to the solution outside the sweep.
struct IlSetViewF {
  int nrhs;
  const float* b;
  float* y;
  float* w;
  float* x;
};

struct IlSetsViewF {
  IlSetViewF set[kMaxSets];
};

// Device pointers of one level's plan; `val` holds the plan's values from val0 on.
struct TilesView {
  const PanelTile* tiles;
  const void* val;
  long long val0;
  const int* idx;
  const RowRec* rec;
  const int* more;
};

// A row range of one node and everything about the node that the flow and leaf kernels
// need, so that a single round of loads starts it.
struct __align__(16) PanelItem {
  int4 a;  // node, row0, row1, rows per tile
  int4 b;  // s, m, RHS set, update-vector offset
  int4 c;  // block offset (low, high 32 bits), own-index offset, update-index offset
  int4 d;  // child-map pointer offset, first child-map entry, child-map entries, unused
  int kc = 0;  // staged columns per chunk
  int unused[3];
};

// Factor values on the device, FP64 or FP32 as the bank's.
struct BankValues {
  DBuf<double> f64;
  DBuf<float> f32;
  const void* p() const { return f64.p ? (const void*)f64.p : (const void*)f32.p; }
  long long bytes() const { return (long long)(f64.n * 8 + f32.n * 4); }
  void release() { f64.release(), f32.release(); }
};

// How a panel level is launched.
struct PanelOption {
  int kind = -1;  // -1 untuned, 0 tiles, 2 leaf warps
  int warps = 8;  // tiles: warps per CTA (4 or 8)
  int n = 1;      // tiles: 32-right-hand-side groups per CTA; leaf warps: right-hand sides per lane
};

struct PanelPlan {
  PanelLevel tiles;      // panel_plan.hpp
  BankValues val;          // the tiles' values
  long long val0 = 0;      // ... from this one of the plan on
  long long n_val = 0;     // ... so many
  bool assembled = false;  // forward: nodes with children, whose positions are assembled first
  DBuf<PanelItem> warp;  // leaf levels: one item per node, a warp each (else empty)
  BankValues warp_val;   // ... and the nodes' blocks, column-major
  long long n_warp_val = 0;
  int max_k = 0;         // leaf levels: largest column count
  int warp_rows = 0;     // leaf levels: most rows of a node
  PanelOption tuned;     // the autotuner's choice (kind -1: heuristic)
  int launches() const { return tiles.n == 0 ? 0 : (assembled ? 2 : 1); }
};

// A flow sweep of one direction (one persistent launch; solve.cu): work
// entries in topological order, the items they name, and per item the node
// counter it waits on (with its target) and the one it signals.
struct FlowPlan {
  int top = 0;       // tree levels it covers, from the root side (the rest: level launches)
  int rpl = 0;       // right-hand sides per lane (32 * rpl per chunk)
  int n_chunks = 0;  // right-hand-side chunks the entries cover
  int n_entries = 0;
  int kc_cap = 0, ds_rows = 0, ri_max = 0, sc_rows = 0, max_s = 1, max_f = 1, cm_cap = 0, nbuf = 1;
  int warp_max_k = 0, warp_rows_pad = 0;
  size_t smem = 0;
  int grid = 0;      // persistent CTAs (resident capacity, at most one per entry)
  DBuf<int4> entries, sync;
  DBuf<PanelItem> items;
};

// Host description of the factor tree a flow plan is built from (bank-wide
// node numbering; per node: sizes, RHS set, offsets, child-map pointer and
// parent, and the nodes of each height).
struct FlowNodes {
  const std::vector<int>& s;
  const std::vector<int>& m;
  const std::vector<int>& node_set;
  const std::vector<int>& w_off;
  const std::vector<int>& own_off;
  const std::vector<int>& upd_off;
  const std::vector<int>& cm_off;
  const std::vector<int>& cmap_ptr;
  const std::vector<long long>& goff;
  const std::vector<long long>& hoff;
  const std::vector<int>& parent;
  std::vector<std::vector<int>> up, down;  // by height, from the leaves and from the root
};

// A flow plan before upload: the launch shape, the items with their waits and
// signals ((wait counter or -1, target, signal counter or -1, 0)), and the
// entries in ticket order ((kind, first item, item count, RHS chunk)).
struct FlowPlanHost {
  bool ok = false;  // false: its staging does not fit in shared memory
  int n_chunks = 0;
  int kc_cap = 1, ds_rows = 1, ri_max = 4, sc_rows = 0, max_s = 1, max_f = 1, cm_cap = 0, nbuf = 1;
  int warp_max_k = 0, warp_rows_pad = 0;
  size_t smem = 0;
  std::vector<PanelItem> items;
  std::vector<int4> sync, entries;
};

// Builds one direction's flow plan over the `top` tree levels nearest the root
// (the greatest heights; top >= the level count: all of them) for rpl right-hand sides per lane and at most
// max_nrhs right-hand sides per set (host only; esz: bytes per value; kc_max:
// staged block columns per chunk; n_sm: multiprocessors to fill).
FlowPlanHost plan_flow(const FlowNodes& nd, bool forward, int top, int rpl, int max_nrhs, int kc_max, int esz,
                       int n_sm);

struct PanelTuning {
  int chunk = 0;     // most staged block columns per chunk (0: what shared memory holds)
  int min_ctas = 0;  // CTAs a level must reach before shorter tiles are used (0: one per SM)
  bool flow = true;      // hold what the flow sweeps read until one is chosen or none
  bool options = true;   // ... and what every option of a level reads (autotune needs both)
};

class FactorBank {
 public:
  // factors[i] is bound to RHS set i.  precision: PECS_PREC_FP64 or FP32_IR.
  // panel: many right-hand sides per set (the panel kernels, interleaved layout only).
  // max_nrhs: the most right-hand sides any set will carry
  void build(const std::vector<const MfFactor*>& factors, int precision, bool panel = false,
             PanelTuning tuning = PanelTuning(), int max_nrhs = 0);
  // y = forward(b), x = backward(y); w is workspace.  All sets must be bound.
  void solve(const RowSets& sets, int max_nrhs, cudaStream_t st) const;  // few right-hand sides
  void load_row_kernels(int most_rhs) const { rows_.load_kernels(most_rhs); }
  void solve(const IlSetsView& sets, int max_nrhs, cudaStream_t st) const;
  void solve(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st) const;
  int set_wtotal(int set) const { return set_wtotal_[set]; }
  int precision() const { return prec_; }
  long long entries() const { return entries_; }
  // Device bytes of the factor values, and those that one sweep reads: zeros outside the
  // blocks' triangles are left out, rows padded.  A panel bank holds several forms of
  // its blocks until its kernels are chosen, then one -- with a flow sweep two.
  long long bytes() const;
  long long sweep_bytes() const;
  int kernel_launches_per_solve() const;
  bool panel() const { return panel_; }
  // Panel banks: choose each level's tiling option by timing whole sweeps on
  // these right-hand sides (the sweep's outputs are garbage afterwards).
  // tuned_ms(): the tuned sweep's time.
  // flow_mode: 0 = the flow sweep when it times faster than the tuned levels,
  // 1 = the fastest flow sweep wherever one applies, -1 = levels only.
  void autotune(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st, int reps = 3, int flow_mode = 0);
  void autotune(const IlSetsView& sets, int max_nrhs, cudaStream_t st, int reps = 3, int flow_mode = 0);
  // Few-right-hand-side banks: time the level sweep against the flow sweep on
  // these sets (a few sweeps each; outputs are garbage afterwards) and keep
  // the faster (flow_mode 0), the flow sweep (1) or the levels (-1).
  void tune_rows_flow(const IlSetsView& sets, int max_nrhs, cudaStream_t st, int flow_mode = 0, int reps = 3);
  bool rows_flow() const { return !panel_ && rows_.flow_on(); }
  // Untuned banks: the flow sweep with the most right-hand sides per lane that
  // applies to these sets (the level sweep if none does).
  void force_flow(const IlSetsViewF& sets, int max_nrhs);
  void force_flow(const IlSetsView& sets, int max_nrhs);
  double tuned_ms() const { return panel_ ? tuned_ms_ : rows_.tuned_ms(); }
  // Panel banks: right-hand sides per lane of the flow sweep in use (0: every
  // level its own launch), and the tree levels it covers from the root side.
  int flow_rpl() const { return flow_sel_ < 0 ? 0 : flow_cfg_[flow_sel_].rpl; }
  int flow_top() const {
    return rows_flow() ? rows_.n_levels() : (flow_sel_ < 0 ? 0 : flow_cfg_[flow_sel_].top);
  }
  // 1 if a flow sweep's wait ran out since the bank was built or the flag was
  // last cleared (that sweep's results were written as NaN); synchronises
  int flow_error(bool clear = false) const;
  // Diagnostic: the next forward flow sweep finds the first factor's root
  // counter far below its target, so that root's waits run out.
  void debug_arm_flow_stall() const;
  // Diagnostic: device time of each level launch of one sweep (forward levels,
  // then backward), CUDA events recorded between the launches, mean of reps
  // sweeps after one warm-up; the events keep consecutive levels from
  // overlapping, so the times are upper bounds of the in-sweep ones.
  std::vector<double> time_levels(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st, int reps) const;
  int tune_launches() const { return tune_launches_; }

 private:
  int prec_ = PECS_PREC_FP64;
  int n_sets_ = 0, max_nrhs_ = 0;
  int set_wtotal_[kMaxSets] = {0, 0, 0, 0};
  long long entries_ = 0;
  DBuf<int> own_idx_, upd_idx_, cmap_ptr_, cmap_idx_;
  BankValues G_, H_;  // flow sweeps: every block, column-major
  std::vector<PanelPlan> pfwd_, pbwd_;
  bool panel_ = false;
  PanelTuning tune_;
  DBuf<PanelTile> tiles_[2];  // level sweeps: tiles and their index lists per direction
  DBuf<int> tidx_[2], more_;
  DBuf<RowRec> rec_;
  TilesView tiles_view(int d, const PanelPlan& L) const;
  template <typename SVT>
  void solve_panel(const SVT& sets, int max_nrhs, cudaStream_t st) const;
  template <typename SVT>
  void autotune_panel(const SVT& sets, int max_nrhs, cudaStream_t st, int reps, int flow_mode);
  template <typename SVT>
  void force_flow_impl(const SVT& sets, int max_nrhs);
  template <typename SVT>
  int panel_rpl(const SVT& sets, int max_nrhs) const;
  double tuned_ms_ = 0.0;
  int tune_launches_ = 0;
  // flow sweeps built at creation: levels covered from the root side x staged
  // columns per chunk x right-hand sides per lane, both directions each
  struct FlowConfig {
    int top = 0, kc = 0, rpl = 0;
    FlowPlan plan[2];  // forward, backward
    long long values = 0;  // factor values that both read
  };
  std::vector<FlowConfig> flow_cfg_;
  int flow_sel_ = -1;     // the configuration in use (-1: level launches only)
  DBuf<int> flow_state_;  // [2][nodes] counters, 2 tickets, error flag
  int n_nodes_ = 0;
  int stall_node_ = -1;  // the first factor's root (debug_arm_flow_stall)
  RowsSweep rows_;       // banks with few right-hand sides per set (not panel_)
  RowSets row_sets(const IlSetsView& sets) const;
  void release_unused();
  template <typename SVT>
  bool flow_ok(const SVT& sets, int max_nrhs, int cfg) const;
  template <typename SVT>
  void solve_flow(const SVT& sets, int max_nrhs, int cfg, cudaStream_t st) const;
  BankView view() const;
};

}  // namespace pecs
