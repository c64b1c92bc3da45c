// Tile plan of the panel banks' level sweeps (solve.cuh).  Host only.
#pragma once
#include <vector>

#include "rows_plan.hpp"

namespace pecs {

// rows x cols values from value `off` on, [column][padded row], for one CTA and a
// chunk of right-hand sides.
struct alignas(16) PanelTile {
  long long off;
  int rows, pad, cols;  // rows, rows padded to 8, 16 or 32 (FP64: 4), columns
  int set;
  int idx;   // the columns' sources (padded to a multiple of 4), then the rows' destinations
  int npt;   // forward: the last npt rows add what the assembly wrote to their update slots
  int leaf;  // forward: node without children (columns read from the right-hand side)
  int unused[3];
};

// One tree level of a direction.
struct PanelLevel {
  int first = 0, n = 0;      // tiles
  int cols = 0, pad = 0;     // the most of a tile
  bool passes = false;       // a tile has pass-through rows
  // forward, per set: records of the front positions of nodes with children
  int rec[kRowsMaxSets] = {}, n_rec[kRowsMaxSets] = {};
};

struct PanelTilesPlan {
  struct Dir {
    std::vector<PanelTile> tiles;
    std::vector<PanelLevel> levels;  // forward by height, backward from the greatest height down
    std::vector<int> idx;
    long long n_values = 0;
    std::vector<int> node, row0, col0;  // of each tile (packing)
  };
  Dir dir[2];  // forward, backward
  // Forward, columns: own dof; rows: own dof or ~update slot.  Backward, columns: own
  // dof or ~update dof; rows: own dof.  Records: src as the forward rows.
  std::vector<RowRec> rec;
  std::vector<int> more;
  std::vector<NodeSpans> spans;  // per node, bank-wide
  std::vector<int> base;         // first node of each set
};

// Rows of a tile.  FP32 levels are bound by latency and the vectors' reading, so tiles
// are tall.  FP64 levels are bound by the FP64 unit (2 operations a clock: a tile of 32 x 32
// sums and 100 columns keeps a multiprocessor for 25 us), so what counts is that every
// multiprocessor has the same work and that no operation goes to padding.  us per
// carrier / Poisson sweep for 32 rows (16 on small levels), 8 (4 on small levels), 4:
// 16x16+15x16 cells, 33 instances 304 / 165, 202 / 91, 207 / 94; 33x31+32x31, 66 instances
// 1,547 / 453, 1,126 / 273, 1,069 / 276; 64x64+63x64, 64 instances 5,104 / 979, 4,117 / 699,
// 3,994 / 644.
constexpr int kPanelRowsF32 = 32, kPanelRowsF64 = 4;

// chunks: chunks of 32 right-hand sides per set; min_ctas: tiles x chunks that a level
// should have (else shorter tiles); most_rows: kPanelRowsF32 or kPanelRowsF64
PanelTilesPlan plan_panel(const std::vector<const MfFactor*>& factors, int chunks, int min_ctas,
                          int most_rows = kPanelRowsF32);

void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, double* out);
void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, float* out);

}  // namespace pecs
