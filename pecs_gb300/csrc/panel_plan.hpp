// Tile plan of the panel banks' level sweeps (solve.cuh).  Host only.
#pragma once
#include <vector>

#include "rows_plan.hpp"

namespace pecs {

// rows x cols values from value `off` on, [column][padded row], for one CTA and a
// chunk of right-hand sides.
struct alignas(16) PanelTile {
  long long off;
  int rows, pad, cols;  // rows, rows padded to 8, 16 or 32, columns
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

// chunks: chunks of 32 right-hand sides per set; min_ctas: tiles x chunks that a level
// should have (else shorter tiles)
PanelTilesPlan plan_panel(const std::vector<const MfFactor*>& factors, int chunks, int min_ctas);

void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, double* out);
void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, float* out);

}  // namespace pecs
