// Host plan of the panel banks' level sweeps (panel_plan.hpp).
#include "panel_plan.hpp"

#include <algorithm>
#include <stdexcept>

#include "dense.hpp"

namespace pecs {

PanelTilesPlan plan_panel(const std::vector<const MfFactor*>& factors, int chunks, int min_ctas, int most_rows) {
  PanelTilesPlan P;
  const int n_sets = (int)factors.size();
  int n_levels = 0;
  for (const MfFactor* F : factors) {
    P.base.push_back((int)P.spans.size());
    for (int j = 0; j < (int)F->nodes.size(); ++j) {
      P.spans.emplace_back();
      n_levels = std::max(n_levels, F->nodes[j].height + 1);
    }
  }
  for (int q = 0; q < n_sets; ++q)
    dense::parallel_for((int)factors[q]->nodes.size(), 64, [&](int j) { P.spans[P.base[q] + j] = node_spans(*factors[q], j); });
  // update slots, and the nodes of each height
  std::vector<std::vector<int>> w_off(n_sets);
  std::vector<std::vector<std::pair<int, int>>> lv(n_levels);  // (set, node), set by set
  for (int q = 0; q < n_sets; ++q) {
    int w = 0;
    for (int j = 0; j < (int)factors[q]->nodes.size(); ++j) {
      w_off[q].push_back(w);
      w += factors[q]->nodes[j].m;
      lv[factors[q]->nodes[j].height].push_back({q, j});
    }
  }
  // records: the children's update slots that land on each front position
  P.dir[0].levels.resize(n_levels);
  {
    std::vector<std::vector<int>> fpos(n_sets), lists;
    for (int q = 0; q < n_sets; ++q) fpos[q].assign(factors[q]->n, -1);
    for (int l = 0; l < n_levels; ++l) {
      PanelLevel& L = P.dir[0].levels[l];
      for (auto [q, j] : lv[l]) {
        const MfNode& x = factors[q]->nodes[j];
        if (x.children.empty()) continue;
        const int f = x.s + x.m;
        for (int t = 0; t < f; ++t) fpos[q][t < x.s ? x.own[t] : x.upd[t - x.s]] = t;
        lists.assign(f, {});
        for (int c : x.children)
          for (int a = 0; a < factors[q]->nodes[c].m; ++a) {
            const int p = fpos[q][factors[q]->nodes[c].upd[a]];
            if (p < 0) throw std::runtime_error("extend-add map mismatch");
            lists[p].push_back(w_off[q][c] + a);
          }
        for (int t = 0; t < f; ++t) fpos[q][t < x.s ? x.own[t] : x.upd[t - x.s]] = -1;
        if (L.n_rec[q] == 0) L.rec[q] = (int)P.rec.size();
        L.n_rec[q] += f;
        for (int p = 0; p < f; ++p) P.rec.push_back(make_rec(p < x.s ? x.own[p] : ~(w_off[q][j] + p - x.s), lists[p], P.more));
      }
    }
  }
  for (int d = 0; d < 2; ++d) {
    const bool fwd = d == 0;
    PanelTilesPlan::Dir& D = P.dir[d];
    D.levels.resize(n_levels);
    for (int l = 0; l < n_levels; ++l) {
      PanelLevel& L = D.levels[l];
      const auto& nodes = lv[fwd ? l : n_levels - 1 - l];
      L.first = (int)D.tiles.size();
      auto rows_of = [&](const MfNode& x) { return fwd ? x.s + x.m : x.s; };
      // tiles of most_rows rows, half of them where those are fewer than min_ctas
      long long n = 0;
      for (auto [q, j] : nodes) n += (rows_of(factors[q]->nodes[j]) + most_rows - 1) / most_rows;
      const int cap = most_rows > kPanelRowsF64 && n * chunks < min_ctas ? most_rows / 2 : most_rows;
      for (auto [q, j] : nodes) {
        const MfNode& x = factors[q]->nodes[j];
        const NodeSpans& sp = P.spans[P.base[q] + j];
        const int rows = rows_of(x);
        // forward: no tile across the end of the own rows (their columns end where the
        // triangular part does) unless the node is one tile
        const bool two = fwd && x.m > 0 && rows > cap;
        for (int r0 = 0, r1; r0 < rows; r0 = r1) {
          const int end = two && r0 < x.s ? x.s : rows;
          r1 = std::min(end, r0 + cap);
          int k0 = 0, K = 0;
          sp.columns(fwd, x.s, x.m, r0, r1, k0, K);
          PanelTile t{};
          t.off = D.n_values;
          t.rows = r1 - r0;
          t.pad = cap <= 4 ? 4 : t.rows <= 8 ? 8 : (t.rows <= 16 ? 16 : 32);
          t.cols = K;
          t.set = q;
          t.idx = (int)D.idx.size();
          t.leaf = x.children.empty();
          t.npt = fwd && !t.leaf ? std::max(0, r1 - std::max(r0, x.s)) : 0;
          for (int k = 0; k < K; ++k) {
            const int c = fwd ? sp.order[k] : k0 + k;
            D.idx.push_back(c < x.s ? x.own[c] : ~x.upd[c - x.s]);
          }
          D.idx.resize((D.idx.size() + 3) & ~(size_t)3, 0);
          for (int r = r0; r < r0 + t.pad; ++r)
            D.idx.push_back(r >= r1 ? 0 : (r < x.s ? x.own[r] : ~(w_off[q][j] + r - x.s)));
          D.n_values += (long long)K * t.pad;
          D.node.push_back(j);
          D.row0.push_back(r0);
          D.col0.push_back(k0);
          D.tiles.push_back(t);
          ++L.n;
          L.cols = std::max(L.cols, K);
          L.pad = std::max(L.pad, t.pad);
          L.passes = L.passes || t.npt > 0;
        }
      }
    }
  }
  return P;
}

namespace {
template <typename T>
void pack(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, T* out) {
  const PanelTilesPlan::Dir& D = P.dir[d];
  dense::parallel_for((int)D.tiles.size(), 64, [&](int i) {
    const PanelTile& t = D.tiles[i];
    const MfFactor& F = *factors[t.set];
    const int j = D.node[i], s = F.nodes[j].s, f = s + F.nodes[j].m;
    const NodeSpans& sp = P.spans[P.base[t.set] + j];
    T* o = out + t.off;
    for (int k = 0; k < t.cols; ++k)
      for (int r = 0; r < t.pad; ++r) {
        const int row = D.row0[i] + r;
        double v = 0.0;
        if (r < t.rows) v = d == 0 ? F.Gf[j][(size_t)row * s + sp.order[k]] : F.Hb[j][(size_t)row * f + D.col0[i] + k];
        o[(size_t)k * t.pad + r] = (T)v;
      }
  });
}
}  // namespace

void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, double* out) {
  pack(P, factors, d, out);
}
void pack_panel(const PanelTilesPlan& P, const std::vector<const MfFactor*>& factors, int d, float* out) {
  pack(P, factors, d, out);
}

}  // namespace pecs
