// Tile plan of the few-right-hand-side solve sweeps (rows_plan.hpp).
#include "rows_plan.hpp"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <stdexcept>

#include "dense.hpp"

namespace pecs {

NodeSpans node_spans(const MfFactor& F, int j) {
  NodeSpans S;
  const int s = F.nodes[j].s, f = s + F.nodes[j].m;
  const std::vector<double>&G = F.Gf[j], &H = F.Hb[j];
  std::vector<int> first(s, s);
  S.order.resize(s), S.start.resize(s), S.reach.assign(s + 1, s);
  for (int r = 0; r < s; ++r)
    for (int c = 0; c < s; ++c)
      if (first[c] == s && G[(size_t)r * s + c] != 0.0) first[c] = r;
  std::iota(S.order.begin(), S.order.end(), 0);
  std::stable_sort(S.order.begin(), S.order.end(), [&](int a, int b) { return first[a] < first[b]; });
  for (int k = 0; k < s; ++k) S.start[k] = first[S.order[k]];
  for (int r = s - 1; r >= 0; --r) {
    int c = 0;
    while (c < s && H[(size_t)r * f + c] == 0.0) ++c;
    S.reach[r] = std::min(S.reach[r + 1], c);
  }
  return S;
}

void NodeSpans::columns(bool fwd, int s, int m, int r0, int r1, int& k0, int& K) const {
  k0 = 0;
  K = fwd ? s : s + m;
  if (fwd && r1 <= s) K = (int)(std::lower_bound(start.begin(), start.end(), r1) - start.begin());
  if (!fwd) k0 = std::min(reach[r0], K - 1), K -= k0;
  K = std::max(K, 1);
}

RowRec make_rec(int src, const std::vector<int>& l, std::vector<int>& more) {
  RowRec r;
  r.src = src;
  const int n = (int)l.size(), k = n <= kRowsSlots ? n : kRowsSlots - 1;
  for (int i = 0; i < kRowsSlots; ++i) r.slot[i] = i < k ? l[i] : -1;
  if (n > k) {
    r.slot[kRowsSlots - 1] = -2 - (int)more.size();
    more.push_back(n - k);
    more.insert(more.end(), l.begin() + k, l.end());
  }
  return r;
}

RowsSmem rows_smem(const RowShape& P, int vr, int rb, int ts) {
  const size_t kColBytes = 32 * 1024;  // staged source values; longer rows in chunks
  const unsigned col = 16u / vr * rb;  // bytes of a column's source values
  // a team's partial sums: at most ts x vector x right-hand sides per thread, and the strides' slack
  const int rt = rb <= 4 ? rb : (rb == 6 ? 3 : 4);
  const unsigned sums = (unsigned)ts * 16 * rt + 144u * rb;
  auto layout = [&](int kc) {
    RowsSmem m;
    m.kc = kc;
    m.buf = (unsigned)P.vals * (16u / vr);
    const bool two = P.chunks > 1 || P.cols > kc;
    m.ds = 16 + (two ? 2 : 1) * m.buf;
    m.cu = (m.ds + std::max(kc * col, sums) + 15) & ~15u;
    m.team_bytes = (m.cu + (unsigned)P.npt * rb * 8 + 15) & ~15u;
    return m;
  };
  RowsSmem m = layout(std::max(1, std::min(P.cols, (int)(kColBytes / col))));
  // A team's size follows its level's average node, the layout its widest tile: eight
  // teams with 32 KB of columns each are more than a multiprocessor has.  They stage
  // fewer columns at a time.  The values (at most 10 vectors per thread and buffer), sums
  // and pass-through rows leave room for 13 KB of columns in a team of 32.
  const size_t most = (kRowsSmem / (kRowsThreads / ts)) & ~(size_t)15;
  if (m.team_bytes > most) {
    const size_t rest = 16 + 2 * (size_t)m.buf + (size_t)P.npt * rb * 8 + 32;
    m = layout((int)std::max<size_t>(1, rest < most ? (most - rest) / col : 1));
  }
  return m;
}

namespace {

// A batch applies small leaves thread by output; its columns are read once per
// output, so only FP64 values (no conversions) and short rows.
constexpr int kBatchArea = 1280, kBatchCols = 64, kBatchRows = 256;

template <typename T>
void pack(const RowsPlan& P, const std::vector<const MfFactor*>& factors, int d, T* out) {
  const RowsPlan::Dir& D = P.dir[d];
  std::vector<char> batch(D.items.size(), 0);
  for (const RowLevel& L : D.levels)
    for (int i = 0; i < L.n_batch; ++i) batch[L.first + L.n_tile + i] = 1;
  dense::parallel_for((int)D.items.size(), 64, [&](int i) {
    const RowItem& it = D.items[i];
    T* p = out + it.off;
    // a batch's nodes follow one another in the source list
    const int n = batch[i] ? it.pad : 1, pad = batch[i] ? it.rows : it.pad;
    for (int q = 0; q < n; ++q) {
      int g = it.node;
      if (q) g = D.at[D.pos[g] + q];
      const RowsPlan::Node& x = P.nodes[g];
      const int ld = d == 0 ? x.s : x.s + x.m;
      const double* A = (d == 0 ? factors[x.set]->Gf[x.j] : factors[x.set]->Hb[x.j]).data() + (size_t)it.row0 * ld;
      const int k0 = batch[i] ? 0 : it.src - D.src0[g];
      for (int k = 0; k < it.cols; ++k, p += pad) {
        const int c = d == 0 ? P.spans[g].order[k0 + k] : k0 + k;
        for (int r = 0; r < it.rows; ++r) p[r] = (T)A[(size_t)r * ld + c];
        for (int r = it.rows; r < pad; ++r) p[r] = T(0);
      }
    }
  });
}

}  // namespace

RowsPlan plan_rows(const std::vector<const MfFactor*>& factors, int vr, int max_nrhs) {
  RowsPlan R;
  // Tile sizes, in 16-byte vectors of values per thread: as many as spread the
  // level over kCtasPerSm CTAs of every SM, within these bounds.  Fewer make the
  // fixed part of a tile (gathering its columns, adding its partial sums: 2 to 3 us)
  // weigh more, more leave a level's last wave nearly empty.  More right-hand sides
  // do more per value, so their tiles stay smaller, but have at least a few rows per
  // right-hand side: every tile of a node gathers the node's columns again, and for
  // FP32 factors also adds up more partial sums.  Measured on the half cells of
  // 64x64+64x64 cells (us per carrier / Poisson sweep): FP64, k = 1, 2 / 1 right-hand
  // sides: 279 / 118 for one CTA per SM, 223 / 115 for three, 235 / 115 for four;
  // FP32, k = 2, 16 / 8: 451 / 223 for 5 vectors at most, 502 / 226 for 9; FP64, 24 /
  // 12 on 29x37+23x37 cells: 829 / 405 with 0.3 rows, 1005 / 459 with one.
  const bool many = max_nrhs > 4;
  const double most_vecs = many ? 5 : 32, least_vecs = 2, ctas_per_sm = 3, rows_per_rhs = vr == 2 ? 0.3 : 1.0;
  // a chunk of more than four right-hand sides is shared by threads of the same rows
  // (rows.cu: four each; FP64 chunks hold up to 8, FP32 up to 16), and needs fewer
  // values staged at a time
  const int rhs_threads = max_nrhs > 0 && !many ? 1 : (vr == 2 ? 2 : 4);
  // Values staged at a time.  A large level's tiles (more than kLargeVecs vectors per
  // thread) go through two small buffers, so that three CTAs share a multiprocessor
  // and each reads its node's columns for more values; smaller tiles are staged
  // whole.  72x72+72x72 cells, k = 2, RT_2 Poisson elements, FP32, 3 right-hand sides,
  // us per Poisson sweep: 876 for 16 vectors at most and 10 staged, 649 for 32 / 10,
  // 598 for 32 / 5, 609 for 64 / 4; 56x56+56x56, FP64, 1: 810, 736, 688; but 64x64+64x64,
  // k = 1, FP64, 2, with tiles below that: 223 for 10 staged, 228 for 5.
  const double kLargeVecs = 16;
  const int stage_vecs_small = many ? 8 : 10, stage_vecs_large = many ? 8 : 5;
  std::vector<RowsPlan::Node>& nodes = R.nodes;
  int nl[2] = {0, 0};
  for (int fi = 0; fi < (int)factors.size(); ++fi) {
    const MfFactor& F = *factors[fi];
    if (F.Gf.size() != F.nodes.size()) throw std::runtime_error("factor not factorised");
    const int base = (int)nodes.size();
    int w = 0;
    for (int j = 0; j < (int)F.nodes.size(); ++j) {
      const MfNode& x = F.nodes[j];
      nodes.push_back(RowsPlan::Node{fi, j, x.s, x.m, {x.height, x.depth}, -1, w, x.children.empty()});
      w += x.m;
      nl[0] = std::max(nl[0], x.height + 1);
      nl[1] = std::max(nl[1], x.depth + 1);
      R.entries += (long long)(F.Gf[j].size() + F.Hb[j].size());
    }
    for (int j = 0; j < (int)F.nodes.size(); ++j)
      for (int c : F.nodes[j].children) nodes[base + c].parent = base + j;
    R.wtotal.push_back(std::max(1, w));
  }
  // small leaves have nothing behind them in the backward sweep: all of them
  // in its last level, as batches of equal shape
  auto is_batch = [&](int g, int d) {
    const RowsPlan::Node& x = nodes[g];
    return vr == 2 && x.leaf && x.s * (x.s + x.m) <= kBatchArea && (d == 0 || x.s + x.m <= kBatchCols);
  };
  for (int g = 0; g < (int)nodes.size(); ++g)
    if (is_batch(g, 1)) nodes[g].level[1] = nl[1] - 1;
  const int N = (int)nodes.size();
  R.spans.resize(N);
  dense::parallel_for(N, 64, [&](int g) { R.spans[g] = node_spans(*factors[nodes[g].set], nodes[g].j); });
  // nodes in level order (tiles, then batches by shape), and the lists
  std::vector<std::vector<int>> lv[2];
  for (int d = 0; d < 2; ++d) {
    RowsPlan::Dir& D = R.dir[d];
    lv[d].resize(nl[d]);
    for (int g = 0; g < N; ++g) lv[d][nodes[g].level[d]].push_back(g);
    D.src0.resize(N), D.dst0.resize(N), D.pos.resize(N);
    for (auto& l : lv[d]) {
      std::stable_sort(l.begin(), l.end(), [&](int a, int b) {
        const bool ba = is_batch(a, d), bb = is_batch(b, d);
        if (ba != bb) return bb;
        if (!ba) return false;
        const RowsPlan::Node &x = nodes[a], &y = nodes[b];
        return x.set != y.set ? x.set < y.set : x.s != y.s ? x.s < y.s : x.m < y.m;
      });
      for (int g : l) {
        const RowsPlan::Node& x = nodes[g];
        const MfNode& nd = factors[x.set]->nodes[x.j];
        D.pos[g] = (int)D.at.size();
        D.at.push_back(g);
        D.src0[g] = (int)D.src.size();
        for (int t = 0; t < x.s; ++t) D.src.push_back(nd.own[d == 0 ? R.spans[g].order[t] : t]);
        if (d == 1)
          for (int t = 0; t < x.m; ++t) D.src.push_back(~nd.upd[t]);
        D.dst0[g] = (int)D.dst.size();
        D.dst.insert(D.dst.end(), nd.own.begin(), nd.own.end());
        if (d == 0)
          for (int t = 0; t < x.m; ++t) D.dst.push_back(x.w_off + t);
      }
    }
  }
  // records: the children's update slots that land on each front position
  std::vector<int> upd0(N);
  {
    int n_upd = 0;
    for (int g : R.dir[0].at) upd0[g] = n_upd, n_upd += nodes[g].m;
    R.rec.resize(R.dir[0].src.size());
    R.upd.resize(n_upd);
    int base = 0;
    std::vector<int> fpos;
    std::vector<std::vector<int>> lists;
    for (const MfFactor* Fp : factors) {
      const MfFactor& F = *Fp;
      fpos.assign(F.n, -1);
      for (int j = 0; j < (int)F.nodes.size(); ++j) {
        const int g = base + j;
        const MfNode& x = F.nodes[j];
        for (int t = 0; t < x.s; ++t) fpos[x.own[R.spans[g].order[t]]] = t;
        for (int t = 0; t < x.m; ++t) fpos[x.upd[t]] = x.s + t;
        lists.assign(x.s + x.m, {});
        for (int c : x.children)
          for (int a = 0; a < F.nodes[c].m; ++a) {
            const int p = fpos[F.nodes[c].upd[a]];
            if (p < 0) throw std::runtime_error("extend-add map mismatch");
            lists[p].push_back(nodes[base + c].w_off + a);
          }
        for (int t = 0; t < x.s; ++t) fpos[x.own[t]] = -1;
        for (int t = 0; t < x.m; ++t) fpos[x.upd[t]] = -1;
        for (int p = 0; p < x.s + x.m; ++p) {
          RowRec& r = p < x.s ? R.rec[R.dir[0].src0[g] + p] : R.upd[upd0[g] + p - x.s];
          r = make_rec(p < x.s ? x.own[R.spans[g].order[p]] : nodes[g].w_off + p - x.s, lists[p], R.more);
        }
      }
      base += (int)F.nodes.size();
    }
  }
  for (int d = 0; d < 2; ++d) {
    const bool fwd = d == 0;
    RowsPlan::Dir& D = R.dir[d];
    D.levels.assign(nl[d], RowLevel());
    std::vector<int> nsig(N, 0), kid_sig(N, 0);
    auto rows_of = [&](int g) { return fwd ? nodes[g].s + nodes[g].m : nodes[g].s; };
    auto cols_of = [&](int g) { return fwd ? nodes[g].s : nodes[g].s + nodes[g].m; };
    int placed[kRowsMaxSets] = {};
    std::vector<int> d0(N, 0);
    for (int l = 0; l < nl[d]; ++l) {
      RowLevel& L = D.levels[l];
      L.first = (int)D.items.size();
      double area = 0;
      int n = 0;
      for (int g : lv[d][l]) {
        if (!is_batch(g, d)) area += (double)rows_of(g) * cols_of(g), ++n;
      }
      L.n_node = n;
      if (fwd)
        for (int g : lv[d][l]) {  // tile nodes come set by set
          const int q = nodes[g].set;
          if (is_batch(g, d)) continue;
          if (L.n_col[q] == 0) L.col[q] = D.src0[g], L.upd[q] = upd0[g], L.d[q] = placed[q];
          d0[g] = placed[q];
          placed[q] += nodes[g].s;
          L.n_col[q] += nodes[g].s;
          L.n_upd[q] += nodes[g].m;
        }
      // values per thread: enough threads to fill the GPU, then more values
      const double per_thread =
          std::min(most_vecs, std::max(least_vecs, area / vr / ((double)kRowsSms * kRowsThreads * ctas_per_sm)));
      const double rhs_weight = std::max(1.0, 0.1 * max_nrhs);
      const int stage_vecs = per_thread > kLargeVecs ? stage_vecs_large : stage_vecs_small;
      // team: the level's average node in one tile where the level has nodes enough
      int ts = 32;
      while (ts < kRowsThreads && area / std::max(1, n) * rhs_weight > per_thread * vr * ts * 1.5) ts *= 2;
      L.ts = ts;
      const int most_rows = ts * vr / rhs_threads;
      RowShape& F = D.flow_shape[ts == 32 ? 0 : ts == 64 ? 1 : ts == 128 ? 2 : 3];
      for (int g : lv[d][l]) {
        if (is_batch(g, d)) continue;
        const RowsPlan::Node& x = nodes[g];
        const int rows = rows_of(g);
        L.leaf = L.leaf && x.leaf;
        // columns [k0, k0 + K) of rows [r0, r1)
        auto span = [&](int r0, int r1, int& k0) {
          int K = 0;
          R.spans[g].columns(fwd, x.s, x.m, r0, r1, k0, K);
          return K;
        };
        // tiles of about `want` values, the rows of a triangular part in unequal
        // ones; forward, none across the end of the own rows unless the whole node
        // is one tile
        const double want = std::max(per_thread * vr * ts, rows_per_rhs * max_nrhs * cols_of(g));
        const int whole = (int)std::min<double>(want / cols_of(g), most_rows);
        const int nseg = fwd && x.m > 0 && rows > whole ? 2 : 1;
        for (int sg = 0; sg < nseg; ++sg) {
          const int a = sg ? x.s : 0, b = nseg == 2 && sg == 0 ? x.s : rows;
          double area = 0;
          int k0 = 0;
          for (int r = a; r < b; r += vr) area += (double)std::min(vr, b - r) * span(r, std::min(b, r + vr), k0);
          const double each = area / std::max(1.0, std::ceil(area / want - 0.25));
          for (int r0 = a, r1; r0 < b; r0 = r1) {
            int K = 0;
            for (r1 = r0; r1 < b && r1 - r0 < most_rows;) {
              const int e = std::min(b, r1 + vr);
              const int c = span(r0, e, k0);
              if (r1 > r0 && (double)(e - r0) * c > 1.05 * each) break;
              r1 = e;
            }
            K = span(r0, r1, k0);
            RowItem it{};
            it.rows = r1 - r0;
            it.pad = (r1 - r0 + vr - 1) / vr * vr;
            it.cols = K;
            it.set = x.set;
            it.src = D.src0[g] + k0;
            it.dst = D.dst0[g] + r0;
            if (fwd) {
              it.npt = std::max(0, r1 - std::max(r0, x.s));
              it.pt = upd0[g] + std::max(r0, x.s) - x.s;
              it.d = d0[g];
              it.leaf = x.leaf;
            }
            it.off = D.n_values;
            const int rg = it.pad / vr;
            it.magic = (65536 + rg - 1) / rg;
            it.node = g;
            it.row0 = r0;
            it.kc = std::min(K, std::max(1, stage_vecs * ts / rg));
            for (RowShape* P : {&L.shape, &F}) {
              P->cols = std::max(P->cols, K);
              P->npt = std::max(P->npt, it.leaf ? 0 : it.npt);
              P->vals = std::max(P->vals, it.kc * it.pad);
              P->chunks = std::max(P->chunks, (K + it.kc - 1) / it.kc);
            }
            ++L.n_tile;
            ++nsig[g];
            D.n_values += ((long long)K * it.pad + 3) & ~3ll;
            D.items.push_back(it);
          }
        }
      }
      // batches: nodes of equal shape, up to kBatchOutputs rows
      const std::vector<int>& q = lv[d][l];
      for (size_t i = 0; i < q.size();) {
        if (!is_batch(q[i], d)) {
          ++i;
          continue;
        }
        const RowsPlan::Node& x = nodes[q[i]];
        const int rows = rows_of(q[i]), most = std::max(1, kBatchRows / rows);
        size_t e = i;
        while (e < q.size() && (int)(e - i) < most && nodes[q[e]].set == x.set && nodes[q[e]].s == x.s &&
               nodes[q[e]].m == x.m && is_batch(q[e], d)) {
          nsig[q[e]] = 1;
          ++e;
        }
        RowItem it{};
        it.rows = rows;
        it.pad = (int)(e - i);
        it.cols = cols_of(q[i]);
        it.set = x.set;
        it.src = D.src0[q[i]];
        it.dst = D.dst0[q[i]];
        it.npt = fwd ? x.m : 0;
        it.off = D.n_values;
        it.node = q[i];
        ++L.n_batch;
        D.n_values += ((long long)it.pad * rows * it.cols + 3) & ~3ll;
        D.items.push_back(it);
        i = e;
      }
    }
    for (int g = 0; g < N; ++g)
      if (nodes[g].parent >= 0) kid_sig[nodes[g].parent] += nsig[g];
    // flow waits: forward for every item of the children, backward for every
    // item of the parent
    auto sync = [&](int g) {
      const int p = nodes[g].parent;
      return fwd ? RowSync{kid_sig[g] > 0 ? g : -1, kid_sig[g], p, 0} : RowSync{p, p >= 0 ? nsig[p] : 0, g, 0};
    };
    for (const RowLevel& L : D.levels) {
      const int teams = kRowsThreads / L.ts;
      for (int i = 0; i < L.n_tile; i += teams) {
        const int n = std::min(teams, L.n_tile - i);
        D.entries.push_back(RowEntry{L.ts, L.first + i, n, (int)D.sync.size()});
        for (int q = 0; q < n; ++q) D.sync.push_back(sync(D.items[L.first + i + q].node));
      }
      for (int i = 0; i < L.n_batch; ++i) {
        const RowItem& it = D.items[L.first + L.n_tile + i];
        D.entries.push_back(RowEntry{0, L.first + L.n_tile + i, it.pad, (int)D.sync.size()});
        for (int q = 0; q < it.pad; ++q) D.sync.push_back(sync(D.at[D.pos[it.node] + q]));
      }
    }
  }
  return R;
}

void pack_rows(const RowsPlan& P, const std::vector<const MfFactor*>& factors, int d, double* out) {
  pack(P, factors, d, out);
}
void pack_rows(const RowsPlan& P, const std::vector<const MfFactor*>& factors, int d, float* out) {
  pack(P, factors, d, out);
}

}  // namespace pecs
