// Executes the tile plans of FP64 panel banks (pecs_gb300/csrc/panel_plan.cpp, tiles of
// kPanelRowsF64 rows) on the host; compiled and run by test_panel_rows_host.py.
// Every index goes through the plan's own offsets with bounds checked, every value
// is read once, every row written once, and the copies' sizes and places are whole
// 16-byte pieces.  The result must be that of the plain application of the factors.
#include <cmath>
#include <cstdio>
#include <limits>

#include "panel_plan.hpp"

namespace pecs {
void set_error_external(const std::string&) {}  // the library's error hook (engine.cu)
}  // namespace pecs

using namespace pecs;

#define CHECK(c) \
  if (!(c)) return std::printf("FAIL %s\n", #c), 1

// a five-point grid of nx x ny cells of k unknowns, diagonally dominant
static MfFactor grid(int nx, int ny, int k) {
  std::vector<int> r, c, cell;
  std::vector<double> v, xy;
  auto couple = [&](int p, int q) {
    for (int i = p * k; i < p * k + k; ++i)
      for (int j = q * k; j < q * k + k; ++j)
        r.push_back(i), c.push_back(j), v.push_back(i == j ? 6.0 * k : 0.3 + 0.1 * (i % 7 - j % 5));
  };
  for (int q = 0; q < nx * ny; ++q) {
    const int x = q % nx, y = q / nx;
    cell.insert(cell.end(), k, q);
    xy.push_back(x + 0.5), xy.push_back(y + 0.5);
    couple(q, q);
    if (x > 0) couple(q, q - 1);
    if (x + 1 < nx) couple(q, q + 1);
    if (y > 0) couple(q, q - nx);
    if (y + 1 < ny) couple(q, q + nx);
  }
  const Csr A = coo_to_csr(nx * ny * k, r, c, v);
  MfFactor F = mf_analyze(A, cell.data(), nullptr, nx * ny, xy.data(), 8);
  mf_factorize(F, A);
  return F;
}

static int check(const MfFactor& F) {
  const PanelTilesPlan P = plan_panel({&F}, 2, 152, kPanelRowsF64);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  int wt = 1;
  for (const MfNode& nd : F.nodes) wt += nd.m;
  std::vector<double> b(F.n), y(F.n, nan), w(wt, nan), x(F.n, nan), ref(F.n);
  for (int i = 0; i < F.n; ++i) b[i] = std::sin(1.0 + 0.7 * i);
  mf_apply_host(F, b.data(), ref.data());
  for (int d = 0; d < 2; ++d) {
    const PanelTilesPlan::Dir& D = P.dir[d];
    std::vector<double> val(D.n_values, nan);
    pack_panel(P, {&F}, d, val.data());
    std::vector<char> used(D.n_values, 0);
    if (d == 1) x.assign(F.n, nan);  // forward left the assembled columns there
    for (const PanelLevel& L : D.levels) {
      for (int i = L.rec[0]; i < L.rec[0] + L.n_rec[0]; ++i) {
        const RowRec& q = P.rec.at(i);
        double t = 0.0;
        for (int s : q.slot) {
          if (s >= 0) t += w.at(s);
          if (s < -1)
            for (int k = 1; k <= P.more.at(-2 - s); ++k) t += w.at(P.more.at(-2 - s + k));
        }
        (q.src >= 0 ? x.at(q.src) : w.at(~q.src)) = q.src >= 0 ? b[q.src] - t : t;
      }
      for (int i = L.first; i < L.first + L.n; ++i) {
        const PanelTile& it = D.tiles.at(i);
        const int K4 = (it.cols + 3) & ~3;
        CHECK(it.pad == kPanelRowsF64 && it.pad == L.pad && it.rows >= 1 && it.rows <= it.pad);
        CHECK(it.cols >= 1 && it.cols <= L.cols && it.off % 2 == 0 && it.idx % 4 == 0);
        CHECK(it.off + (long long)it.cols * it.pad <= D.n_values && it.idx + K4 + it.pad <= (int)D.idx.size());
        double sum[kPanelRowsF64] = {};
        for (int k = 0; k < it.cols; ++k) {
          const int z = D.idx[it.idx + k];
          const double v = d == 0 ? (it.leaf ? b.at(z) : x.at(z)) : (z >= 0 ? y.at(z) : x.at(~z));
          CHECK(std::isfinite(v));
          for (int r = 0; r < it.pad; ++r) {
            const long long e = it.off + (long long)k * it.pad + r;
            CHECK(!used[e] && (r < it.rows ? std::isfinite(val[e]) : val[e] == 0.0));
            used[e] = 1;
            sum[r] += val[e] * v;
          }
        }
        for (int r = 0; r < it.rows; ++r) {
          const int z = D.idx[it.idx + K4 + r];
          const bool pass = r >= it.rows - it.npt;
          double& out = d == 1 ? x.at(z) : (z >= 0 ? y.at(z) : w.at(~z));
          CHECK(pass ? z < 0 && L.passes && std::isfinite(out) : std::isnan(out));
          out = pass ? out + sum[r] : sum[r];
        }
      }
    }
    for (char c : used) CHECK(c);
  }
  double e2 = 0.0, n2 = 0.0;
  for (int i = 0; i < F.n; ++i) e2 += (x[i] - ref[i]) * (x[i] - ref[i]), n2 += ref[i] * ref[i];
  std::printf("%d unknowns: %zu + %zu tiles, error %.1e\n", F.n, P.dir[0].tiles.size(), P.dir[1].tiles.size(),
              std::sqrt(e2 / n2));
  CHECK(std::sqrt(e2 / n2) < 1e-11);  // the same sums in another order, well conditioned
  return 0;
}

int main() {
  const int sizes[][3] = {{1, 1, 1}, {1, 1, 5}, {3, 1, 1}, {7, 5, 3}, {13, 9, 4}, {21, 20, 5}};
  for (auto& s : sizes)
    if (check(grid(s[0], s[1], s[2]))) return 1;
  std::printf("OK\n");
  return 0;
}
