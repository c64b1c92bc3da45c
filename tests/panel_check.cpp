// Checks the tile plans of the panel banks' level sweeps
// (pecs_gb300/csrc/panel_plan.cpp) on the host; compiled and run by
// test_panel_host.py.  Each plan is executed item by item as the kernel reads
// it: every source, destination, child list and value is taken through the
// plan's own offsets (bounds checked), every row must be written once and every
// value read before it was written is an error.  The result must be that of the
// plain application of the factors.  Prints one line per plan.
#include <cmath>
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <limits>
#include <string>

#include "problem.hpp"
#include "panel_plan.hpp"

namespace pecs {
void set_error_external(const std::string&) {}  // the library's error hook (engine.cu)
}  // namespace pecs

using namespace pecs;

static int fail(const char* what) {
  std::printf("FAIL %s\n", what);
  return 1;
}

#define CHECK(c) \
  if (!(c)) return fail(#c)

static pecs_params half_cell(int nx, int nxe, int ny, int degree, int pairing, double grading) {
  pecs_params p;
  std::memset(&p, 0, sizeof(p));
  p.degree = degree;
  p.full_system = 1;
  p.nx_semi = nx, p.nx_elec = nxe, p.ny = ny;
  p.x_semi0 = 0.0, p.x_semi1 = 1.0, p.x_elec1 = 2.0, p.height = 1.0;
  const int semi[4] = {1, 0, 2, 2}, elec[4] = {0, 1, 2, 2}, pois[4] = {1, 1, 2, 2};
  for (int f = 0; f < 4; ++f) p.bc_semi[f] = semi[f], p.bc_elec[f] = elec[f], p.bc_poisson[f] = pois[f], p.mu[f] = 1.0;
  p.lambda2 = 1e-2, p.eps_semi = 1.0, p.eps_elec = 1.5, p.dt = 1e-3, p.penalty = 1.0;
  p.k_et = p.k_ht = 1e-2, p.junction_x = 0.5;
  p.nd[0] = p.nd[1] = p.n_eq[0] = p.n_eq[1] = 1.0;
  p.p_eq[0] = p.p_eq[1] = 1e-4, p.r_eq = p.o_eq = 1.0;
  p.tau_n = p.tau_p = 1.0, p.n_i = 1e-2;
  p.grading = grading, p.poisson_pairing = pairing;
  return p;
}

static int check(const std::vector<const MfFactor*>& F, int chunks, int min_ctas, const char* name) {
  const PanelTilesPlan P = plan_panel(F, chunks, min_ctas);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  const int ns = (int)F.size();
  std::vector<std::vector<double>> b(ns), y(ns), w(ns), x(ns), ref(ns);
  std::vector<std::vector<char>> done(ns);
  for (int q = 0; q < ns; ++q) {
    const int n = F[q]->n;
    int wt = 0;
    for (const MfNode& nd : F[q]->nodes) wt += nd.m;
    b[q].resize(n);
    for (int i = 0; i < n; ++i) b[q][i] = std::sin(1.0 + 0.7 * i + q);
    y[q].assign(n, nan), x[q].assign(n, nan), ref[q].resize(n), w[q].assign(wt, nan), done[q].assign(wt, 0);
    mf_apply_host(*F[q], b[q].data(), ref[q].data());
  }
  long long kept = 0, stored = 0;
  for (int d = 0; d < 2; ++d) {
    const PanelTilesPlan::Dir& D = P.dir[d];
    if (d == 1)  // forward left the assembled columns there
      for (auto& v : x) std::fill(v.begin(), v.end(), nan);
    std::vector<double> val(D.n_values, nan);
    pack_panel(P, F, d, val.data());
    std::vector<char> used(D.n_values, 0);
    int n_tiles = 0;
    for (const PanelLevel& L : D.levels) {
      CHECK(L.first == n_tiles);
      n_tiles += L.n;
      for (int q = 0; q < ns; ++q) {
        CHECK(d == 0 || L.n_rec[q] == 0);
        for (int i = L.rec[q]; i < L.rec[q] + L.n_rec[q]; ++i) {
          const RowRec& r = P.rec.at(i);
          double t = 0.0;
          for (int j = 0; j < kRowsSlots; ++j) {
            if (r.slot[j] >= 0) {
              CHECK(done[q].at(r.slot[j]));
              t += w[q][r.slot[j]];
            }
            if (r.slot[j] < -1) {
              const int* m = &P.more.at(-2 - r.slot[j]);
              for (int k = 1; k <= m[0]; ++k) {
                CHECK(done[q].at(m[k]));
                t += w[q][m[k]];
              }
            }
          }
          double& out = r.src >= 0 ? x[q].at(r.src) : w[q].at(~r.src);
          CHECK(std::isnan(out));
          out = r.src >= 0 ? b[q].at(r.src) - t : t;
        }
      }
      for (int i = L.first; i < L.first + L.n; ++i) {
        const PanelTile& it = D.tiles.at(i);
        const int q = it.set, K4 = (it.cols + 3) & ~3;
        CHECK(it.pad == 8 || it.pad == 16 || it.pad == 32);
        CHECK(it.rows >= 1 && it.rows <= it.pad && it.pad <= L.pad && it.cols >= 1 && it.cols <= L.cols);
        CHECK(it.off % 8 == 0 && it.idx % 4 == 0 && it.off + (long long)it.cols * it.pad <= D.n_values);
        CHECK(it.idx + K4 + it.pad <= (int)D.idx.size());
        CHECK(it.npt >= 0 && it.npt <= it.rows && (it.npt == 0 || (d == 0 && !it.leaf && L.passes)));
        std::vector<double> sum(it.rows, 0.0);
        for (int k = 0; k < it.cols; ++k) {
          const int z = D.idx[it.idx + k];
          double v;
          if (d == 0) {
            CHECK(z >= 0);
            v = it.leaf ? b[q].at(z) : x[q].at(z);
          } else {
            v = z >= 0 ? y[q].at(z) : x[q].at(~z);
          }
          CHECK(std::isfinite(v));
          for (int r = 0; r < it.pad; ++r) {
            const long long e = it.off + (long long)k * it.pad + r;
            CHECK(!used[e] && std::isfinite(val[e]) && (r < it.rows || val[e] == 0.0));
            used[e] = 1;
            if (r < it.rows) sum[r] += val[e] * v;
          }
        }
        kept += (long long)it.cols * it.pad;
        for (int r = 0; r < it.rows; ++r) {
          const int z = D.idx[it.idx + K4 + r];
          const bool pass = r >= it.rows - it.npt;
          CHECK(d == 0 ? (z < 0 || !pass) : z >= 0);
          double& out = d == 1 ? x[q].at(z) : (z >= 0 ? y[q].at(z) : w[q].at(~z));
          CHECK(pass ? std::isfinite(out) : std::isnan(out));
          out = pass ? out + sum[r] : sum[r];
          if (d == 0 && z < 0) {
            CHECK(!done[q].at(~z));
            done[q][~z] = 1;
          }
        }
      }
    }
    CHECK(n_tiles == (int)D.tiles.size());
    for (char c : used) CHECK(c);
  }
  double worst = 0.0;
  for (int q = 0; q < ns; ++q) {
    stored += F[q]->entries();
    double e2 = 0.0, n2 = 0.0;
    for (size_t i = 0; i < x[q].size(); ++i) {
      CHECK(std::isfinite(x[q][i]));
      e2 += (x[q][i] - ref[q][i]) * (x[q][i] - ref[q][i]);
      n2 += ref[q][i] * ref[q][i];
    }
    worst = std::max(worst, std::sqrt(e2 / n2));
  }
  std::printf("%s chunks %d: tiles %zu + %zu, %.3f of the stored values kept, error %.1e\n", name, chunks,
              P.dir[0].tiles.size(), P.dir[1].tiles.size(), (double)kept / (double)stored, worst);
  CHECK(worst < 1e-11);
  return 0;
}

int main() {
  struct Case {
    int nx, nxe, ny, degree, pairing;
    double grading;
  };
  for (const Case& c : {Case{8, 8, 8, 1, 0, 1.0}, Case{5, 9, 7, 1, 1, 3.0}, Case{6, 4, 5, 2, 0, 1.0},
                        Case{16, 12, 21, 1, 0, 1.0}, Case{9, 11, 10, 2, 1, 1.0}}) {
    Setup S({half_cell(c.nx, c.nxe, c.ny, c.degree, c.pairing, c.grading)});
    MfFactor fs = mf_analyze(S.semi.A[0], S.semi.dof_cell.data(), S.semi.dof_class.data(), S.semi.grid.nc(),
                             S.semi.cell_xy.data(), 8);
    MfFactor fe = mf_analyze(S.elec.A[0], S.elec.dof_cell.data(), nullptr, S.elec.grid.nc(), S.elec.cell_xy.data(), 8);
    MfFactor fp = mf_analyze(S.pois.A, S.pois.dof_cell.data(), nullptr, S.pois.grid.nc(), S.pois.cell_xy.data(), 8);
    mf_factorize(fs, S.semi.A[0]);
    mf_factorize(fe, S.elec.A[0]);
    mf_factorize(fp, S.pois.A);
    for (int chunks : {1, 4})
      for (int min_ctas : {1, 152})
        if (check({&fs, &fe}, chunks, min_ctas, "carriers") || check({&fp}, chunks, min_ctas, "poisson")) return 1;
  }
  std::printf("OK\n");
  return 0;
}
