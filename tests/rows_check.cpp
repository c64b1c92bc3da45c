// Checks the tile plans of the few-right-hand-side sweeps
// (pecs_gb300/csrc/rows_plan.cpp) on the host; compiled and run by
// test_rows_host.py.  Each plan is executed item by item as the kernel reads
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
#include "rows_plan.hpp"

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

static int check(const std::vector<const MfFactor*>& F, int vr, int nrhs, const char* name) {
  const RowsPlan P = plan_rows(F, vr, nrhs);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  const int ns = (int)F.size();
  std::vector<std::vector<double>> b(ns), y(ns), w(ns), x(ns), ref(ns);
  for (int q = 0; q < ns; ++q) {
    const int n = F[q]->n;
    b[q].resize(n);
    for (int i = 0; i < n; ++i) b[q][i] = std::sin(1.0 + 0.7 * i + q);
    y[q].assign(n, nan), x[q].assign(n, nan), ref[q].resize(n), w[q].assign(P.wtotal[q], nan);
    mf_apply_host(*F[q], b[q].data(), ref[q].data());
  }
  long long kept = 0;
  // forward sources: update slots of a record, the overflow list included
  auto children = [&](const RowRec& r, const std::vector<double>& wq) {
    double t = 0.0;
    for (int j = 0; j < kRowsSlots; ++j) {
      if (r.slot[j] >= 0) t += wq.at(r.slot[j]);
      if (r.slot[j] < -1) {
        const int* m = &P.more.at(-2 - r.slot[j]);
        for (int i = 1; i <= m[0]; ++i) t += wq.at(m[i]);
      }
    }
    return t;
  };
  for (int d = 0; d < 2; ++d) {
    const RowsPlan::Dir& D = P.dir[d];
    std::vector<double> val(D.n_values, nan);
    pack_rows(P, F, d, val.data());
    std::vector<char> used(D.n_values, 0);
    size_t n_items = 0;
    std::vector<int> sig(P.nodes.size(), 0), place(ns, 0);
    for (const RowLevel& L : D.levels) {
      CHECK(L.first == (int)n_items);
      n_items += L.n_tile + L.n_batch;
      CHECK(L.ts == 32 || L.ts == 64 || L.ts == 128 || L.ts == 256);
      // assembled columns: every tile column has the place k_assemble gives it
      std::vector<std::vector<double>> asm_d(ns);
      if (d == 0)
        for (int q = 0; q < ns; ++q) {
          CHECK(L.n_col[q] == 0 || L.d[q] == place[q]);
          for (int k = 0; k < L.n_col[q]; ++k) {
            const RowRec& r = P.rec.at(L.col[q] + k);
            asm_d[q].push_back(b[q].at(r.src) - children(r, w[q]));
          }
          for (int k = 0; k < L.n_upd[q]; ++k) CHECK(P.upd.at(L.upd[q] + k).src < P.wtotal[q]);
          place[q] += L.n_col[q];
          CHECK(place[q] <= F[q]->n);
        }
      for (int i = L.first; i < L.first + L.n_tile + L.n_batch; ++i) {
        const RowItem& it = D.items[i];
        const bool batch = i >= L.first + L.n_tile;
        const RowShape& Sf = D.flow_shape[L.ts == 32 ? 0 : L.ts == 64 ? 1 : L.ts == 128 ? 2 : 3];
        const int nodes = batch ? it.pad : 1, pad = batch ? it.rows : it.pad;
        CHECK(it.off % 4 == 0 && it.cols >= 1 && it.rows >= 1);
        CHECK(it.off + (long long)it.cols * pad * nodes <= D.n_values);
        if (!batch) {
          const int rg = it.pad / vr, share = nrhs > 0 && nrhs <= 4 ? 1 : (vr == 2 ? 2 : 4);
          CHECK(it.pad % vr == 0 && it.rows <= it.pad && it.pad < it.rows + vr && rg * share <= L.ts);
          for (int t = 0; t <= L.ts; ++t) CHECK(((t * it.magic) >> 16) == t / rg);
          CHECK(it.kc >= 1 && it.kc <= it.cols && it.kc * rg <= 12 * L.ts);
          for (const RowShape* Z : {&L.shape, &Sf})
            CHECK(it.cols <= Z->cols && (it.leaf || it.npt <= Z->npt) && it.kc * it.pad <= Z->vals &&
                  (it.cols + it.kc - 1) / it.kc <= Z->chunks);
        } else {
          CHECK(vr == 2 && it.row0 == 0 && it.pad >= 1 && it.pad <= kRowsThreads);
        }
        std::vector<double>&bq = b[it.set], &yq = y[it.set], &wq = w[it.set], &xq = x[it.set];
        CHECK(it.npt >= 0 && it.npt <= it.rows && (d == 0 || it.npt == 0));
        for (int q = 0; q < nodes; ++q) {
          std::vector<double> v(it.cols), sum(it.rows, 0.0), cu(it.rows, 0.0);
          const int src = it.src + q * it.cols, dst = it.dst + q * it.rows;
          CHECK(src >= 0 && src + it.cols <= (int)D.src.size() && dst + it.rows <= (int)D.dst.size());
          for (int k = 0; k < it.cols; ++k) {
            const int s_ = D.src[src + k];
            if (d == 0) {
              v[k] = bq.at(s_);
              const RowRec& r = P.rec.at(src + k);
              CHECK(r.src == s_ && (!batch || r.slot[0] == -1));
              v[k] -= children(r, wq);
              if (!batch) CHECK(asm_d[it.set].at(it.d - L.d[it.set] + k) == v[k]);
            } else {
              v[k] = s_ >= 0 ? yq.at(s_) : xq.at(~s_);
            }
            CHECK(std::isfinite(v[k]));
          }
          for (int j = 0; j < it.npt && !batch; ++j) {
            const RowRec& r = P.upd.at(it.pt + j);
            CHECK(r.src == D.dst[dst + it.rows - it.npt + j]);
            CHECK(it.pt + j >= L.upd[it.set] && it.pt + j < L.upd[it.set] + L.n_upd[it.set]);
            cu[it.rows - it.npt + j] = children(r, wq);
            CHECK(!it.leaf || (r.slot[0] == -1 && r.slot[kRowsSlots - 1] == -1));
          }
          for (int k = 0; k < it.cols; ++k)
            for (int r = 0; r < pad; ++r) {
              const long long e = it.off + ((long long)q * it.cols + k) * pad + r;
              CHECK(!used[e] && std::isfinite(val[e]) && (r < it.rows || val[e] == 0.0));
              used[e] = 1;
              if (r < it.rows) sum[r] += val[e] * v[k];
            }
          kept += (long long)it.cols * pad;
          for (int r = 0; r < it.rows; ++r) {
            const int t = D.dst[dst + r];
            double& out = d == 1 ? xq.at(t) : (r < it.rows - it.npt ? yq.at(t) : wq.at(t));
            CHECK(std::isnan(out));
            out = sum[r] + cu[r];
          }
        }
      }
    }
    CHECK(n_items == D.items.size());
    // flow entries in ticket order: every item once, its waits met by earlier entries alone
    std::vector<char> seen(n_items, 0);
    size_t n_sync = 0;
    for (const RowEntry& e : D.entries) {
      CHECK(e.sync == (int)n_sync && e.count >= 1 && e.count * std::max(1, e.ts) <= kRowsThreads);
      n_sync += e.count;
      for (int i = e.first; i < e.first + (e.ts > 0 ? e.count : 1); ++i) {
        CHECK(!seen[i]);
        seen[i] = 1;
      }
      for (int k = 0; k < e.count; ++k) {
        const RowItem& it = D.items[e.first + (e.ts > 0 ? k : 0)];
        const int g = e.ts > 0 ? it.node : D.at.at(D.pos[it.node] + k);
        const RowSync& sy = D.sync.at(e.sync + k);
        CHECK(sy.wait < 0 || sig[sy.wait] == sy.target);
        CHECK(sy.wait == (d == 1 ? P.nodes[g].parent : (P.nodes[g].leaf ? -1 : g)));
        CHECK(sy.signal == (d == 1 ? g : P.nodes[g].parent));
      }
      for (int k = 0; k < e.count; ++k)
        if (D.sync[e.sync + k].signal >= 0) ++sig[D.sync[e.sync + k].signal];
    }
    for (char c : seen) CHECK(c);
  }
  double worst = 0.0;
  for (int q = 0; q < ns; ++q) {
    double e2 = 0.0, n2 = 0.0;
    for (size_t i = 0; i < x[q].size(); ++i) {
      CHECK(std::isfinite(x[q][i]));
      e2 += (x[q][i] - ref[q][i]) * (x[q][i] - ref[q][i]);
      n2 += ref[q][i] * ref[q][i];
    }
    worst = std::max(worst, std::sqrt(e2 / n2));
  }
  std::printf("%s vr %d nrhs %d: items %zu + %zu, %.3f of the stored values kept, error %.1e\n", name, vr, nrhs,
              P.dir[0].items.size(), P.dir[1].items.size(), (double)kept / (double)P.entries, worst);
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
    for (int vr : {2, 4})
      for (int nrhs : {0, 1, 2, 7, 24})
        if (check({&fs, &fe}, vr, nrhs, "carriers") || check({&fp}, vr, nrhs, "poisson")) return 1;
  }
  std::printf("OK\n");
  return 0;
}
