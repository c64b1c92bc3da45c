// Checks the shared memory of every launch of the few-right-hand-side sweeps
// (rows_smem, pecs_gb300/csrc/rows_plan.cpp) on the host; compiled and run by
// test_rows_smem_host.py.  Systems with levels of short teams and long rows: class-0
// cells coupled to one dense cell, and grids with one cell of many unknowns.
#include <algorithm>
#include <cstdio>

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

static MfFactor factor(int n, const std::vector<int>& r, const std::vector<int>& c, const std::vector<double>& v,
                       const std::vector<int>& cell, const std::vector<int>& cls, const std::vector<double>& xy) {
  const Csr A = coo_to_csr(n, r, c, v);
  MfFactor F = mf_analyze(A, cell.data(), cls.data(), (int)xy.size() / 2, xy.data(), 8);
  mf_factorize(F, A);
  return F;
}

// `cells` class-0 cells of k unknowns, all of them coupled to every unknown of one dense
// cell of m
static MfFactor bordered(int cells, int k, int m) {
  const int n = cells * k + m;
  std::vector<int> r, c, cell(n, cells), cls(n, 1);
  std::vector<double> v, xy;
  auto put = [&](int i, int j, double a) { r.push_back(i), c.push_back(j), v.push_back(a); };
  for (int q = 0; q < cells; ++q) {
    for (int i = q * k; i < q * k + k; ++i) {
      cell[i] = q, cls[i] = 0;
      for (int j = q * k; j < q * k + k; ++j) put(i, j, i == j ? 4.0 * m : 0.1);
      for (int j = cells * k; j < n; ++j) put(i, j, 0.5), put(j, i, 0.25);
    }
    xy.push_back(q + 0.5), xy.push_back(0.5);
  }
  for (int i = cells * k; i < n; ++i)
    for (int j = cells * k; j < n; ++j) put(i, j, i == j ? 8.0 * n : 0.1);
  xy.push_back(cells + 0.5), xy.push_back(0.5);
  return factor(n, r, c, v, cell, cls, xy);
}

// a five-point grid of side x side cells of k unknowns, one of them of m
static MfFactor uneven(int side, int k, int m) {
  std::vector<int> first{0}, r, c, cell;
  std::vector<double> v, xy;
  const int cells = side * side, wide = side / 3 * side + side / 3;
  for (int q = 0; q < cells; ++q) {
    first.push_back(first[q] + (q == wide ? m : k));
    cell.insert(cell.end(), first[q + 1] - first[q], q);
    xy.push_back(q % side + 0.5), xy.push_back(q / side + 0.5);
  }
  auto couple = [&](int p, int q) {
    for (int i = first[p]; i < first[p + 1]; ++i)
      for (int j = first[q]; j < first[q + 1]; ++j) {
        r.push_back(i), c.push_back(j);
        v.push_back(i == j ? 8.0 * (m + 5 * k) : 0.3 + 0.01 * (i % 7 - j % 5));
      }
  };
  for (int q = 0; q < cells; ++q) {
    const int x = q % side, y = q / side;
    couple(q, q);
    if (x > 0) couple(q, q - 1);
    if (x + 1 < side) couple(q, q + 1);
    if (y > 0) couple(q, q - side);
    if (y + 1 < side) couple(q, q + side);
  }
  return factor(first.back(), r, c, v, cell, std::vector<int>(first.back(), 1), xy);
}

static int check(const MfFactor& F, int vr, int nrhs, int& narrowed) {
  const RowsPlan P = plan_rows({&F}, vr, nrhs);
  for (int rb : {1, 2, 3, 4, 6, 8, 12, 16}) {
    if (rb > 16 / (vr == 2 ? 2 : 1) || (nrhs > 0 && nrhs <= 4 && rb > 4)) continue;
    auto one = [&](const RowShape& S, int ts, int kc) {  // kc: of the tiles, at most
      const RowsSmem m = rows_smem(S, vr, rb, ts);
      const size_t esz = 16 / vr;
      CHECK((size_t)m.team_bytes * (kRowsThreads / ts) <= kRowsSmem);
      CHECK(m.kc >= 1 && m.team_bytes % 16 == 0 && m.buf % 16 == 0 && m.ds % 16 == 0 && m.cu % 16 == 0);
      CHECK(m.buf >= S.vals * esz);
      // a second buffer wherever a tile has more columns than are staged at a time
      CHECK(m.ds >= 16 + (std::min(kc, m.kc) < S.cols ? 2 : 1) * (size_t)m.buf);
      // source values, and the partial sums of up to ts / RG x vr x rb values over them
      const int rt = rb <= 4 ? rb : (rb == 6 ? 3 : 4);
      CHECK(m.cu >= m.ds + (size_t)m.kc * rb * esz && m.cu >= m.ds + (size_t)ts * 16 * rt + 136u * rb);
      CHECK(m.team_bytes >= m.cu + (size_t)S.npt * rb * 8);
      narrowed += m.kc < S.cols && (size_t)m.kc * rb * esz < 32 * 1024 - rb * esz;
      return 0;
    };
    for (int d = 0; d < 2; ++d) {
      const RowsPlan::Dir& D = P.dir[d];
      for (const RowLevel& L : D.levels) {
        int kc = 1 << 30;
        for (int i = 0; i < L.n_tile; ++i) kc = std::min(kc, D.items[L.first + i].kc < D.items[L.first + i].cols ? D.items[L.first + i].kc : kc);
        if (L.n_tile > 0 && one(L.shape, L.ts, kc)) return 1;
      }
      for (int q = 0; q < 4; ++q)
        if (D.flow_shape[q].cols > 0 && one(D.flow_shape[q], 32 << q, 1 << 30)) return 1;
    }
  }
  return 0;
}

static int check_all(const MfFactor& F, const char* name) {
  int narrowed = 0;
  for (int vr : {2, 4})
    for (int nrhs : {0, 1, 3, 4, 5, 8, 16, 31})
      if (check(F, vr, nrhs, narrowed)) {
        std::printf("%s: vr %d, %d right-hand sides\n", name, vr, nrhs);
        return 1;
      }
  std::printf("%s: %d launch shapes with fewer columns staged\n", name, narrowed);
  return 0;
}

int main() {
  if (check_all(bordered(2500, 3, 380), "2500 cells of 3 and one of 380")) return 1;
  if (check_all(bordered(3000, 2, 450), "3000 cells of 2 and one of 450")) return 1;
  if (check_all(bordered(3000, 3, 500), "3000 cells of 3 and one of 500")) return 1;
  if (check_all(bordered(40, 3, 380), "40 cells of 3 and one of 380")) return 1;
  if (check_all(uneven(200, 2, 900), "200x200 cells of 2, one of 900")) return 1;
  if (check_all(uneven(100, 4, 600), "100x100 cells of 4, one of 600")) return 1;
  std::printf("OK\n");
  return 0;
}
