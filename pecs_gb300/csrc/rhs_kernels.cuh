// Per-step right-hand-side kernels of the IMEX loop.
//
// k_carrier_rhs restates assemble_local_semiconductor_rhs /
// assemble_local_electrolyte_rhs plus the M u^{n-1} mat-vec of
// assemble_semiconductor_rhs / assemble_electrolyte_rhs (reference
// source/SolarCell.cpp:1037-1726): drift q/eps (p . D) u^{n-1} with D the RT
// field of the Poisson solution evaluated at the carrier quadrature points,
// SRH, the semiconductor--electrolyte interface Robin transfer and Schottky
// terms; generation and Dirichlet data are time independent and arrive
// pre-assembled in `bconst`.  One thread per (cell, carrier): a k=1 cell owns
// 4 density dofs and 4 field dofs (96 bytes), so a warp per cell would leave
// most lanes idle; neighbouring threads read neighbouring dof blocks, so the
// loads of a warp are contiguous.
//
// k_poisson_rhs restates assemble_local_Poisson_rhs_for_semiconductor /
// _for_electrolyte (SolarCell.cpp:487-815): -(v, sum q_i u_i) on the Phi rows
// of the matching Poisson cell plus the constant doping/Dirichlet part.
#pragma once
#include "fp_bits.cuh"
#include <type_traits>
#include <cuda_runtime.h>

namespace pecs {

struct Tables {
  const double* fphi;   // 4*n1*nq face values
  const double* fw;     // nq
  const double* charge; // Poisson charge matrix sum_q phiP_a phi_b w_q on the unit square, nphi x n1
};

// One-dimensional factors of the carrier element's tables, a kernel argument: the
// products take them as constant-bank operands, without loads.  All cells are
// axis-aligned rectangles and every basis is a tensor product (fe.hpp), so the
// element integrals are products of these.
// K: LDG degree; KP: the Poisson element is RT_{KP-1} x DGQ_{KP-1}.  V: double, or
// float2 (FP32 pairs); Tq: the arithmetic type of the quadrature terms.
template <int K, int KP, typename V, typename Tq>
struct Tab1D {
  static constexpr int m = K + 1, nq = K + 2;
  Tq L[nq][m];      // Lagrange basis at the Gauss points
  Tq w[nq];         // Gauss weights
  V mass[m][m];     // int l_a l_b
  V X[m][m][KP + 1];  // int l_a l_b xi_j, xi: the RT normal direction's basis
  V Y[m][m][KP];      // int l_a l_b eta_j, eta: the tangential direction's
};

struct RegionDev {
  int nc;              // cells
  int nd;              // dofs per carrier vector
  int field1;          // PECS_FIELD_N (semi) or PECS_FIELD_R (elec)
  int is_semi;
  int iface_face;      // face of this region's cells on the interface
  int partner_face;    // face of the partner cell
  double inv_eps;      // 1/permittivity of the region
  double inv_dt;
  const double2* h;    // (hx, hy) per cell
  const int4* bid;     // boundary id per face (-1 interior)
  const int* rt;       // nc*nrt Poisson RT dofs of the matching Poisson cell
  const int* phid;     // nc*nphi Poisson Phi dofs
  const int* partner;  // partner cell in the other region or -1
  const int* iface;    // interface index or -1
  const double2* ph;   // partner (hx, hy)
};

struct InstDev {
  double k_et, k_ht, tau_n, tau_p, n_i, s_n, s_p;
  int srh;
  int pad;
};

struct FieldPtrs {
  const double* u[5];   // state read (instance stride nd[f])
  double* out[5];       // written vectors (rhs)
  const double* bc[5];  // constant rhs parts
  int nd[5];
};

// K: LDG degree; KP - 1: degree of the Poisson element RT_{KP-1} x DGQ_{KP-1}
// (KP = K: the reference's pairing, SolarCell.cpp:23-24; KP = K + 1: the
// RT_K x DGQ_K pairing of the benchmark configurations)
template <int K, int KP>
struct Dims {
  static constexpr int n1 = (K + 1) * (K + 1);
  static constexpr int nq = K + 2;
  static constexpr int Q = nq * nq;
  static constexpr int nrt = 2 * KP * (KP + 1);
  static constexpr int nphi = KP * KP;
};

// state values into the quadrature type: on the integer pipe for the FP32 path
// (fp_bits.cuh), plain for FP64
template <typename Tq>
__device__ __forceinline__ Tq to_q(double x) {
  if constexpr (sizeof(Tq) == 4) return d2f_trunc(x); else return x;
}

// Sums of products in double, or in FP32 pairs: products exact through fmaf, the
// high parts added by TwoSum, the low parts in plain FP32 (the residuals' scheme;
// ~46 bits of the sum).
struct SumF64 {
  using V = double;
  double s = 0.0;
  __device__ __forceinline__ void add(double a, double b) { s += a * b; }
  __device__ __forceinline__ double get() const { return s; }
};
struct SumFF {
  using V = float2;
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(float2 a, float2 b) {
    const float p = a.x * b.x;
    const float pe = fmaf(a.x, b.x, -p) + fmaf(a.x, b.y, a.y * b.x);
    const float t = h + p;
    const float z = t - h;
    const float e = (h - (t - z)) + (p - z);
    h = t;
    l += e + pe;
  }
  __device__ __forceinline__ float2 get() const { return ff_fast_two_sum(h, l); }
};

__device__ __forceinline__ double v_of(double x, double) { return x; }
__device__ __forceinline__ float2 v_of(double x, float2) { return d2ff(x); }
__device__ __forceinline__ double v_mul(double a, double b) { return a * b; }
__device__ __forceinline__ float2 v_mul(float2 a, float2 b) { return ff_mul(a, b); }
__device__ __forceinline__ double v_neg(double a) { return -a; }
__device__ __forceinline__ float2 v_neg(float2 a) { return make_float2(-a.x, -a.y); }
// constant part + value, as double (pairs: 32-bit integer operations only)
__device__ __forceinline__ double v_out(double bc, double v) { return bc + v; }
__device__ __forceinline__ double v_out(double bc, float2 v) { return ff2d_i32(ff_add(d2ff(bc), v)); }
__device__ __forceinline__ double v_out(double bc, double v, double q) { return bc + v + q; }
__device__ __forceinline__ double v_out(double bc, float2 v, float q) {
  return ff2d_i32(ff_add(ff_add(d2ff(bc), v), q));
}

// grid: x over (cells of both regions) * 2 carriers, y over instances.
// Tq is the arithmetic type of the quadrature terms (SRH, interface, Schottky).
// Tq = double is the FP64 path.  Tq = float is the mixed path: (1/dt) M u^{n-1} and
// the drift term of the current equations, (q/eps) u D, keep ~46-bit accuracy --
// the drift is large (|D|/h relative to the density terms) and its rounding
// would leave a per-step noise of ~eps32 |D| dt / h in the densities, above a 1e-8
// steady-state criterion -- but run in FP32-pair arithmetic on the FP32 pipe
// (fp_bits.cuh; inputs split on the integer pipe); the small recombination and
// interface terms run in plain FP32 (GB300 issues FP32 operations ~60x faster than
// FP64, conversions included).
//
// The kernel is bound by its arithmetic: the FP64 path by the FP64 unit, where a
// warp instruction takes 64 cycles of its quarter SM however few warps there are; the
// mixed path by the FP32 and integer pipes.  So the element integrals are taken
// direction by direction (drift: for each tangential RT index, the normal
// direction's 1-D matrix sum_j X_abj D_j, applied to u along it, then Y along the other:
// 44 products per carrier at degree 1 where the full tensors took 80, 288 against 1,080
// at degree 2), the tables are constant operands, and the recombination, the same for
// both carriers, is evaluated by the two threads of a cell at half of the
// quadrature points each.  Measured per launch, us, before -> after: 64 instances of
// the 64x64+64x64 half cell, degree 1, mixed 232 -> 156; one instance, FP64 32 -> 21;
// 8 instances, degree 2, mixed 263 -> 119; 12 instances of 29x37+23x37 cells,
// degree 2, FP64 224 -> 80; 3 instances of 72x72+72x72, degree 2, RT_2 FP64 300 -> 118.
template <int K, int KP, typename Tq>
__global__ void __launch_bounds__(128, (K == 1 && sizeof(Tq) == 4) ? 8 : 1)
    k_carrier_rhs(const __grid_constant__ Tab1D<K, KP, typename std::conditional<sizeof(Tq) == 4, float2, double>::type, Tq> T,
                  RegionDev semi, RegionDev elec, int n_regions, FieldPtrs F,
                  const InstDev* __restrict__ inst, const double* __restrict__ iface_ne,
                  const double* __restrict__ iface_pe, int n_iface, const double* __restrict__ sch_ne,
                  const double* __restrict__ sch_pe, const int* __restrict__ active) {
  using D = Dims<K, KP>;
  using Sum = typename std::conditional<sizeof(Tq) == 4, SumFF, SumF64>::type;
  using V = typename Sum::V;
  constexpr int n1 = D::n1, nq = D::nq, nrt = D::nrt, m = K + 1;
  const int i = blockIdx.y;
  if (active && !active[i]) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nsemi2 = 2 * semi.nc;
  const int ntot = nsemi2 + (n_regions > 1 ? 2 * elec.nc : 0);
  if (t >= ntot) return;
  const bool in_semi = t < nsemi2;
  const RegionDev& R = in_semi ? semi : elec;
  const RegionDev& O = in_semi ? elec : semi;
  if (!in_semi) t -= nsemi2;
  const int c = t >> 1, which = t & 1;  // which: 0 carrier_1, 1 carrier_2
  const int f1 = R.field1, f = f1 + which;
  const int nc = R.nc, nd = R.nd;
  const InstDev P = inst[i];
  const double* u1p = F.u[f1] + (size_t)i * F.nd[f1] + 2 * nc * n1 + c * n1;
  const double* u2p = F.u[f1 + 1] + (size_t)i * F.nd[f1 + 1] + 2 * nc * n1 + c * n1;
  const double* Pv = F.u[4] + (size_t)i * F.nd[4];
  const double* bcp = F.bc[f] + (size_t)i * nd;
  double* outp = F.out[f] + (size_t)i * nd;
  const double2 h = R.h[c];
  Tq u1[n1], u2[n1];
  V u[n1];  // the thread's own carrier
#pragma unroll
  for (int a = 0; a < n1; ++a) {
    const double x1 = u1p[a], x2 = u2p[a];
    u[a] = v_of(which ? x2 : x1, V());
    u1[a] = to_q<Tq>(x1);
    u2[a] = to_q<Tq>(x2);
  }
  // current rows: (charge / eps) hx hy sum_bc T_abc u_b D_c.  dir 0: x components
  // (normal direction x); dir 1 with the roles of x and y exchanged
  const V area = v_mul(v_of(h.x, V()), v_of(h.y, V()));
  {
    V sc = v_mul(v_of(R.inv_eps, V()), area);
    if (!which) sc = v_neg(sc);
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      Sum W[m][m];  // [normal a1][tangential a2]
#pragma unroll 1
      for (int j2 = 0; j2 < KP; ++j2) {
        V Dv[KP + 1];
#pragma unroll
        for (int j1 = 0; j1 <= KP; ++j1) {
          const int b = dir == 0 ? j1 + (KP + 1) * j2 : nrt / 2 + j2 + KP * j1;
          Dv[j1] = v_of(Pv[R.rt[c * nrt + b]], V());
        }
        V C[m][m];  // symmetric
#pragma unroll
        for (int a = 0; a < m; ++a)
#pragma unroll
          for (int b = a; b < m; ++b) {
            Sum s;
#pragma unroll
            for (int j1 = 0; j1 <= KP; ++j1) s.add(T.X[a][b][j1], Dv[j1]);
            C[a][b] = C[b][a] = s.get();
          }
#pragma unroll
        for (int a1 = 0; a1 < m; ++a1) {
          V vv[m];
#pragma unroll
          for (int b2 = 0; b2 < m; ++b2) {
            Sum s;
#pragma unroll
            for (int b1 = 0; b1 < m; ++b1) s.add(C[a1][b1], dir == 0 ? u[b1 + m * b2] : u[b2 + m * b1]);
            vv[b2] = s.get();
          }
#pragma unroll
          for (int a2 = 0; a2 < m; ++a2)
#pragma unroll
            for (int b2 = 0; b2 < m; ++b2) W[a1][a2].add(T.Y[a2][b2][j2], vv[b2]);
        }
      }
      const size_t o = (size_t)dir * nc * n1 + c * n1;
#pragma unroll
      for (int a1 = 0; a1 < m; ++a1)
#pragma unroll
        for (int a2 = 0; a2 < m; ++a2) {
          const int a = dir == 0 ? a1 + m * a2 : a2 + m * a1;
          outp[o + a] = v_out(bcp[o + a], v_mul(sc, W[a1][a2].get()));
        }
    }
  }
  // quadrature terms of the density rows
  Tq r[n1];
#pragma unroll
  for (int a = 0; a < n1; ++a) r[a] = Tq(0);
  if (in_semi && P.srh) {
    // Quadrature rows of this thread: nq / 2 whole ones from its end, and where nq
    // is odd its part of the middle one (thread 0 the larger).  The other thread of
    // the cell adds the rest.
    const Tq hxhy_q = std::is_same<Tq, double>::value ? (Tq)(h.x * h.y) : to_q<Tq>(h.x) * to_q<Tq>(h.y);
    const Tq ni = to_q<Tq>(P.n_i), taun = to_q<Tq>(P.tau_n), taup = to_q<Tq>(P.tau_p);
#pragma unroll 1
    for (int row = 0; row < (nq + 1) / 2; ++row) {
      const bool middle = nq % 2 == 1 && row == nq / 2;
      const int qy = which ? nq - 1 - row : row;
      Tq Ly[m];
#pragma unroll
      for (int a = 0; a < m; ++a) Ly[a] = T.L[qy][a];
      Tq g1[m], g2[m], hr[m];
#pragma unroll
      for (int ax = 0; ax < m; ++ax) {
        g1[ax] = g2[ax] = hr[ax] = Tq(0);
#pragma unroll
        for (int ay = 0; ay < m; ++ay) {
          g1[ax] += Ly[ay] * u1[ax + m * ay];
          g2[ax] += Ly[ay] * u2[ax + m * ay];
        }
      }
      const int x0 = middle && which ? (nq + 1) / 2 : 0;
      const int x1 = middle && !which ? (nq + 1) / 2 : nq;
#pragma unroll 1
      for (int qx = x0; qx < x1; ++qx) {
        Tq n = 0, p = 0;
#pragma unroll
        for (int ax = 0; ax < m; ++ax) {
          n += T.L[qx][ax] * g1[ax];
          p += T.L[qx][ax] * g2[ax];
        }
        const Tq JxW = T.w[qx] * T.w[qy] * hxhy_q;
        const Tq Rq = (ni * ni - n * p) / (taun * (n + ni) + taup * (p + ni)) * JxW;
#pragma unroll
        for (int ax = 0; ax < m; ++ax) hr[ax] += T.L[qx][ax] * Rq;
      }
#pragma unroll
      for (int ay = 0; ay < m; ++ay)
#pragma unroll
        for (int ax = 0; ax < m; ++ax) r[ax + m * ay] += Ly[ay] * hr[ax];
    }
    // both threads of a cell are here; each gets the same sum
    const unsigned pair = 3u << (threadIdx.x & 30);
#pragma unroll
    for (int a = 0; a < n1; ++a) r[a] += __shfl_xor_sync(pair, r[a], 1);
  }
  // interface Robin transfer (SolarCell.cpp:1265-1347, 1630-1716); a face's traces
  // are its own nodes' values
  const int4 bid = R.bid[c];
  const int bids[4] = {bid.x, bid.y, bid.z, bid.w};
  if (n_regions > 1 && R.iface[c] >= 0 && (R.iface_face == 0 ? bids[0] : bids[1]) == 0) {
    const int pc = R.partner[c], ii = R.iface[c];
    const double* o1p = F.u[O.field1] + (size_t)i * F.nd[O.field1] + 2 * O.nc * n1 + pc * n1;
    const double* o2p = F.u[O.field1 + 1] + (size_t)i * F.nd[O.field1 + 1] + 2 * O.nc * n1 + pc * n1;
    const bool right = R.iface_face == 1, p_right = R.partner_face == 1;
    const Tq flen = to_q<Tq>(h.y);
    const Tq ket = to_q<Tq>(P.k_et), kht = to_q<Tq>(P.k_ht);
    Tq f1v[m], f2v[m], g1v[m], g2v[m], hr[m];
#pragma unroll
    for (int y = 0; y < m; ++y) {
      f1v[y] = right ? u1[K + m * y] : u1[m * y];
      f2v[y] = right ? u2[K + m * y] : u2[m * y];
      g1v[y] = to_q<Tq>(o1p[(p_right ? K : 0) + m * y]);
      g2v[y] = to_q<Tq>(o2p[(p_right ? K : 0) + m * y]);
      hr[y] = Tq(0);
    }
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
      Tq a1 = 0, a2 = 0, b1 = 0, b2 = 0;
#pragma unroll
      for (int y = 0; y < m; ++y) {
        a1 += T.L[q][y] * f1v[y];
        a2 += T.L[q][y] * f2v[y];
        b1 += T.L[q][y] * g1v[y];
        b2 += T.L[q][y] * g2v[y];
      }
      // semiconductor-side values n, p and electrolyte-side r, o
      const Tq n = in_semi ? a1 : b1, p = in_semi ? a2 : b2;
      const Tq rr = in_semi ? b1 : a1, oo = in_semi ? b2 : a2;
      const Tq ne = to_q<Tq>(iface_ne[(size_t)i * n_iface * nq + ii * nq + q]);
      const Tq pe = to_q<Tq>(iface_pe[(size_t)i * n_iface * nq + ii * nq + q]);
      const Tq Jf = T.w[q] * flen;
      const Tq tn = -ket * (n - ne) * oo * Jf;
      const Tq tp = kht * (p - pe) * rr * Jf;
      Tq coef;
      if (in_semi)
        coef = which ? tp : tn;
      else
        coef = which ? -(tn + tp) : (tn + tp);
#pragma unroll
      for (int y = 0; y < m; ++y) hr[y] += T.L[q][y] * coef;
    }
#pragma unroll
    for (int y = 0; y < m; ++y) {
      if (right)
        r[K + m * y] += hr[y];
      else
        r[m * y] += hr[y];
    }
  }
  // Schottky faces (SolarCell.cpp:1348-1404)
  if (in_semi && sch_ne) {
#pragma unroll
    for (int fc = 0; fc < 4; ++fc) {
      if (bids[fc] != 3) continue;
      const Tq flen = to_q<Tq>((fc == 0 || fc == 1) ? h.y : h.x);
#pragma unroll 1
      for (int q = 0; q < nq; ++q) {
        Tq val = 0;
#pragma unroll
        for (int y = 0; y < m; ++y) {
          const int a = fc == 0 ? m * y : fc == 1 ? K + m * y : fc == 2 ? y : y + m * K;
          val += T.L[q][y] * (which ? u2[a] : u1[a]);
        }
        const size_t o = (size_t)i * nc * 4 * nq + (size_t)(c * 4 + fc) * nq + q;
        const Tq Jf = T.w[q] * flen;
        const Tq coef = which ? to_q<Tq>(P.s_p) * (val - to_q<Tq>(sch_pe[o])) * Jf
                              : -to_q<Tq>(P.s_n) * (val - to_q<Tq>(sch_ne[o])) * Jf;
#pragma unroll
        for (int y = 0; y < m; ++y) {
          const int a = fc == 0 ? m * y : fc == 1 ? K + m * y : fc == 2 ? y : y + m * K;
          r[a] += T.L[q][y] * coef;
        }
      }
    }
  }
  // density rows: constant part + (1/dt) M u^{n-1} + quadrature terms
  const V md = v_mul(area, v_of(R.inv_dt, V()));
  V mx[n1];
#pragma unroll
  for (int ay = 0; ay < m; ++ay)
#pragma unroll
    for (int ax = 0; ax < m; ++ax) {
      Sum s;
#pragma unroll
      for (int b = 0; b < m; ++b) s.add(T.mass[ax][b], u[b + m * ay]);
      mx[ax + m * ay] = s.get();
    }
#pragma unroll
  for (int ay = 0; ay < m; ++ay)
#pragma unroll
    for (int ax = 0; ax < m; ++ax) {
      Sum s;
#pragma unroll
      for (int b = 0; b < m; ++b) s.add(T.mass[ay][b], mx[ax + m * b]);
      const size_t o = (size_t)2 * nc * n1 + c * n1 + ax + m * ay;
      outp[o] = v_out(bcp[o], v_mul(s.get(), md), r[ax + m * ay]);
    }
}

// grid: x over max(n_rt_total, cells of both regions), y over instances
template <int K, int KP>
__global__ void __launch_bounds__(128)
    k_poisson_rhs(Tables T, RegionDev semi, RegionDev elec, int n_regions, FieldPtrs F,
                  int n_rt_total, const int* __restrict__ active) {
  using D = Dims<K, KP>;
  constexpr int n1 = D::n1, Q = D::Q, nphi = D::nphi;
  const int i = blockIdx.y;
  if (active && !active[i]) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const double* bc = F.bc[4] + (size_t)i * F.nd[4];
  double* out = F.out[4] + (size_t)i * F.nd[4];
  if (t < n_rt_total) out[t] = bc[t];
  const int ntot = semi.nc + (n_regions > 1 ? elec.nc : 0);
  if (t >= ntot) return;
  const bool in_semi = t < semi.nc;
  const RegionDev& R = in_semi ? semi : elec;
  const int c = in_semi ? t : t - semi.nc;
  const int f1 = R.field1;
  const double* u1 = F.u[f1] + (size_t)i * F.nd[f1] + 2 * R.nc * n1 + c * n1;
  const double* u2 = F.u[f1 + 1] + (size_t)i * F.nd[f1 + 1] + 2 * R.nc * n1 + c * n1;
  const double2 h = R.h[c];
  // charge density (-u1 + u2) (charge numbers -1, +1) against the Poisson test
  // functions: the quadrature folded into the nphi x n1 matrix T.charge, so
  // each cell costs nphi * n1 FP64 FMAs
  double du[n1];
#pragma unroll
  for (int b = 0; b < n1; ++b) du[b] = u2[b] - u1[b];
  const double hxhy = h.x * h.y;
  double acc[nphi];
#pragma unroll
  for (int a = 0; a < nphi; ++a) {
    double t = 0.0;
#pragma unroll
    for (int b = 0; b < n1; ++b) t += T.charge[a * n1 + b] * du[b];
    acc[a] = t * hxhy;
  }
#pragma unroll
  for (int a = 0; a < nphi; ++a) {
    const int d = R.phid[c * nphi + a];
    out[d] = bc[d] - acc[a];
  }
}

}  // namespace pecs
