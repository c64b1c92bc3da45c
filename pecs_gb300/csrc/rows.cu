// Few-right-hand-side solve sweeps (rows.cuh): kernels, tile plans, launches.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <type_traits>

#include "bulk_copy.cuh"
#include "rows.cuh"
#include "sweep_sync.cuh"

namespace pecs {

namespace {

constexpr size_t kMostColBytes = 200 * 1024;  // one right-hand side of the widest front a bank takes
constexpr int kAsmMinRhs = 5;              // right-hand sides from which columns are assembled once per node
constexpr int kAsmMinRb = 3;               // smallest chunk those counts are cut into
constexpr int kAsmTiles = 8;               // tiles per node from which kAsmMinRb right-hand sides are enough

template <typename T>
struct VecOf;
template <>
struct VecOf<double> {
  using type = double2;
  static constexpr int n = 2;
};
template <>
struct VecOf<float> {
  using type = float4;
  static constexpr int n = 4;
};

template <int RB>
__device__ __forceinline__ void fma_vec(double (&acc)[2][RB], const double2& m, const double (&d)[RB]) {
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    acc[0][r] += m.x * d[r];
    acc[1][r] += m.y * d[r];
  }
}
template <int RB>
__device__ __forceinline__ void fma_vec(float (&acc)[4][RB], const float4& m, const float (&d)[RB]) {
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    acc[0][r] += m.x * d[r];
    acc[1][r] += m.y * d[r];
    acc[2][r] += m.z * d[r];
    acc[3][r] += m.w * d[r];
  }
}
template <int RB>
__device__ __forceinline__ void st_vec(double* p, const double (&acc)[2][RB], int r) {
  *reinterpret_cast<double2*>(p) = make_double2(acc[0][r], acc[1][r]);
}
template <int RB>
__device__ __forceinline__ void st_vec(float* p, const float (&acc)[4][RB], int r) {
  *reinterpret_cast<float4*>(p) = make_float4(acc[0][r], acc[1][r], acc[2][r], acc[3][r]);
}

// Right-hand sides per thread of a chunk of RB
template <int RB>
struct RowsRt {
  static constexpr int n = RB <= 4 ? RB : (RB == 6 ? 3 : 4);
};

// RB consecutive staged values (aligned to their size where that is 8 or 16 bytes)
template <typename T, int RB>
__device__ __forceinline__ void ld_row(const T* p, T (&v)[RB]) {
  constexpr int bytes = RB * (int)sizeof(T);
  if constexpr (sizeof(T) == 8 && bytes % 16 == 0) {
#pragma unroll
    for (int q = 0; q < RB / 2; ++q) {
      const double2 t = reinterpret_cast<const double2*>(p)[q];
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else if constexpr (sizeof(T) == 4 && bytes % 16 == 0) {
#pragma unroll
    for (int q = 0; q < RB / 4; ++q) {
      const float4 t = reinterpret_cast<const float4*>(p)[q];
      v[4 * q] = t.x;
      v[4 * q + 1] = t.y;
      v[4 * q + 2] = t.z;
      v[4 * q + 3] = t.w;
    }
  } else if constexpr (sizeof(T) == 4 && bytes % 8 == 0) {
#pragma unroll
    for (int q = 0; q < RB / 2; ++q) {
      const float2 t = reinterpret_cast<const float2*>(p)[q];
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int r = 0; r < RB; ++r) v[r] = p[r];
  }
}

// barrier of one team: a warp, or 64 to 256 threads of the CTA (team index + 1
// names the hardware barrier; 0 is the CTA's own)
__device__ __forceinline__ void team_sync(int ts, int team) {
  if (ts == 32)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;\n" ::"r"(team + 1), "r"(ts) : "memory");
}

// Partial sums: stride between right-hand sides, in values: one 16-byte step off a
// multiple of 128 bytes, so that outputs read with the right-hand side fastest
// meet few bank conflicts.
template <typename T>
__host__ __device__ inline int red_stride(int n) {
  constexpr int line = 128 / (int)sizeof(T), vec = 16 / (int)sizeof(T);
  return (n + line - 1) / line * line + vec;
}

// A column's value -- b minus the children's updates -- or (COL = false) a
// pass-through row's: the children's sum.
template <bool COL>
__device__ __forceinline__ double rec_value(const RowRec& q, const RowSet& st, const int* __restrict__ more, int R,
                                            int r) {
  const double* w = st.w + r;
  double b = 0.0, u[kRowsSlots];
  if (COL) b = __ldcg(st.b + (size_t)q.src * st.sd + (size_t)r * st.sr);
#pragma unroll
  for (int j = 0; j < kRowsSlots; ++j) {
    u[j] = 0.0;
    if (q.slot[j] >= 0) u[j] = __ldcg(w + (size_t)q.slot[j] * R);
  }
  // most positions have few children; the rest is a branch, so that it does not pass
  // through the FP64 unit where no lane of a warp has more (a vote of the whole warp in
  // its place, behind the records' loads: 16x16 junction 26.73 ms for 100 steps, 26.55)
  double s = u[0];
  if (q.slot[1] >= 0) s += u[1];
  if (q.slot[2] >= 0) {
#pragma unroll
    for (int j = 2; j < kRowsSlots; ++j)
      if (q.slot[j] >= 0) s += u[j];
    if (q.slot[kRowsSlots - 1] < -1) {
      const int* m = more + (-2 - q.slot[kRowsSlots - 1]);
      for (int j = 1; j <= m[0]; ++j) s += __ldcg(w + (size_t)m[j] * R);
    }
  }
  return COL ? (q.slot[0] >= 0 ? b - s : b) : s;
}

// FP32 factors: y and the sweep's copy of x are single precision (rows.cuh)
template <typename T>
__device__ __forceinline__ T* row_y(const RowSet& st) { return reinterpret_cast<T*>(st.y); }
__device__ __forceinline__ float* row_xf(const RowSet& st, int n) {
  return reinterpret_cast<float*>(st.y) + (size_t)n * st.nrhs;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}

// Columns [0, kc) of the chunk's source values into shared memory: row(p) is
// column p's R interleaved values.  Whole 16-byte pieces by asynchronous copies
// where the rows allow (all of them in flight at once), else value by value; always
// from L2: rows are shorter than cache lines, whose other rows earlier launches wrote.
template <typename T, int RB, typename Row>
__device__ __forceinline__ void stage(T* Ds, int kc, int rb, int R, int t, int ts, Row row) {
  constexpr int VR = 16 / (int)sizeof(T);
  if (RB % VR == 0 && R % VR == 0) {
    constexpr int NV = RB % VR == 0 ? RB / VR : 1;
    for (int e0 = t; e0 < kc * NV; e0 += 4 * ts) {
      const T* q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * ts;
        q[u] = e < kc * NV ? row(e / NV) + rb + (e % NV) * VR : nullptr;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * ts;
        if (e >= kc * NV) continue;
        if (rb + (e % NV) * VR < R)
          cp_async16(Ds + e * VR, q[u]);
        else
#pragma unroll
          for (int j = 0; j < VR; ++j) Ds[e * VR + j] = T(0);
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  } else {
    for (int e0 = t; e0 < kc * RB; e0 += 4 * ts) {
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + u * ts;
        v[u] = e < kc * RB && rb + e % RB < R ? __ldcg(row(e / RB) + rb + e % RB) : T(0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e0 + u * ts < kc * RB) Ds[e0 + u * ts] = v[u];
    }
  }
}

// One tile applied to right-hand sides [chunk * RB, chunk * RB + RB) of its set.
// Before wait() only what no other launch or item writes is read: the tile's
// values (one bulk copy into shared memory; a thread then reads those that it
// needs itself) and the source records.  wait() (every thread of the team) returns
// false when the inputs could not be waited for; the tile then writes NaN.  ASM: the
// columns were assembled beforehand (k_assemble).
template <typename T, int RB, bool FWD, bool ASM, typename Wait>
__device__ __forceinline__ void rows_tile(const RowsDirView& B, const RowSets& S, const RowItem* __restrict__ item,
                                          int chunk, int ts, int team, const RowsSmem& M, unsigned char* smem,
                                          Wait wait) {
  using V = typename VecOf<T>::type;
  constexpr int VR = VecOf<T>::n;
  const int t = (int)threadIdx.x & (ts - 1);
  const RowItem I = *item;
  constexpr int RT = RowsRt<RB>::n, RG = RB / RT;  // right-hand sides per thread, threads that share a row vector
  const int per = I.pad, K = I.cols, rg = per / VR;
  const int KG = min((ts / RG * I.magic) >> 16, K);  // columns handled at a time
  const int kc_max = min(I.kc, M.kc);
  const unsigned bar = smem_u32(smem), buf = bar + 16;
  const T* val = static_cast<const T*>(B.val) + I.off;
  if (t == 0) {
    bar_init(bar);
    bar_init(bar + 8);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    bulk_load(buf, val, min(K, kc_max) * per * (int)sizeof(T), bar);
    if (K > kc_max)
      bulk_load(buf + M.buf, val + (size_t)kc_max * per, min(K - kc_max, kc_max) * per * (int)sizeof(T), bar + 8);
  }
  const RowSet& st = S.set[I.set];
  const int R = st.nrhs, rb = chunk * RB;
  // thread -> (right-hand sides rt.., row vector, column group); lanes with the same
  // row vector and the same right-hand sides read the same shared-memory words
  const int rt = t % RG * RT, kg = (t / RG * I.magic) >> 16, rv = t / RG - kg * rg;
  T* Ds = reinterpret_cast<T*>(smem + M.ds);
  double* cu = reinterpret_cast<double*>(smem + M.cu);
  const bool direct = FWD && !ASM;
  const int npt = direct && !I.leaf ? I.npt : 0;
  // outputs: G = 1 << lg lanes each, right-hand sides fastest
  const int no = I.rows * RB;
  int lg = 0;
  while ((2 << lg) <= KG && (no << (lg + 1)) <= ts && lg < 5) ++lg;
  const int o_first = min(t >> lg, no - 1);
  const int dst_first = B.dst[I.dst + o_first / RB];
  int kc = min(K, kc_max);
  RowRec rec{};
  if (direct && !I.leaf) {
    const int p = t / RB;
    if (p < kc)
      rec = B.rec[I.src + p];
    else if (p - kc < npt)
      rec = B.upd[I.pt + p - kc];
  }
  bool ok = wait();
  T acc[VR][RT];
#pragma unroll
  for (int v = 0; v < VR; ++v)
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[v][r] = T(0);
  for (int k0 = 0, q = 0;; ++q) {
    // (1) source values of the columns
    if (direct && I.leaf) {
      const int* src = B.src + I.src + k0;
      for (int e0 = t; e0 < kc * RB; e0 += 4 * ts) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = e0 + u * ts, r = rb + e % RB;
          v[u] = e < kc * RB && r < R ? __ldcg(st.b + (size_t)src[e / RB] * st.sd + (size_t)r * st.sr) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (e0 + u * ts < kc * RB) Ds[e0 + u * ts] = (T)v[u];
      }
    } else if (direct) {
      const int ne = (kc + (k0 == 0 ? npt : 0)) * RB;
      for (int e = t; e < ne; e += ts) {
        const int p = e / RB, r = e % RB;
        const bool col = p < kc;
        if (k0 > 0 || e != t) rec = col ? B.rec[I.src + k0 + p] : B.upd[I.pt + p - kc];
        double v = 0.0;
        if (rb + r < R) v = col ? rec_value<true>(rec, st, B.more, R, rb + r) : rec_value<false>(rec, st, B.more, R, rb + r);
        if (col)
          Ds[e] = (T)v;
        else
          cu[e - kc * RB] = v;
      }
    } else if (FWD) {
      stage<T, RB>(Ds, kc, rb, R, t, ts, [&](int p) {
        return reinterpret_cast<const T*>(st.d) + (size_t)(I.d + k0 + p) * R;
      });
    } else if (st.sr == 1 || sizeof(T) == 4) {
      const int* src = B.src + I.src + k0;
      const T* y = row_y<T>(st);
      const T* x = sizeof(T) == 4 ? reinterpret_cast<const T*>(row_xf(st, st.n)) : reinterpret_cast<const T*>(st.x);
      stage<T, RB>(Ds, kc, rb, R, t, ts, [&](int p) {
        const int z = src[p];
        return z >= 0 ? y + (size_t)z * R : x + (size_t)(~z) * R;
      });
    } else {
      const int* src = B.src + I.src + k0;
      for (int e0 = t; e0 < kc * RB; e0 += 4 * ts) {
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = e0 + u * ts, r = rb + e % RB;
          v[u] = T(0);
          if (e < kc * RB && r < R) {
            const int z = src[e / RB];
            v[u] = z >= 0 ? __ldcg(row_y<T>(st) + (size_t)z * R + r)
                          : (T)__ldcg(st.x + (size_t)(~z) + (size_t)r * st.sr);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (e0 + u * ts < kc * RB) Ds[e0 + u * ts] = v[u];
      }
    }
    team_sync(ts, team);
    // (2) the tile's columns, kg, kg + KG, ... : VR rows x RB sums per thread
    const int b = q & 1;
    ok = bar_wait(bar + 8 * b, (q >> 1) & 1) && ok;
    if (kg < KG) {
      const V* m = reinterpret_cast<const V*>(smem + 16 + b * M.buf) + kg * rg + rv;
      const T* d = Ds + kg * RB + rt;
#pragma unroll 4
      for (int k = kg; k < kc; k += KG) {
        T dv[RT];
        ld_row<T, RT>(d, dv);
        fma_vec<RT>(acc, *m, dv);
        m += KG * rg;
        d += KG * RB;
      }
    }
    k0 += kc;
    if (k0 >= K) break;
    kc = min(K - k0, kc_max);
    team_sync(ts, team);  // source values and value buffer b are free
    if (t == 0 && k0 + kc < K)
      bulk_load(buf + b * M.buf, val + (size_t)(k0 + kc) * per, min(K - k0 - kc, kc_max) * per * (int)sizeof(T),
                bar + 8 * b);
  }
  // (3) partial sums -> row totals -> destination
  T* red = Ds;
  const int rs = red_stride<T>(KG * per);
  team_sync(ts, team);          // the partial sums overlay the source values
  if (kg < KG) {
#pragma unroll
    for (int r = 0; r < RT; ++r) st_vec<RT>(red + (rt + r) * rs + kg * per + rv * VR, acc, r);
  }
  team_sync(ts, team);
  const int nown = I.rows - I.npt;
  auto emit = [&](int row, int r, int d, T sum, double add) {
    if (!ok) sum = (T)__longlong_as_double(0x7ff8000000000000ll);
    if (!FWD) {
      st.x[(size_t)d * st.sd + (size_t)(rb + r) * st.sr] = (double)sum;
      if constexpr (sizeof(T) == 4) row_xf(st, st.n)[(size_t)d * R + rb + r] = sum;
    } else if (row < nown) {
      row_y<T>(st)[(size_t)d * R + rb + r] = sum;
    } else {
      st.w[(size_t)d * R + rb + r] = I.leaf ? (double)sum : add + (double)sum;
    }
  };
  // what the children add to output (row, r) of destination d
  auto below = [&](int row, int r, int d) {
    if (!FWD || row < nown || I.leaf || rb + r >= R) return 0.0;
    return ASM ? __ldcg(st.w + (size_t)d * R + rb + r) : cu[(row - nown) * RB + r];
  };
  if (lg > 0) {  // one output per G lanes, each adding every G-th column group
    const int G = 1 << lg, g = t & (G - 1), o = t >> lg, row = o / RB, r = o % RB;
    if (((t & ~31) >> lg) < no) {
      const double add = o < no ? below(row, r, dst_first) : 0.0;
      T s = T(0);
      if (o < no) {
        const T* q = red + r * rs + row;
        for (int k = g; k < KG; k += G) s += q[k * per];
      }
      for (int off = G >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (g == 0 && o < no && rb + r < R) emit(row, r, dst_first, s, add);
    }
  } else {
    constexpr int Q = 4;  // outputs in flight per thread
    for (int o0 = t; o0 < no; o0 += Q * ts) {
      int d[Q];
      double add[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int o = o0 + q * ts;
        d[q] = o < no ? (o == t ? dst_first : B.dst[I.dst + o / RB]) : 0;
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int o = o0 + q * ts;
        add[q] = o < no ? below(o / RB, o % RB, d[q]) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int o = o0 + q * ts, row = o / RB, r = o % RB;
        if (o >= no || rb + r >= R) continue;
        T s = T(0);
        for (int k = 0; k < KG; ++k) s += red[r * rs + k * per + row];
        emit(row, r, d[q], s, add[q]);
      }
    }
  }
}

// A batch of small leaves (FP64 factors): a thread per output, the columns' values
// read where they are.
template <int RB, bool FWD, typename Wait>
__device__ __forceinline__ void rows_batch(const RowsDirView& B, const RowSets& S, const RowItem* __restrict__ item,
                                           int chunk, Wait wait) {
  const RowItem I = *item;
  const RowSet& st = S.set[I.set];
  const int R = st.nrhs, rb = chunk * RB;
  const bool ok = wait();
  const int rows = I.rows, K = I.cols, per_node = rows * RB, no = I.pad * per_node;
  const float inv = 1.0f / (float)per_node;
  for (int o = threadIdx.x; o < no; o += kRowsThreads) {
    const int q = (int)(((float)o + 0.5f) * inv), e = o - q * per_node;
    const int row = e / RB, r = rb + e % RB;
    if (r >= R) continue;
    const double* m = static_cast<const double*>(B.val) + I.off + (size_t)q * rows * K + row;
    const int* src = B.src + I.src + q * K;
    const int d = B.dst[I.dst + q * rows + row];
    double acc = 0.0;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      const int s = src[k];
      double v;
      if (FWD)
        v = __ldcg(st.b + (size_t)s * st.sd + (size_t)r * st.sr);
      else if (s >= 0)
        v = __ldcg(st.y + (size_t)s * R + r);
      else
        v = __ldcg(st.x + (size_t)(~s) * st.sd + (size_t)r * st.sr);
      acc += __ldg(m + (size_t)k * rows) * v;
    }
    if (!ok) acc = __longlong_as_double(0x7ff8000000000000ll);
    if (!FWD)
      st.x[(size_t)d * st.sd + (size_t)r * st.sr] = acc;
    else
      (row < rows - I.npt ? st.y : st.w)[(size_t)d * R + r] = acc;
  }
}

// One tree level.  What bounds it (GB300): levels of small trees the latency of one
// tile -- records and columns from L2, partial sums, the next launch: 4 us a level
// on 16x16 cells; FP64 levels of the 64x64+64x64 half cell the FP64 unit (one warp
// instruction per 64 cycles and quarter SM: 50 us of products per carrier sweep of
// 2 right-hand sides); FP32 with 8 and more right-hand sides the update vectors.
// Values go through shared memory by one bulk copy issued before the wait because
// loads into registers were moved behind it (1.5 us of DRAM latency per level, and 32
// registers); a sweep, us before -> after this kernel against the earlier warp-per-
// row one, carriers / Poisson: 16x16 p-n junction 171 / 134 -> 56 / 53; half cell,
// FP64, 1 instance 519 / 222 -> 223 / 115; 64x64+64x64, k = 2, FP32, 8 instances
// 2754 / 1043 -> 451 / 223; 29x37+23x37, k = 2, FP64, 12 instances 1963 / 1593 ->
// 829 / 405.
template <typename T, int RB, bool FWD, bool ASM>
__global__ void __launch_bounds__(kRowsThreads, RB <= 2 ? 4 : 3)
    k_rows(RowsDirView B, RowSets S, int first, int n_tile, int tile_blocks, int ts_log, RowsSmem M) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  auto wait = [] {
    pdl_wait();
    return true;
  };
  if ((int)blockIdx.x < tile_blocks) {
    const int team = threadIdx.x >> ts_log;
    const int i = ((int)blockIdx.x << (8 - ts_log)) + team;
    if (i >= n_tile) return;
    rows_tile<T, RB, FWD, ASM>(B, S, B.items + first + i, (int)blockIdx.y, 1 << ts_log, team, M,
                               smem_raw + team * M.team_bytes, wait);
  } else if constexpr (sizeof(T) == 8) {
    rows_batch<RB, FWD>(B, S, B.items + first + n_tile + (int)blockIdx.x - tile_blocks, (int)blockIdx.y, wait);
  }
}

// The columns and pass-through sums of one level's tile nodes, once per node
// instead of once per tile: column values -> d in the blocks' type, the children's
// sums of the update rows -> w.
struct AsmRange {
  int col, n_col, d, upd, n_upd;  // first column record, columns, first place in d, first update record, records
};
struct AsmRanges {
  AsmRange set[kRowsMaxSets];
};

template <typename T>
__global__ void __launch_bounds__(256) k_assemble(RowsDirView B, RowSets S, AsmRanges A) {
  pdl_trigger();
  const AsmRange& g = A.set[blockIdx.y];
  const RowSet& st = S.set[blockIdx.y];
  const int R = st.nrhs;
  const unsigned e = blockIdx.x * 256 + threadIdx.x;
  const int p = (int)(e / (unsigned)R), r = (int)e - p * R;
  const bool in = p < g.n_col + g.n_upd, col = p < g.n_col;
  RowRec q{};
  if (in) q = col ? B.rec[g.col + p] : B.upd[g.upd + p - g.n_col];
  pdl_wait();
  if (!in) return;
  if (col)
    reinterpret_cast<T*>(st.d)[(size_t)(g.d + p) * R + r] = (T)rec_value<true>(q, st, B.more, R, r);
  else
    st.w[(size_t)q.src * R + r] = rec_value<false>(q, st, B.more, R, r);
}

// Flow sweep: one persistent launch per direction over the same items in
// topological order, with a ticket queue, per-node counters, bounded waits, release
// signals deferred past the next entry's first barrier and each direction
// zeroing the other's counters, as the panel flow sweep (k_panel_flow).
struct RowsFlowView {
  const RowEntry* entries;
  const RowSync* sync;
  int* ctr;
  int* other_ctr;
  int n_ctr;
  int* queue;
  int* other_queue;
  int* err;
  int n_entries;
};

struct RowsSmem4 {
  RowsSmem ts[4];  // teams of 32, 64, 128, 256 threads
};

template <typename T, int RB, bool FWD>
__global__ void __launch_bounds__(kRowsThreads, 2)
    k_rows_flow(RowsDirView B, RowSets S, RowsFlowView F, RowsSmem4 M) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_ticket, s_ok[kRowsThreads / 32];
  const int tid = threadIdx.x;
  for (int i = blockIdx.x * kRowsThreads + tid; i < F.n_ctr; i += gridDim.x * kRowsThreads) F.other_ctr[i] = 0;
  if (blockIdx.x == 0 && tid == 0) *F.other_queue = 0;
  int pending = -1;  // the counter this thread still has to signal
  if (tid == 0) s_ticket = atomicAdd(F.queue, 1);
  for (;;) {
    __syncthreads();
    const int t = s_ticket;
    if (pending >= 0) red_release_gpu(F.ctr + pending, 1);
    pending = -1;
    __syncthreads();
    if (t >= F.n_entries) break;
    if (tid == 0) s_ticket = atomicAdd(F.queue, 1);
    const RowEntry e = F.entries[t];
    if (e.ts > 0) {
      const int lg = 31 - __clz(e.ts), team = tid >> lg;
      if (team < e.count) {
        const RowSync sy = F.sync[e.sync + team];
        const RowsSmem& m = M.ts[lg - 5];
        const bool lead = (tid & (e.ts - 1)) == 0;
        unsigned char* sm = smem_raw + team * m.team_bytes;
        rows_tile<T, RB, FWD, false>(B, S, B.items + e.first + team, 0, e.ts, team, m, sm, [&] {
                                       if (lead) s_ok[team] = sy.wait < 0 || flow_wait(F.ctr + sy.wait, sy.target, F.err);
                                       team_sync(e.ts, team);
                                       return s_ok[team] != 0;
                                     });
        // the next tile's bulk copy may land where this one wrote through the generic proxy
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        team_sync(e.ts, team);
        if (lead) {
          // the next tile in this slice sets its own barriers up
          asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(sm)) : "memory");
          asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(sm) + 8) : "memory");
          pending = sy.signal;
        }
      }
    } else if constexpr (sizeof(T) == 8) {
      RowSync sy{-1, 0, -1, 0};
      if (tid < e.count) sy = F.sync[e.sync + tid];
      rows_batch<RB, FWD>(B, S, B.items + e.first, 0, [&] {
        return __syncthreads_and(sy.wait < 0 || flow_wait(F.ctr + sy.wait, sy.target, F.err)) != 0;
      });
      __syncthreads();
      pending = sy.signal;
    }
  }
}

// Right-hand sides per chunk: the registers hold VR x RB sums.  Fewest
// multiplications (chunks x RB), a chunk's re-reading of the tile counted like
// `extra` right-hand sides.
template <typename T>
int choose_rb(int nrhs) {
  const int d64[] = {1, 2, 3, 4, 6, 8}, d32[] = {1, 2, 3, 4, 6, 8, 12, 16};
  const int* v = sizeof(T) == 8 ? d64 : d32;
  const int nv = sizeof(T) == 8 ? 6 : 8, extra = sizeof(T) == 8 ? 1 : 6;
  int best = 1;
  long long cost = -1;
  for (int i = 0; i < nv; ++i) {
    const long long n = (nrhs + v[i] - 1) / v[i], c = n * (v[i] + extra);
    if (cost < 0 || c <= cost) cost = c, best = v[i];
  }
  return best;
}

// calls f(std::integral_constant<int, RB>)
template <typename T, typename F>
void with_rb(int rb, F f) {
  switch (rb) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 12:
      if constexpr (sizeof(T) == 4) f(std::integral_constant<int, 12>{});
      break;
    case 16:
      if constexpr (sizeof(T) == 4) f(std::integral_constant<int, 16>{});
      break;
    default: f(std::integral_constant<int, 8>{}); break;
  }
}

template <typename T>
RowsSmem smem_of(const RowShape& P, int rb, int ts) {
  return rows_smem(P, VecOf<T>::n, rb, ts);
}

void check_smem(size_t bytes) {
  if (bytes > kRowsSmem) throw PecsError(PECS_E_ARG, "front too large for shared memory");
}

template <typename T, int RB, bool FWD, bool ASM>
void launch_level(const RowsDirView& B, const RowSets& S, int n_sets, const RowLevel& L, int max_nrhs,
                  cudaStream_t st) {
  if (L.n_tile + L.n_batch == 0) return;
  const int lg = L.ts == 32 ? 5 : L.ts == 64 ? 6 : L.ts == 128 ? 7 : 8, teams = kRowsThreads / L.ts;
  if (ASM && L.n_tile > 0) {
    AsmRanges A{};
    long long most = 0;
    for (int q = 0; q < n_sets; ++q) {
      A.set[q] = AsmRange{L.col[q], L.n_col[q], L.d[q], L.upd[q], L.n_upd[q]};
      most = std::max(most, (long long)(L.n_col[q] + L.n_upd[q]) * S.set[q].nrhs);
    }
    launch_pdl(k_assemble<T>, dim3((unsigned)((most + 255) / 256), n_sets), 256, 0, st, B, S, A);
  }
  const RowsSmem m = smem_of<T>(L.shape, RB, L.ts);
  check_smem((size_t)m.team_bytes * teams);
  const int tb = (L.n_tile + teams - 1) / teams;
  launch_pdl(k_rows<T, RB, FWD, ASM>, dim3(tb + L.n_batch, (max_nrhs + RB - 1) / RB), kRowsThreads,
             (size_t)m.team_bytes * teams, st, B, S, L.first, L.n_tile, tb, lg, m);
}

void allow_smem(const void* fn) {
  PECS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem));
}

}  // namespace

void RowsSweep::build(const std::vector<const MfFactor*>& factors, int precision, int max_nrhs) {
  prec_ = precision;
  const bool f64 = precision == PECS_PREC_FP64;
  const RowsPlan R = plan_rows(factors, f64 ? 2 : 4, max_nrhs);
  n_nodes_ = (int)R.nodes.size();
  n_sets_ = (int)factors.size();
  stall_node_ = -1;
  for (int g = 0; g < (int)factors[0]->nodes.size() && stall_node_ < 0; ++g)
    if (R.nodes[g].parent < 0 && !factors[0]->nodes[g].children.empty()) stall_node_ = g;
  for (size_t si = 0; si < R.wtotal.size(); ++si) wtotal_[si] = R.wtotal[si], dofs_[si] = factors[si]->n;
  entries_ = R.entries;
  bytes_ = 0;
  rec_.upload(R.rec);
  upd_.upload(R.upd);
  more_.upload(R.more);
  for (int d = 0; d < 2; ++d) {
    const RowsPlan::Dir& H = R.dir[d];
    Dir& D = dir_[d];
    for (const RowLevel& L : H.levels)
      if ((size_t)L.shape.cols * (f64 ? 8 : 4) > kMostColBytes)
        throw PecsError(PECS_E_ARG, "front too large for shared memory");
    if (f64) {
      std::unique_ptr<double[]> v(new double[H.n_values]);
      pack_rows(R, factors, d, v.get());
      D.v64.upload(v.get(), H.n_values);
    } else {
      std::unique_ptr<float[]> v(new float[H.n_values]);
      pack_rows(R, factors, d, v.get());
      D.v32.upload(v.get(), H.n_values);
    }
    bytes_ += H.n_values * (f64 ? 8 : 4);
    D.items.upload(H.items);
    D.src.upload(H.src);
    D.dst.upload(H.dst);
    D.entries.upload(H.entries);
    D.sync.upload(H.sync);
    D.n_entries = (int)H.entries.size();
    D.levels = H.levels;
    std::copy(H.flow_shape, H.flow_shape + 4, D.flow_shape);
  }
  flow_state_.alloc(2 * (size_t)n_nodes_ + 3);
  flow_state_.zero();
  flow_on_ = false;
  ready_rb_ = 0;
  flow_ = FlowLaunch();
}

// The kernels for chunks of RB right-hand sides take their shared memory (only
// these: setting an attribute loads the kernel).
template <typename T, int RB>
void RowsSweep::ready() const {
  if (ready_rb_ == RB) return;
  allow_smem((const void*)k_rows<T, RB, true, false>);
  allow_smem((const void*)k_rows<T, RB, false, false>);
  if constexpr (RB >= kAsmMinRb) allow_smem((const void*)k_rows<T, RB, true, true>);
  ready_rb_ = RB;
}

void RowsSweep::load_kernels(int most_rhs) const {
  auto go = [&](auto tag) {
    using T = decltype(tag);
    for (int n = 1, last = 0; n <= most_rhs; ++n) {
      const int rb = choose_rb<T>(n);
      if (rb != last) with_rb<T>(rb, [&](auto c) { ready<T, decltype(c)::value>(); });
      last = rb;
    }
  };
  if (prec_ == PECS_PREC_FP64)
    go(double{});
  else
    go(float{});
}

// Assembling a level's columns costs a launch, and saves every tile of a node the
// reading of the children's updates.  From five right-hand sides on that always
// paid; for three and four it does at levels of many tiles per node.  us per Poisson
// sweep of 3, never / from 2 / 4 / 8 tiles per node on: 72x72+72x72 cells, k = 2, FP32
// 603 / 486 / 494 / 501; 40x40+40x40, k = 2, FP64 271 / 261 / 261 / 260; 16x16+16x16,
// k = 1, FP64 67.6 / 74.9 / 69.1 / 67.8.
static bool assembles(const RowLevel& L, int max_nrhs) {
  if (L.leaf || L.n_tile == 0) return false;
  return max_nrhs >= kAsmMinRhs || (max_nrhs >= kAsmMinRb && L.n_tile >= kAsmTiles * L.n_node);
}

int RowsSweep::launches_per_solve(int max_nrhs) const {
  if (flow_on_) return 2;
  int n = 0;
  for (int d = 0; d < 2; ++d)
    for (const RowLevel& L : dir_[d].levels) {
      n += L.n_tile + L.n_batch > 0;
      if (d == 0 && assembles(L, max_nrhs)) ++n;
    }
  return n;
}

void RowsSweep::solve(const RowSets& sets, int max_nrhs, cudaStream_t st) const {
  auto go = [&](auto tag) {
    using T = decltype(tag);
    const int rb = choose_rb<T>(max_nrhs);
    with_rb<T>(rb, [&](auto c) {
      constexpr int RB = decltype(c)::value;
      if (flow_on_ && max_nrhs <= RB) {
        solve_flow<T, RB>(sets, st);
        return;
      }
      ready<T, RB>();
      bool room = true;
      for (int q = 0; q < n_sets_; ++q) room = room && sets.set[q].d;
      for (const RowLevel& L : dir_[0].levels) {
        if constexpr (RB >= kAsmMinRb) {
          if (room && assembles(L, max_nrhs)) {
            launch_level<T, RB, true, true>(view(0), sets, n_sets_, L, max_nrhs, st);
            continue;
          }
        }
        launch_level<T, RB, true, false>(view(0), sets, n_sets_, L, max_nrhs, st);
      }
      for (const RowLevel& L : dir_[1].levels)
        launch_level<T, RB, false, false>(view(1), sets, n_sets_, L, max_nrhs, st);
    });
  };
  if (prec_ == PECS_PREC_FP64)
    go(double{});
  else
    go(float{});
}

template <typename T, int RB>
void RowsSweep::solve_flow(const RowSets& sets, cudaStream_t st) const {
  if (flow_.rb != RB) {
    int dev = 0, n_sm = 0;
    PECS_CUDA(cudaGetDevice(&dev));
    PECS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    for (int d = 0; d < 2; ++d) {
      size_t bytes = 0;
      for (int q = 0; q < 4; ++q)
        bytes = std::max(bytes, (size_t)smem_of<T>(dir_[d].flow_shape[q], RB, 32 << q).team_bytes *
                                    (kRowsThreads >> (5 + q)));
      check_smem(bytes);
      const void* fn = d == 0 ? (const void*)k_rows_flow<T, RB, true> : (const void*)k_rows_flow<T, RB, false>;
      allow_smem(fn);
      int per_sm = 0;
      PECS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kRowsThreads, bytes));
      flow_.bytes[d] = bytes;
      flow_.grid[d] = std::max(1, std::min(dir_[d].n_entries, std::max(1, per_sm) * n_sm));
    }
    flow_.rb = RB;
  }
  int* base = flow_state_.p;
  for (int d = 0; d < 2; ++d) {
    const RowsFlowView F{dir_[d].entries.p, dir_[d].sync.p, base + (size_t)d * n_nodes_,
                         base + (size_t)(1 - d) * n_nodes_, n_nodes_, base + 2 * (size_t)n_nodes_ + d,
                         base + 2 * (size_t)n_nodes_ + 1 - d, base + 2 * (size_t)n_nodes_ + 2, dir_[d].n_entries};
    RowsSmem4 m;
    for (int q = 0; q < 4; ++q) m.ts[q] = smem_of<T>(dir_[d].flow_shape[q], RB, 32 << q);
    if (d == 0)
      k_rows_flow<T, RB, true><<<flow_.grid[d], kRowsThreads, flow_.bytes[d], st>>>(view(d), sets, F, m);
    else
      k_rows_flow<T, RB, false><<<flow_.grid[d], kRowsThreads, flow_.bytes[d], st>>>(view(d), sets, F, m);
    PECS_CUDA(cudaGetLastError());
  }
}

void RowsSweep::tune_flow(const RowSets& sets, int max_nrhs, cudaStream_t st, int mode, int reps) {
  flow_on_ = false;
  const int rb = prec_ == PECS_PREC_FP64 ? choose_rb<double>(max_nrhs) : choose_rb<float>(max_nrhs);
  if (mode < 0 || max_nrhs > rb || dir_[0].n_entries == 0) return;
  if (mode > 0) {
    flow_on_ = true;
    return;
  }
  cudaEvent_t e0, e1;
  PECS_CUDA(cudaEventCreate(&e0));
  PECS_CUDA(cudaEventCreate(&e1));
  auto time = [&](bool flow) {
    flow_on_ = flow;
    solve(sets, max_nrhs, st);  // warm-up
    float best = 1e30f;
    for (int r = 0; r < reps; ++r) {
      PECS_CUDA(cudaEventRecord(e0, st));
      solve(sets, max_nrhs, st);
      PECS_CUDA(cudaEventRecord(e1, st));
      PECS_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      PECS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best = std::min(best, ms);
    }
    return best;
  };
  const float lev = time(false), flo = time(true);
  if (flow_error(false) != 0) throw PecsError(PECS_E_CUDA, "flow sweep: a wait for a node's inputs ran out");
  if (std::getenv("PECS_TUNE_LOG"))
    std::fprintf(stderr, "rows flow: %.4f ms (levels %.4f ms)\n", flo, lev);
  flow_on_ = flo < lev;
  tuned_ms_ = std::min(flo, lev);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
}

int RowsSweep::flow_error(bool clear) const {
  if (flow_state_.n == 0) return 0;
  int e = 0;
  int* p = flow_state_.p + 2 * (size_t)n_nodes_ + 2;
  PECS_CUDA(cudaMemcpy(&e, p, sizeof(int), cudaMemcpyDeviceToHost));
  if (clear) PECS_CUDA(cudaMemset(p, 0, sizeof(int)));
  return e;
}

void RowsSweep::debug_arm_flow_stall() const {
  if (flow_state_.n == 0 || stall_node_ < 0) throw PecsError(PECS_E_STATE, "no flow sweep to stall");
  PECS_CUDA(cudaDeviceSynchronize());
  const int v = -(1 << 30);
  PECS_CUDA(cudaMemcpy(flow_state_.p + stall_node_, &v, sizeof(int), cudaMemcpyHostToDevice));
}

}  // namespace pecs
