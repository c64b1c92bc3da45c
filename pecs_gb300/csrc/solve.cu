// Multifrontal solve kernels of the panel banks and their host-side plans
// (solve.cuh): one launch per tree level, or one persistent dataflow launch per
// direction (flow sweeps) over the same items.  Banks with few right-hand sides
// per set: rows.cu.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <numeric>
#include <type_traits>

#include "bulk_copy.cuh"
#include "panel_plan.hpp"
#include "solve.cuh"
#include "sweep_sync.cuh"

namespace pecs {

namespace {

// ---- panel path --------------------------------------------------------------
constexpr size_t kPanelSmem = 160 * 1024;
constexpr size_t kTileSmem = 200 * 1024;   // most of a level launch
constexpr size_t kTileOnce = 100 * 1024;   // columns staged in one go up to here, else in two buffers
constexpr size_t kTileBuffer = 48 * 1024;  // ... of this size
constexpr size_t kWarpSmem = 48 * 1024;  // leaf levels: shared memory per CTA

// RPL consecutive values of one interleaved row (offset a multiple of RPL),
// double or float storage, registers of type VR (the storage type converts
// only where the two differ -- on GB300 every FP64 operation, conversions
// included, runs on the narrow FP64 unit, so the FP32 path keeps none).
template <int RPL, typename VR>
__device__ __forceinline__ void ld_rhs(const double* p, VR (&v)[RPL]) {
  if constexpr (RPL == 1) {
    v[0] = (VR)p[0];
  } else {
#pragma unroll
    for (int q = 0; q < RPL / 2; ++q) {
      const double2 t = reinterpret_cast<const double2*>(p)[q];
      v[2 * q] = (VR)t.x;
      v[2 * q + 1] = (VR)t.y;
    }
  }
}

template <int RPL, typename VR>
__device__ __forceinline__ void ld_rhs(const float* p, VR (&v)[RPL]) {
  if constexpr (RPL == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = (VR)t.x, v[1] = (VR)t.y, v[2] = (VR)t.z, v[3] = (VR)t.w;
  } else if constexpr (RPL == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = (VR)t.x, v[1] = (VR)t.y;
  } else {
    v[0] = (VR)p[0];
  }
}

template <int RPL, typename VR>
__device__ __forceinline__ void st_rhs(double* p, const VR (&v)[RPL]) {
  if constexpr (RPL == 1) {
    p[0] = (double)v[0];
  } else {
#pragma unroll
    for (int q = 0; q < RPL / 2; ++q)
      reinterpret_cast<double2*>(p)[q] = make_double2((double)v[2 * q], (double)v[2 * q + 1]);
  }
}

template <int RPL, typename VR>
__device__ __forceinline__ void st_rhs(float* p, const VR (&v)[RPL]) {
  if constexpr (RPL == 4) {
    *reinterpret_cast<float4*>(p) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  } else if constexpr (RPL == 2) {
    *reinterpret_cast<float2*>(p) = make_float2((float)v[0], (float)v[1]);
  } else {
    p[0] = (float)v[0];
  }
}

// n consecutive shared-memory values (16-byte aligned when n * sizeof(T) >= 16).
template <typename T, int N>
__device__ __forceinline__ void lds(const T* p, T (&v)[N]) {
  if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
      const float4 t = reinterpret_cast<const float4*>(p)[q];
      v[4 * q] = t.x;
      v[4 * q + 1] = t.y;
      v[4 * q + 2] = t.z;
      v[4 * q + 3] = t.w;
    }
  } else if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
      const double2 t = reinterpret_cast<const double2*>(p)[q];
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = p[q];
  }
}

template <typename T, int N, typename VR>
__device__ __forceinline__ void sts(T* p, const VR (&v)[N]) {
  if constexpr (sizeof(T) == 4 && N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N / 4; ++q)
      reinterpret_cast<float4*>(p)[q] =
          make_float4((float)v[4 * q], (float)v[4 * q + 1], (float)v[4 * q + 2], (float)v[4 * q + 3]);
  } else if constexpr (sizeof(T) == 8 && N % 2 == 0) {
#pragma unroll
    for (int q = 0; q < N / 2; ++q)
      reinterpret_cast<double2*>(p)[q] = make_double2((double)v[2 * q], (double)v[2 * q + 1]);
  } else {
#pragma unroll
    for (int q = 0; q < N; ++q) p[q] = (T)v[q];
  }
}

// Flow sweeps: one item = rows [r0, r1) of one node's block (Gf for the forward sweep, Hb
// for the backward sweep; both column-major with leading dimension = row
// count), applied to the right-hand-side chunk blockIdx.y (32 * RPL RHS).
// Rows are tiled ri at a time (ri in {4, 8, 16, 32}): warp (g, part) owns rows
// 4g..4g+3 of the tile and the chunk columns k = part (mod 32 / ri); partial
// sums of the column parts are added through shared memory.
//
// The kernel is bound by memory latency, so each column chunk is staged with
// asynchronous copies (cp.async: global -> shared without registers): the
// block tile, the chunk's right-hand-side rows (lanes over right-hand sides,
// coalesced) and, in the forward sweep, the children's update rows that land
// on the chunk's columns are all in flight at once, followed by one wait.
// The item record carries everything about its node (sizes, offsets, the
// node's child-map range), and the node's index metadata is staged once, so
// the chain of dependent loads per item is: record -> metadata -> copies.
// nbuf = 2: the staging buffers are doubled and chunk c + 1 is copied while
// chunk c is multiplied (items with more than one chunk).
template <typename T>
__host__ __device__ constexpr size_t panel_smem_bytes(int ds_rows, int rc, int kc, int ri_max,
                                                      int sc_rows, int meta_ints, int nbuf = 1) {
  return (size_t)nbuf * ((size_t)ds_rows * rc + (size_t)kc * ri_max + (size_t)sc_rows * rc) * sizeof(T) +
         (size_t)meta_ints * sizeof(int);
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"(BYTES)
                 : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}



// RPL consecutive T of one interleaved row -> shared memory (16-byte pieces
// where the row segment allows; zero fill for lanes past the last RHS)
template <typename T, int RPL>
__device__ __forceinline__ void stage_row(T* dst, const T* src, bool ok) {
  constexpr int BYTES = RPL * (int)sizeof(T);
  if (!ok) {
#pragma unroll
    for (int q = 0; q < RPL; ++q) dst[q] = T(0);
    return;
  }
  if constexpr (BYTES <= 16) {
    cp_async<BYTES>(dst, src);
  } else {
#pragma unroll
    for (int o = 0; o < BYTES / 16; ++o) cp_async<16>(reinterpret_cast<char*>(dst) + 16 * o,
                                                      reinterpret_cast<const char*>(src) + 16 * o);
  }
}

template <typename T>
__device__ __forceinline__ T quiet_nan() {
  if constexpr (sizeof(T) == 4)
    return __int_as_float(0x7fc00000);
  else
    return __longlong_as_double(0x7ff8000000000000ll);
}

// Staging shape of a panel launch (its shared-memory layout): staged block
// columns per chunk, staged right-hand-side rows, the tallest row tile, staged
// child-update rows per chunk, and the index metadata sizes.
struct PanelShape {
  int kc_cap, ds_rows, ri_max, sc_rows, max_s, max_f, cm_cap;
  int nbuf;  // staging buffers (2: the next chunk is copied during this one's products)
};

// One panel item (rows [r0, r1) of one node) applied to the right-hand-side
// chunk starting at rc0 (chunk index `chunk`).  wait_inputs() is called by
// every thread once the block tile's copies are in flight and before any
// vector is read; it returns false when the inputs could not be waited for,
// and the item then writes NaN (the solve's results are flagged non-finite).
template <typename T, int RPL, bool FWD, typename SVT, typename Wait>
__device__ __forceinline__ void panel_tile(const BankView& B, const SVT& S, const PanelItem& I, int rc0,
                                           const PanelShape& P, unsigned char* smem_raw, Wait wait_inputs) {
  constexpr int RC = 32 * RPL;
  constexpr int NW = kSolveThreads / 32;
  const int r0 = I.a.y, r1 = I.a.z, ri = I.a.w;
  const int s = I.b.x, m = I.b.y, f = s + m, w_off = I.b.w;
  const auto st = S.set[I.b.z];
  // the sweep vectors have the block's type (FP64 banks: double, FP32: float)
  static_assert(std::is_same<typename std::remove_cv<typename std::remove_pointer<decltype(st.y)>::type>::type,
                             T>::value, "sweep vectors must have the block's type");
  const int R = st.nrhs;
  if (rc0 >= R) return;
  const int max_s = P.max_s, max_f = P.max_f, cm_cap = P.cm_cap, ri_max = P.ri_max;
  const int ds_rows = P.ds_rows, sc_rows = P.sc_rows;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rl = rc0 + lane * RPL;  // first right-hand side of this lane
  const bool lane_ok = rl < R;      // R is a multiple of RPL
  const int K = FWD ? s : f;
  const int ld = FWD ? f : s;
  const T* M = static_cast<const T*>(FWD ? B.G : B.H) + (((long long)I.c.y << 32) | (unsigned)I.c.x);
  const int nrows = r1 - r0;
  const int wpr = 32 / ri;  // warps sharing a row group (column parts)
  const int g = warp / wpr, part = warp % wpr;
  const int kc_cap = min(I.kc, P.kc_cap);
  bool bad = false;
  const int nbuf = P.nbuf;
  // staging buffers, nbuf of each: Ds [ds_rows][RC] (nbuf * ds_rows >= 32 when
  // ri < 32: the column-part reduction reuses them), Gs [kc_cap][ri], Sc
  // [sc_rows][RC] child-update rows of a chunk
  T* Ds0 = reinterpret_cast<T*>(smem_raw);
  T* Gs0 = Ds0 + (size_t)nbuf * ds_rows * RC;
  T* Sc0 = Gs0 + (size_t)nbuf * P.kc_cap * ri_max;
  // index metadata of the whole node:
  //   forward:  src_s[s] = own rows; cp_s[f + 1] = child-update ranges per front
  //             position (relative to the node's first entry); cm_s = child rows
  //   backward: src_s[f] = own rows (y) / ~update rows (x)
  int* src_s = reinterpret_cast<int*>(Sc0 + (size_t)nbuf * sc_rows * RC);
  int* cp_s = src_s + (FWD ? max_s : max_f);
  int* cm_s = cp_s + max_f + 1;
  const int cbase = I.d.y, ncm = I.d.z;
  {
    const int* own = B.own_idx + I.c.z;
    if (FWD) {
      const int* cptr = B.cmap_ptr + I.d.x;
      for (int p = tid; p < s; p += kSolveThreads) src_s[p] = own[p];
      for (int p = tid; p <= f; p += kSolveThreads) cp_s[p] = cptr[p] - cbase;
      const int n = min(ncm, cm_cap);
      for (int c = tid; c < n; c += kSolveThreads) cm_s[c] = B.cmap_idx[cbase + c];
    } else {
      const int* upd = B.upd_idx + I.c.w;
      for (int p = tid; p < f; p += kSolveThreads) src_s[p] = p < s ? own[p] : ~upd[p - s];
    }
  }
  __syncthreads();
  T acc[4][RPL];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < RPL; ++q) acc[i][q] = T(0);
  // (A) asynchronous copies of one chunk into buffer b: block tile (read-only,
  // may start before the inputs are waited for), then right-hand-side rows and
  // child-update rows
  const int ri_log = 31 - __clz(ri);  // ri is a power of two
  auto stage_block = [&](int k0, int b) {
    const int kc = min(kc_cap, K - k0);
    T* Gs = Gs0 + (size_t)b * P.kc_cap * ri_max;
    const T* Mk = M + (size_t)k0 * ld + r0;
    for (int idx = tid; idx < kc * ri; idx += kSolveThreads) {
      const int k = idx >> ri_log, i = idx & (ri - 1);
      if (i < nrows)
        cp_async<sizeof(T)>(Gs + idx, Mk + (size_t)k * ld + i);
      else
        Gs[idx] = T(0);
    }
  };
  auto stage_rows = [&](int k0, int b) {
    const int kc = min(kc_cap, K - k0);
    T* Ds = Ds0 + (size_t)b * ds_rows * RC;
    for (int k = warp; k < kc; k += NW) {
      const int sr = src_s[k0 + k];
      const T* src = FWD ? st.b + (size_t)sr * R
                         : (sr >= 0 ? st.y + (size_t)sr * R : st.x + (size_t)(~sr) * R);
      stage_row<T, RPL>(Ds + (size_t)k * RC + lane * RPL, src + rl, lane_ok);
    }
    if (FWD) {
      T* Sc = Sc0 + (size_t)b * sc_rows * RC;
      const int cb = cp_s[k0];
      const int ne = cp_s[k0 + kc] - cb;  // <= sc_rows (plan)
      for (int e = warp; e < ne; e += NW) {
        const int c = cb + e;
        const int wi = c < cm_cap ? cm_s[c] : B.cmap_idx[cbase + c];
        stage_row<T, RPL>(Sc + (size_t)e * RC + lane * RPL, st.w + (size_t)wi * R + rl, lane_ok);
      }
    }
    cp_async_commit();
  };
  if (K > 0) stage_block(0, 0);
  bad = !wait_inputs();  // vectors below are written by earlier work
  if (K > 0) stage_rows(0, 0);
  int chunk_i = 0;
  for (int k0 = 0; k0 < K; k0 += kc_cap, ++chunk_i) {
    const int kc = min(kc_cap, K - k0);
    const int b = nbuf == 2 ? (chunk_i & 1) : 0;
    const bool more = k0 + kc_cap < K;
    if (more && nbuf == 2) {
      stage_block(k0 + kc_cap, b ^ 1);
      stage_rows(k0 + kc_cap, b ^ 1);
      cp_async_wait_group<1>();
    } else {
      cp_async_wait_group<0>();
    }
    __syncthreads();
    T* Ds = Ds0 + (size_t)b * ds_rows * RC;
    const T* Gs = Gs0 + (size_t)b * P.kc_cap * ri_max;
    if (FWD) {
      // (B) subtract the children's updates from the staged right-hand sides
      const T* Sc = Sc0 + (size_t)b * sc_rows * RC;
      const int cb = cp_s[k0];
      for (int k = warp; k < kc; k += NW) {
        const int p = k0 + k;
        const int e0 = cp_s[p] - cb, e1 = cp_s[p + 1] - cb;
        if (e1 > e0) {
          T v[RPL], u[RPL];
          lds<T, RPL>(Ds + (size_t)k * RC + lane * RPL, v);
          for (int e = e0; e < e1; ++e) {
            lds<T, RPL>(Sc + (size_t)e * RC + lane * RPL, u);
#pragma unroll
            for (int q = 0; q < RPL; ++q) v[q] -= u[q];
          }
          sts<T, RPL>(Ds + (size_t)k * RC + lane * RPL, v);
        }
      }
      __syncthreads();
    }
    // (C) register tiles
    const T* Gp = Gs + 4 * g;
    const T* Dp = Ds + lane * RPL;
#pragma unroll 4
    for (int k = part; k < kc; k += wpr) {
      T gv[4], dv[RPL];
      lds<T, 4>(Gp + k * ri, gv);
      lds<T, RPL>(Dp + (size_t)k * RC, dv);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < RPL; ++q) acc[i][q] += gv[i] * dv[q];
    }
    __syncthreads();  // buffer b is restaged two chunks later (one, single-buffered)
    if (more && nbuf == 1) {
      stage_block(k0 + kc_cap, 0);
      stage_rows(k0 + kc_cap, 0);
    }
  }
  // row i of the item -> its destination
  auto emit = [&](int i, T (&v)[RPL]) {
    const int row = r0 + i;
    if (bad) {
#pragma unroll
      for (int q = 0; q < RPL; ++q) v[q] = quiet_nan<T>();
    }
    if (FWD) {
      if (row < s) {
        st_rhs<RPL>(st.y + (size_t)src_s[row] * R + rl, v);
      } else {
        for (int c = cp_s[row]; c < cp_s[row + 1]; ++c) {
          const int wi = c < cm_cap ? cm_s[c] : B.cmap_idx[cbase + c];
          T u[RPL];
          ld_rhs<RPL>(st.w + (size_t)wi * R + rl, u);
#pragma unroll
          for (int q = 0; q < RPL; ++q) v[q] += u[q];
        }
        st_rhs<RPL>(st.w + (size_t)(w_off + row - s) * R + rl, v);
      }
    } else {
      st_rhs<RPL>(st.x + (size_t)src_s[row] * R + rl, v);
    }
  };
  if (wpr == 1) {
    if (lane_ok) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * g + i < nrows) emit(4 * g + i, acc[i]);
    }
  } else {
    T* red = Ds0;  // [wpr][ri][RC] = 32 * RC values
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < RPL; ++q)
        red[((size_t)part * ri + 4 * g + i) * RC + lane * RPL + q] = acc[i][q];
    __syncthreads();
    if (lane_ok) {
      for (int i = warp; i < nrows; i += NW) {
        T v[RPL];
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          T t = T(0);
          for (int p = 0; p < wpr; ++p) t += red[((size_t)p * ri + i) * RC + lane * RPL + q];
          v[q] = t;
        }
        emit(i, v);
      }
    }
  }
}

// ---- level sweeps --------------------------------------------------------------
// A tile applies up to 32 rows of a node's block to a chunk of 32 * NW right-hand
// sides.  A warp holds the sums of all of the tile's rows for 32 of them (lanes 4 x 8:
// pad / 4 rows by 4 right-hand sides each); the warps left over split the columns
// and add their sums through shared memory.  What bounds a level is latency -- it
// has 1 to 10 MB of values and a few of arithmetic per multiprocessor -- so a
// tile needs one round trip for what is constant (record, then values and index list
// by bulk copies, under the previous level's tail) and one for the vectors' rows.
// Forward, the nodes' columns and pass-through sums are formed once by k_panel_assemble
// in a launch before (into x, which the backward sweep overwrites): in each tile of
// a node that was 4 to 11 times the reading, and half of the shared memory.
// 64x64+64x64 cells, 64 instances, FP32, us per carrier sweep of 128 / Poisson sweep of
// 64 right-hand sides: 510 / 188 with the columns assembled in every tile and the blocks
// read column-major (4-byte copies), 346 / 115 with both done once, 337 / 110 with packed
// multiply-adds and fewer instructions in the assembly.  Tried without gain: 8 x 8
// sums per thread (343 / 110), four smaller buffers (339 to 367), pass-through rows
// loaded into the sums (366 / 129).  The multiply-adds alone are 65 / 13.
struct TileShape {
  int kc, lg_nw;          // staged columns; log2 of 32-right-hand-side groups per CTA
  unsigned a, b, p;       // shared-memory offsets: values, vector rows, pass-through rows
  unsigned a_buf, b_buf;  // one buffer of values, of rows
};

// MR x 4 sums of one thread.  FP32: two rows per register pair, so that one packed
// instruction (fma.rn.f32x2, each half rounded as fmaf) does two of them.
template <typename T, int MR>
struct TileAcc {
  T v_[MR][4];
  __device__ __forceinline__ void set(int i, const T (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) v_[i][q] = v[q];
  }
  __device__ __forceinline__ void get(int i, T (&v)[4]) const {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = v_[i][q];
  }
  __device__ __forceinline__ void fma(const T (&a)[MR], const T (&d)[4]) {
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) v_[i][q] += a[i] * d[q];
  }
};
template <int MR>
struct TileAcc<float, MR> {
  unsigned long long v_[MR / 2][4];
  static __device__ __forceinline__ unsigned long long pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
  }
  static __device__ __forceinline__ float2 unpack(unsigned long long p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
  }
  __device__ __forceinline__ void set(int i, const float (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float2 t = i % 2 ? unpack(v_[i / 2][q]) : make_float2(0.f, 0.f);
      (i % 2 ? t.y : t.x) = v[q];
      v_[i / 2][q] = pack(t.x, t.y);
    }
  }
  __device__ __forceinline__ void get(int i, float (&v)[4]) const {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 t = unpack(v_[i / 2][q]);
      v[q] = i % 2 ? t.y : t.x;
    }
  }
  __device__ __forceinline__ void fma(const float (&a)[MR], const float (&d)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned long long dd = pack(d[q], d[q]);
#pragma unroll
      for (int i = 0; i < MR / 2; ++i)
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v_[i][q]) : "l"(pack(a[2 * i], a[2 * i + 1])), "l"(dd));
    }
  }
};

// 4 right-hand sides from column c of a row (c a multiple of 4; R: their number)
template <typename T>
__device__ __forceinline__ void st4(T* row, int c, int R, const T (&v)[4]) {
  if (R % 4 == 0) {
    if (c < R) sts<T, 4>(row + c, v);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q < R) row[c + q] = v[q];
  }
}

template <typename T, int MR, bool FWD, typename SV>
__device__ __forceinline__ void tile_apply(const TilesView& B, const SV& st, const PanelTile& I, const TileShape& P,
                                           int c0, unsigned char* smem) {
  constexpr int BM = 4 * MR;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x;
  const int lg = P.lg_nw, nw = warp & ((1 << lg) - 1), kg = warp >> lg, KG = nthr >> (5 + lg);
  const int BN = 32 << lg, R = st.nrhs, K = I.cols, kc_max = P.kc, K4 = (K + 3) & ~3;
  const unsigned bar = smem_u32(smem);
  const T* val = static_cast<const T*>(B.val) + (I.off - B.val0);
  const int* idx = reinterpret_cast<const int*>(smem + 16);
  if (tid == 0) {
    bar_init(bar);
    bar_init(bar + 8);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    const unsigned nv = min(K, kc_max) * BM * (unsigned)sizeof(T), ni = (K4 + BM) * 4u;
    bar_expect(bar, nv + ni);
    bulk_copy(bar + 16, B.idx + I.idx, ni, bar);
    bulk_copy(bar + P.a, val, nv, bar);
    if (K > kc_max)
      bulk_load(bar + P.a + P.a_buf, val + (size_t)kc_max * BM, min(K - kc_max, kc_max) * BM * (unsigned)sizeof(T), bar + 8);
  }
  __syncthreads();
  bool ok = bar_wait(bar, 0);
  pdl_wait();  // vectors below are written by earlier work
  // n rows given by their indices -> dst [n][BN], zeros past the last right-hand side
  auto stage = [&](T* dst, const int* rows, int n, auto row_of) {
    constexpr int V = 16 / (int)sizeof(T);
    if (R % V == 0) {
      const int lp = lg + (sizeof(T) == 4 ? 3 : 4);  // log2 of 16-byte pieces per row
      for (int e = tid; e < n << lp; e += nthr) {
        const int c = c0 + (e & ((1 << lp) - 1)) * V;
        if (c < R)
          cp_async<16>(dst + (size_t)e * V, row_of(rows[e >> lp]) + c);
        else
          *reinterpret_cast<float4*>(dst + (size_t)e * V) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
      for (int e = tid; e < n << (lg + 5); e += nthr) {
        const int c = c0 + (e & (BN - 1));
        if (c < R)
          cp_async<sizeof(T)>(dst + e, row_of(rows[e >> (lg + 5)]) + c);
        else
          dst[e] = T(0);
      }
    }
  };
  auto stage_columns = [&](int k0, int b) {
    T* dst = reinterpret_cast<T*>(smem + P.b + b * P.b_buf);
    const int n = min(kc_max, K - k0);
    if constexpr (FWD) {
      const T* src = I.leaf ? st.b : st.x;
      stage(dst, idx + k0, n, [&](int z) { return src + (size_t)z * R; });
    } else {
      stage(dst, idx + k0, n,
            [&](int z) { return z >= 0 ? static_cast<const T*>(st.y) + (size_t)z * R : static_cast<const T*>(st.x) + (size_t)(~z) * R; });
    }
  };
  stage_columns(0, 0);
  T* Ps = reinterpret_cast<T*>(smem + P.p);
  if (FWD && I.npt > 0)
    stage(Ps, idx + K4 + I.rows - I.npt, I.npt, [&](int z) { return static_cast<const T*>(st.w) + (size_t)(~z) * R; });
  cp_async_commit();
  if (K > kc_max) stage_columns(kc_max, 1);
  cp_async_commit();
  const int rg = lane >> 3, cg = lane & 7;
  TileAcc<T, MR> acc;
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    const T zero[4] = {T(0), T(0), T(0), T(0)};
    acc.set(i, zero);
  }
  for (int k0 = 0, c = 0;; ++c) {
    const int b = c & 1, kc = min(kc_max, K - k0);
    cp_async_wait_group<1>();  // chunk c; the next one's copies may be in flight
    if (c > 0) ok = bar_wait(bar + 8 * b, (c >> 1) & 1) && ok;
    __syncthreads();
    const T* a = reinterpret_cast<const T*>(smem + P.a + b * P.a_buf) + kg * BM + rg * MR;
    const T* d = reinterpret_cast<const T*>(smem + P.b + b * P.b_buf) + kg * BN + nw * 32 + cg * 4;
#pragma unroll 4
    for (int k = kg; k < kc; k += KG) {
      T av[MR], dv[4];
      lds<T, MR>(a, av);
      lds<T, 4>(d, dv);
      acc.fma(av, dv);
      a += KG * BM;
      d += KG * BN;
    }
    k0 += kc;
    if (k0 >= K) break;
    __syncthreads();  // buffer b is free
    const int next = k0 + min(kc_max, K - k0);
    if (next < K) {
      if (tid == 0)
        bulk_load(bar + P.a + b * P.a_buf, val + (size_t)next * BM, min(K - next, kc_max) * BM * (unsigned)sizeof(T), bar + 8 * b);
      stage_columns(next, b);
    }
    cp_async_commit();
  }
  pdl_trigger();
  // row totals -> destination
  auto emit = [&](int row, int c, T (&v)[4]) {
    const int z = idx[K4 + row];
    if (FWD && row >= I.rows - I.npt) {
      T u[4];
      lds<T, 4>(Ps + (size_t)(row - (I.rows - I.npt)) * BN + c, u);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] += u[q];
    }
    if (!ok) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = quiet_nan<T>();
    }
    T* dst = FWD ? (z >= 0 ? st.y + (size_t)z * R : st.w + (size_t)(~z) * R) : st.x + (size_t)z * R;
    st4(dst, c0 + c, R, v);
  };
  if (KG == 1) {
#pragma unroll
    for (int i = 0; i < MR; ++i) {
      T v[4];
      acc.get(i, v);
      if (rg * MR + i < I.rows) emit(rg * MR + i, nw * 32 + cg * 4, v);
    }
    return;
  }
  __syncthreads();  // the partial sums overlay the values and rows
  T* red = reinterpret_cast<T*>(smem + P.a);  // [KG][BM][BN]
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    T v[4];
    acc.get(i, v);
    sts<T, 4>(red + (size_t)(kg * BM + rg * MR + i) * BN + nw * 32 + cg * 4, v);
  }
  __syncthreads();
  for (int e = tid; e < I.rows << (lg + 3); e += nthr) {
    const int row = e >> (lg + 3), c = (e & ((8 << lg) - 1)) * 4;
    T v[4] = {T(0), T(0), T(0), T(0)};
    for (int g = 0; g < KG; ++g) {
      T u[4];
      lds<T, 4>(red + (size_t)(g * BM + row) * BN + c, u);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] += u[q];
    }
    emit(row, c, v);
  }
}

template <typename T, bool FWD, typename SVT>
__global__ void __launch_bounds__(kSolveThreads)
    k_panel_tiles(TilesView B, SVT S, int first, TileShape P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PanelTile I = B.tiles[first + blockIdx.x];
  const auto& st = S.set[I.set];
  const int c0 = (int)blockIdx.y * (32 << P.lg_nw);
  if (c0 >= st.nrhs) return;
  if constexpr (sizeof(T) == 8)
    tile_apply<T, 1, FWD>(B, st, I, P, c0, smem_raw);
  else if (I.pad == 32)
    tile_apply<T, 8, FWD>(B, st, I, P, c0, smem_raw);
  else if (I.pad == 16)
    tile_apply<T, 4, FWD>(B, st, I, P, c0, smem_raw);
  else
    tile_apply<T, 2, FWD>(B, st, I, P, c0, smem_raw);
}

// Forward, before a level's tiles: its nodes' columns, b minus the children's updates,
// into x, and the pass-through sums into their update slots.  V right-hand sides of a
// front position per thread.
struct AsmSets {
  int rec[kMaxSets], n[kMaxSets];
};

template <typename T, int V, typename SVT>
__global__ void __launch_bounds__(kSolveThreads) k_panel_assemble(TilesView B, SVT S, AsmSets A, int lg) {
  // 2^lg threads share a position
  const auto& st = S.set[blockIdx.y];
  const int R = st.nrhs;
  const unsigned e = blockIdx.x * (unsigned)kSolveThreads + threadIdx.x;
  const int p = (int)(e >> lg);
  const bool in = p < A.n[blockIdx.y];
  int4 q0 = make_int4(0, -1, -1, -1), q1 = make_int4(-1, -1, -1, -1);
  if (in) {
    const int4* rec = reinterpret_cast<const int4*>(B.rec + A.rec[blockIdx.y] + p);
    q0 = rec[0];
    q1 = rec[1];
  }
  pdl_trigger();
  pdl_wait();
  if (!in) return;
  for (int r = (int)(e & ((1u << lg) - 1)) * V; r < R; r += V << lg) {
    const T* w = st.w + r;
    T v[V], u[4][V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      v[i] = T(0);
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j][i] = T(0);
    }
    if (q0.x >= 0) ld_rhs<V>(st.b + (size_t)q0.x * R + r, v);
    if (q0.y >= 0) ld_rhs<V>(w + (size_t)q0.y * R, u[0]);
    if (q0.z >= 0) ld_rhs<V>(w + (size_t)q0.z * R, u[1]);
    if (q0.w >= 0) ld_rhs<V>(w + (size_t)q0.w * R, u[2]);
    if (q1.x >= 0) ld_rhs<V>(w + (size_t)q1.x * R, u[3]);
    const T sign = q0.x >= 0 ? T(-1) : T(1);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] += sign * u[j][i];
    auto add = [&](int slot) {
      T t[V];
      ld_rhs<V>(w + (size_t)slot * R, t);
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] += sign * t[i];
    };
    if (q1.y >= 0) {  // few positions have so many children
      add(q1.y);
      if (q1.z >= 0) add(q1.z);
      if (q1.w >= 0) add(q1.w);
      if (q1.w < -1) {
        const int* m = B.more + (-2 - q1.w);
        for (int j = 1; j <= m[0]; ++j) add(m[j]);
      }
    }
    st_rhs<V>(q0.x >= 0 ? st.x + (size_t)q0.x * R + r : st.w + (size_t)(~q0.x) * R + r, v);
  }
}

// Leaf levels: a warp per node (all of its rows) and right-hand-side chunk,
// eight independent nodes per CTA and no CTA barrier.  A level qualifies when
// its nodes are small (at most kWarpMaxK columns and kWarpMaxRows rows) and,
// in the forward sweep, have no children (so the staged right-hand sides need
// no update subtraction and the outputs no pass-through sums).  The warp
// stages its node's whole block and right-hand-side rows with cp.async.
constexpr int kWarpMaxK = 64;
constexpr int kWarpMaxRows = 64;
constexpr int kWarpNodesPerCta = kSolveThreads / 32;

template <typename T>
__host__ __device__ constexpr size_t panel_warp_bytes(int max_k, int rows_pad, int rc) {
  // rounded to 16 bytes: every warp's slice starts 16-byte aligned
  return ((((size_t)max_k * rc + (size_t)max_k * rows_pad) * sizeof(T) + (size_t)max_k * sizeof(int)) +
          15) & ~(size_t)15;
}

// One leaf-level node applied by one warp to the right-hand-side chunk at rc0;
// `base` is the warp's shared-memory slice.  wait_inputs() (every lane) is
// called once the block's copies are in flight and before any vector is read;
// false: the inputs could not be waited for and the node writes NaN.  main_done() is
// called once the node no longer reads its inputs.
template <typename T, int RPL, bool FWD, typename SVT, typename Wait, typename Done>
__device__ __forceinline__ void panel_warp_node(const BankView& B, const SVT& S, const PanelItem& I, int rc0,
                                                int max_k, int rows_pad, unsigned char* base, Wait wait_inputs,
                                                Done main_done) {
  constexpr int RC = 32 * RPL;
  const int lane = threadIdx.x & 31;
  const int s = I.b.x, m = I.b.y, f = s + m, w_off = I.b.w;
  const auto st = S.set[I.b.z];
  const int R = st.nrhs;
  if (rc0 >= R) return;
  const int rl = rc0 + lane * RPL;
  const bool lane_ok = rl < R;
  const int K = FWD ? s : f;
  const int rows = FWD ? f : s;  // = the leading dimension of the block
  const T* M = static_cast<const T*>(FWD ? B.G : B.H) + (((long long)I.c.y << 32) | (unsigned)I.c.x);
  T* Ds = reinterpret_cast<T*>(base);        // [max_k][RC]
  T* Gs = Ds + (size_t)max_k * RC;           // [max_k][rows_pad]
  int* src_s = reinterpret_cast<int*>(Gs + (size_t)max_k * rows_pad);  // [max_k]
  {
    const int* own = B.own_idx + I.c.z;
    const int* upd = B.upd_idx + I.c.w;
    for (int p = lane; p < K; p += 32) src_s[p] = FWD ? own[p] : (p < s ? own[p] : ~upd[p - s]);
  }
  for (int e = lane; e < K * rows_pad; e += 32) {
    const int k = e / rows_pad, r = e - k * rows_pad;
    if (r < rows)
      cp_async<sizeof(T)>(Gs + e, M + (size_t)k * rows + r);
    else
      Gs[e] = T(0);
  }
  __syncwarp();
  const bool bad = !wait_inputs();  // vectors below are written by earlier work
  for (int k = 0; k < K; ++k) {
    const int sr = src_s[k];
    const T* src = FWD ? st.b + (size_t)sr * R
                       : (sr >= 0 ? st.y + (size_t)sr * R : st.x + (size_t)(~sr) * R);
    stage_row<T, RPL>(Ds + (size_t)k * RC + lane * RPL, src + rl, lane_ok);
  }
  cp_async_wait_all();
  __syncwarp();
  main_done();
  if (!lane_ok) return;
  for (int r4 = 0; r4 < rows; r4 += 4) {
    T acc[4][RPL];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < RPL; ++q) acc[i][q] = T(0);
    for (int k = 0; k < K; ++k) {
      T gv[4], dv[RPL];
      lds<T, 4>(Gs + (size_t)k * rows_pad + r4, gv);
      lds<T, RPL>(Ds + (size_t)k * RC + lane * RPL, dv);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < RPL; ++q) acc[i][q] += gv[i] * dv[q];
    }
    if (bad) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < RPL; ++q) acc[i][q] = quiet_nan<T>();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r4 + i;
      if (row >= rows) break;
      if (FWD) {
        if (row < s)
          st_rhs<RPL>(st.y + (size_t)src_s[row] * R + rl, acc[i]);
        else
          st_rhs<RPL>(st.w + (size_t)(w_off + row - s) * R + rl, acc[i]);
      } else {
        st_rhs<RPL>(st.x + (size_t)src_s[row] * R + rl, acc[i]);
      }
    }
  }
}

template <typename T, int RPL, bool FWD, typename SVT>
__global__ void __launch_bounds__(kSolveThreads)
    k_panel_warp(BankView B, SVT S, const PanelItem* __restrict__ items, int n_items, int max_k,
                 int rows_pad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int idx = blockIdx.x * kWarpNodesPerCta + warp;
  if (idx >= n_items) return;
  const PanelItem I = items[idx];
  panel_warp_node<T, RPL, FWD, SVT>(
      B, S, I, (int)blockIdx.y * 32 * RPL, max_k, rows_pad,
      smem_raw + (size_t)warp * panel_warp_bytes<T>(max_k, rows_pad, 32 * RPL),
      [] {
        pdl_wait();
        return true;
      },
      [] { pdl_trigger(); });
}

// ---- flow sweeps -------------------------------------------------------------
// One persistent launch per sweep direction instead of one launch per tree
// level.  The direction's work entries are listed in topological order
// (forward from the lowest height up, backward from the greatest down); every CTA repeatedly takes the
// next entry from a ticket counter and, before reading any vector, waits until
// the entry's node has its inputs: forward, every item of its children has
// finished (their update rows are written); backward, every item of its
// parent has finished (the parent finished only after its own parent, so all
// ancestors' solution rows are written).  An entry only ever waits on entries
// with smaller tickets, which CTAs already running hold, so the sweep always
// progresses whatever the number of resident CTAs.  Finished items add one to
// a per-node counter with release semantics; waits read it with acquire
// semantics.  Each direction's launch zeroes the other direction's counters
// and ticket, so consecutive sweeps start from zero without extra launches.
// Vectors produced inside a launch are whole 128-byte lines per row (checked
// on the host), so no line read from L1 can be stale.
struct FlowView {
  const int4* entries;  // (0: one CTA item / 1: up to 8 warp items, first item, item count, RHS chunk)
  const PanelItem* items;
  const int4* sync;     // per item: (wait counter or -1, wait target, signal counter or -1, 0)
  int* ctr;             // this direction's per-node counters
  int* other_ctr;       // the other direction's (zeroed here)
  int n_ctr;
  int* queue;           // this direction's ticket counter
  int* other_queue;
  int* err;             // set to 1 when a wait runs out
  int n_entries;
};

template <typename T, int RPL, bool FWD, typename SVT>
__global__ void __launch_bounds__(kSolveThreads, 3)
    k_panel_flow(BankView B, SVT S, FlowView F, PanelShape P, int warp_max_k, int warp_rows_pad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_ticket, s_ok;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = blockIdx.x * kSolveThreads + tid; i < F.n_ctr; i += gridDim.x * kSolveThreads) F.other_ctr[i] = 0;
  if (blockIdx.x == 0 && tid == 0) *F.other_queue = 0;
  // The next ticket is taken while the current entry runs, and an entry's
  // completion is signalled (by lane 0 of the warp that owns it) after the
  // barrier that starts the next one, so neither round trip sits between
  // two entries.
  int pending = -1;  // lane 0: the counter this warp still has to signal
  if (tid == 0) s_ticket = atomicAdd(F.queue, 1);
  for (;;) {
    __syncthreads();
    const int t = s_ticket;
    if (lane == 0 && pending >= 0) red_release_gpu(F.ctr + pending, 1);
    pending = -1;
    __syncthreads();  // every thread has read s_ticket
    if (t >= F.n_entries) break;
    if (tid == 0) s_ticket = atomicAdd(F.queue, 1);
    const int4 e = F.entries[t];
    const int rc0 = e.w * 32 * RPL;
    if (e.x == 0) {
      const int4 sy = F.sync[e.y];
      panel_tile<T, RPL, FWD, SVT>(
          B, S, F.items[e.y], rc0, P, smem_raw, [&] {
            if (tid == 0) s_ok = sy.x < 0 || flow_wait(F.ctr + sy.x, sy.y, F.err);
            __syncthreads();
            return s_ok != 0;
          });
      if (tid == 0) pending = sy.z;
    } else if (warp < e.z) {
      const int ii = e.y + warp;
      const int4 sy = F.sync[ii];
      panel_warp_node<T, RPL, FWD, SVT>(
          B, S, F.items[ii], rc0, warp_max_k, warp_rows_pad,
          smem_raw + (size_t)warp * panel_warp_bytes<T>(warp_max_k, warp_rows_pad, 32 * RPL),
          [&] {
            int ok = 1;
            if (lane == 0) ok = sy.x < 0 || flow_wait(F.ctr + sy.x, sy.y, F.err);
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
          },
          [] {});
      __syncwarp();
      if (lane == 0) pending = sy.z;
    }
  }
}

constexpr size_t kFlowSmem = 96 * 1024;    // flow launches: leaf-warp slices within this
constexpr size_t kFlowScBytes = 32 * 1024;  // flow launches: staged child-update rows per chunk
constexpr int kFlowCmMax = 1024;            // flow launches: staged child-map entries per node

template <typename T, typename SVT>
const void* flow_kernel(int rpl, bool forward) {
  if (forward)
    return rpl == 1 ? (const void*)k_panel_flow<T, 1, true, SVT>
                    : (rpl == 2 ? (const void*)k_panel_flow<T, 2, true, SVT> : (const void*)k_panel_flow<T, 4, true, SVT>);
  return rpl == 1 ? (const void*)k_panel_flow<T, 1, false, SVT>
                  : (rpl == 2 ? (const void*)k_panel_flow<T, 2, false, SVT> : (const void*)k_panel_flow<T, 4, false, SVT>);
}

template <typename T, int RPL, typename SVT>
void launch_flow(bool forward, const BankView& B, const SVT& S, const FlowPlan& FP, const FlowView& F,
                 cudaStream_t st) {
  const PanelShape shape{FP.kc_cap, FP.ds_rows, FP.ri_max, FP.sc_rows, FP.max_s, FP.max_f, FP.cm_cap, FP.nbuf};
  if (forward)
    k_panel_flow<T, RPL, true, SVT><<<FP.grid, kSolveThreads, FP.smem, st>>>(B, S, F, shape, FP.warp_max_k,
                                                                            FP.warp_rows_pad);
  else
    k_panel_flow<T, RPL, false, SVT><<<FP.grid, kSolveThreads, FP.smem, st>>>(B, S, F, shape, FP.warp_max_k,
                                                                             FP.warp_rows_pad);
  PECS_CUDA(cudaGetLastError());
}

template <typename T, typename SVT>
void set_panel_smem_limit() {
  auto set = [&](const void* fn, size_t lim) {
    PECS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim));
  };
  set((const void*)k_panel_tiles<T, true, SVT>, kTileSmem);
  set((const void*)k_panel_tiles<T, false, SVT>, kTileSmem);
}

// Shared memory of a level's tiles: the columns of its longest tile at once where
// they fit kTileOnce (two CTAs on a multiprocessor), else in two buffers.
template <typename T>
TileShape tile_shape(const PanelLevel& L, const PanelOption& o, int chunk, size_t& smem) {
  const int bn = 32 * o.n, kgroups = o.warps / o.n;
  const size_t col = (size_t)(L.pad + bn) * sizeof(T);
  TileShape P{};
  P.lg_nw = o.n == 4 ? 2 : (o.n == 2 ? 1 : 0);
  P.kc = L.cols;
  if (chunk > 0) P.kc = std::min(P.kc, chunk);
  if ((size_t)P.kc * col > kTileOnce) P.kc = std::max(1, (int)(kTileBuffer / col));
  const int nbuf = P.kc < L.cols ? 2 : 1;
  P.a = 16 + (unsigned)(((L.cols + 3) & ~3) + 32) * 4;
  P.a_buf = (unsigned)((size_t)P.kc * L.pad * sizeof(T));
  P.b = P.a + nbuf * P.a_buf;
  P.b_buf = (unsigned)((size_t)P.kc * bn * sizeof(T));
  size_t end = P.b + (size_t)nbuf * P.b_buf;
  if (kgroups > 1) end = std::max(end, P.a + (size_t)kgroups * L.pad * bn * sizeof(T));
  P.p = (unsigned)end;
  if (L.passes) end += (size_t)L.pad * bn * sizeof(T);
  smem = end;
  return P;
}

template <typename T, bool FWD, typename SVT>
void launch_tiles(const TilesView& B, const SVT& S, int n_sets, const PanelPlan& L, const PanelOption& o,
                  int max_nrhs, int chunk, cudaStream_t st) {
  if (FWD && L.assembled) {
    AsmSets A{};
    int most = 0;
    bool vec = true;
    constexpr int V = 16 / (int)sizeof(T);
    for (int q = 0; q < n_sets; ++q) {
      A.rec[q] = L.tiles.rec[q], A.n[q] = L.tiles.n_rec[q];
      most = std::max(most, A.n[q]);
      vec = vec && S.set[q].nrhs % V == 0;
    }
    int lg = 3;  // threads per position
    while (lg < 8 && ((vec ? V : 1) << lg) < max_nrhs) ++lg;
    const dim3 grid((unsigned)((((long long)most << lg) + kSolveThreads - 1) / kSolveThreads), n_sets);
    launch_pdl(vec ? k_panel_assemble<T, V, SVT> : k_panel_assemble<T, 1, SVT>, grid, kSolveThreads, 0, st, B, S, A, lg);
  }
  size_t smem = 0;
  const TileShape P = tile_shape<T>(L.tiles, o, chunk, smem);
  if (smem > kTileSmem) throw PecsError(PECS_E_ARG, "panel staging exceeds shared memory");
  const int rc = 32 * o.n;
  launch_pdl(k_panel_tiles<T, FWD, SVT>, dim3(L.tiles.n, (max_nrhs + rc - 1) / rc), 32 * o.warps, smem, st, B, S,
             L.tiles.first, P);
}

template <typename T, int RPL, typename SVT>
void launch_panel_warp(bool forward, const BankView& B, const SVT& S, const PanelPlan& L,
                       int max_nrhs, cudaStream_t st) {
  constexpr int RC = 32 * RPL;
  const int rows_pad = (L.warp_rows + 3) & ~3, n = (int)L.warp.n;
  const size_t smem = kWarpNodesPerCta * panel_warp_bytes<T>(L.max_k, rows_pad, RC);
  const dim3 grid((n + kWarpNodesPerCta - 1) / kWarpNodesPerCta, (max_nrhs + RC - 1) / RC);
  BankView V = B;
  V.G = V.H = L.warp_val.p();  // the items' offsets
  launch_pdl(forward ? k_panel_warp<T, RPL, true, SVT> : k_panel_warp<T, RPL, false, SVT>, grid, kSolveThreads, smem, st,
             V, S, (const PanelItem*)L.warp.p, n, L.max_k, rows_pad);
}

// The valid options of a level for rpl_max right-hand sides per lane.
template <typename T>
std::vector<PanelOption> panel_options(const PanelPlan& L, int max_nrhs, int rpl_max) {
  std::vector<PanelOption> v;
  if (L.warp.n > 0)
    for (int rpl = rpl_max; rpl >= 1; rpl /= 2) {
      const int rows_pad = (L.warp_rows + 3) & ~3;
      if (kWarpNodesPerCta * panel_warp_bytes<T>(L.max_k, rows_pad, 32 * rpl) <= kWarpSmem)
        v.push_back(PanelOption{2, 8, rpl});
    }
  for (int n = 4; n >= 1; n /= 2)
    for (int warps : {8, 4})
      if (n == 1 || 16 * n < max_nrhs) v.push_back(PanelOption{0, warps, n});
  return v;
}

// Untuned banks: leaf warps where the level has them; else the most right-hand sides per
// CTA that give every multiprocessor two.
template <typename T>
PanelOption panel_default_option(const PanelPlan& L, int max_nrhs, int rpl_max, const PanelTuning& tu) {
  if (L.warp.n > 0) {
    int rpl = rpl_max;
    const int rows_pad = (L.warp_rows + 3) & ~3;
    while (rpl > 1 && kWarpNodesPerCta * panel_warp_bytes<T>(L.max_k, rows_pad, 32 * rpl) > kWarpSmem) rpl /= 2;
    return PanelOption{2, 8, rpl};
  }
  int n = max_nrhs > 64 ? 4 : (max_nrhs > 32 ? 2 : 1);
  while (n > 1 && (long long)L.tiles.n * ((max_nrhs + 32 * n - 1) / (32 * n)) < 2 * tu.min_ctas) n /= 2;
  return PanelOption{0, 8, n};
}

template <typename T, typename SVT>
void launch_panel_level(bool forward, const BankView& B, const TilesView& V, const SVT& S, int n_sets,
                        const PanelPlan& L, int max_nrhs, int rpl_max, const PanelTuning& tu, cudaStream_t st) {
  if (L.tiles.n == 0) return;
  PanelOption o = L.tuned;
  if (o.kind < 0 || (o.kind == 2 && o.n > rpl_max)) o = panel_default_option<T>(L, max_nrhs, rpl_max, tu);
  if (o.kind == 2) {
    switch (o.n) {
      case 1: launch_panel_warp<T, 1, SVT>(forward, B, S, L, max_nrhs, st); break;
      case 2: launch_panel_warp<T, 2, SVT>(forward, B, S, L, max_nrhs, st); break;
      default: launch_panel_warp<T, 4, SVT>(forward, B, S, L, max_nrhs, st); break;
    }
  } else if (forward) {
    launch_tiles<T, true, SVT>(V, S, n_sets, L, o, max_nrhs, tu.chunk, st);
  } else {
    launch_tiles<T, false, SVT>(V, S, n_sets, L, o, max_nrhs, tu.chunk, st);
  }
}
}  // namespace

FlowPlanHost plan_flow(const FlowNodes& nd, bool forward, int top, int rpl, int max_nrhs, int kc_max, int esz,
                       int n_sm) {
  FlowPlanHost H;
  const int n_nodes = (int)nd.s.size();
  const std::vector<std::vector<int>>& lv_all = forward ? nd.up : nd.down;
  // the covered levels in ticket order (forward: the greatest heights, from the
  // lowest of them up; backward: the same from the greatest down)
  const int L = (int)lv_all.size();
  top = std::min(std::max(top, 1), L);
  const std::vector<std::vector<int>> lv(forward ? lv_all.begin() + (L - top) : lv_all.begin(),
                                         forward ? lv_all.end() : lv_all.begin() + top);
  const int RC = 32 * rpl;
  H.n_chunks = (std::max(1, max_nrhs) + RC - 1) / RC;
  kc_max = std::max(1, kc_max);
  const int sc_cap = std::max(8, (int)(kFlowScBytes / ((size_t)RC * esz)));
  auto warp_bytes = [&](int k, int r) {
    return esz == 8 ? panel_warp_bytes<double>(k, r, RC) : panel_warp_bytes<float>(k, r, RC);
  };
  auto rows_of = [&](int g) { return forward ? nd.s[g] + nd.m[g] : nd.s[g]; };
  // per level: leaf warps (small nodes, forward without children, the warp
  // slices within budget) or CTA row tiles (32 rows, fewer where a level has
  // too few tiles to fill the GPU)
  std::vector<int> warp_level(lv.size(), 0), cap_level(lv.size(), 32);
  int wk = 0, wr = 0;
  for (size_t l = 0; l < lv.size(); ++l) {
    bool leaf = true;
    int mk = 0, mr = 0;
    for (int g : lv[l]) {
      const int f = nd.s[g] + nd.m[g];
      const int rows = rows_of(g), k = forward ? nd.s[g] : f;
      const bool kids = nd.cmap_ptr[nd.cm_off[g] + f] > nd.cmap_ptr[nd.cm_off[g]];
      if (k > kWarpMaxK || rows > kWarpMaxRows || (forward && kids)) leaf = false;
      mk = std::max(mk, k);
      mr = std::max(mr, rows);
    }
    const int nk = std::max(wk, mk), nr = std::max(wr, (mr + 3) & ~3);
    if (leaf && kWarpNodesPerCta * warp_bytes(nk, nr) <= kFlowSmem) {
      warp_level[l] = 1;
      wk = nk;
      wr = nr;
      continue;
    }
    int cap = 32;
    while (cap > 4) {
      long long t = 0;
      for (int g : lv[l]) t += (rows_of(g) + cap - 1) / cap;
      if (t * H.n_chunks >= n_sm) break;
      cap /= 2;
    }
    cap_level[l] = cap;
  }
  H.warp_max_k = wk;
  H.warp_rows_pad = wr;
  // items per node (signals per chunk), then the items with their waits
  std::vector<int> nsig(n_nodes, 0), per_node(n_nodes, 1);
  for (size_t l = 0; l < lv.size(); ++l)
    for (int g : lv[l]) {
      const int rows = rows_of(g);
      if (warp_level[l]) {
        nsig[g] = 1;
        per_node[g] = rows;
      } else {
        const int cap = cap_level[l];
        const int nit = (rows + cap - 1) / cap;
        per_node[g] = (rows + nit - 1) / nit;
        nsig[g] = (rows + per_node[g] - 1) / per_node[g];
      }
    }
  std::vector<int> kid_sig(n_nodes, 0);
  for (int g = 0; g < n_nodes; ++g)
    if (nd.parent[g] >= 0) kid_sig[nd.parent[g]] += nsig[g];
  int min_ri = 32, max_k_tiles = 0;
  for (size_t l = 0; l < lv.size(); ++l) {
    const size_t first = H.items.size();
    for (int g : lv[l]) {
      const int s = nd.s[g], m = nd.m[g], f = s + m;
      const int rows = rows_of(g);
      const long long off = forward ? nd.goff[g] : nd.hoff[g];
      const int cb = nd.cmap_ptr[nd.cm_off[g]];
      const int ncm = nd.cmap_ptr[nd.cm_off[g] + f] - cb;
      const int p = nd.parent[g];
      const int4 sy = forward ? make_int4(kid_sig[g] > 0 ? g : -1, kid_sig[g] * H.n_chunks, p, 0)
                              : make_int4(p, p >= 0 ? nsig[p] * H.n_chunks : 0, g, 0);
      PanelItem it;
      it.b = make_int4(s, m, nd.node_set[g], nd.w_off[g]);
      it.c = make_int4((int)(off & 0xffffffffll), (int)(off >> 32), nd.own_off[g], nd.upd_off[g]);
      if (warp_level[l]) {
        it.a = make_int4(g, 0, rows, 32);
        it.d = make_int4(nd.cm_off[g], cb, 0, 0);
        H.items.push_back(it);
        H.sync.push_back(sy);
        continue;
      }
      // the widest chunk (<= kc_max columns) whose child-update rows fit
      int kc = kc_max, rows_sc = 0;
      for (;; kc /= 2) {
        rows_sc = 0;
        if (forward) {
          const int* cp = nd.cmap_ptr.data() + nd.cm_off[g];
          for (int k0 = 0; k0 < s; k0 += kc) rows_sc = std::max(rows_sc, cp[std::min(k0 + kc, s)] - cp[k0]);
        }
        if (rows_sc <= sc_cap || kc == 1) break;
      }
      H.kc_cap = std::max(H.kc_cap, kc);
      max_k_tiles = std::max(max_k_tiles, forward ? s : f);
      H.sc_rows = std::max(H.sc_rows, rows_sc);
      H.max_s = std::max(H.max_s, s);
      H.max_f = std::max(H.max_f, f);
      H.cm_cap = std::max(H.cm_cap, std::min(ncm, kFlowCmMax));
      const int per = per_node[g];
      int ri = 4;
      while (ri < per) ri *= 2;
      H.ri_max = std::max(H.ri_max, ri);
      min_ri = std::min(min_ri, ri);
      it.d = make_int4(nd.cm_off[g], cb, ncm, 0);
      it.kc = kc;
      for (int r0 = 0; r0 < rows; r0 += per) {
        it.a = make_int4(g, r0, std::min(rows, r0 + per), ri);
        H.items.push_back(it);
        H.sync.push_back(sy);
      }
    }
    // entries: the level's items, each for every chunk (consecutive, so the
    // chunks of one tile share its block in L2); leaf warps in groups
    for (size_t i = first; i < H.items.size();) {
      const int n = warp_level[l] ? (int)std::min<size_t>(kWarpNodesPerCta, H.items.size() - i) : 1;
      for (int c = 0; c < H.n_chunks; ++c) H.entries.push_back(make_int4(warp_level[l], (int)i, n, c));
      i += n;
    }
  }
  H.nbuf = max_k_tiles > H.kc_cap ? 2 : 1;  // items of several chunks: double-buffered staging
  H.ds_rows = min_ri < 32 ? std::max(H.kc_cap, 32 / H.nbuf) : H.kc_cap;
  const int meta = forward ? H.max_s + H.max_f + 1 + H.cm_cap : H.max_f;
  const size_t tile_smem =
      esz == 8 ? panel_smem_bytes<double>(H.ds_rows, RC, H.kc_cap, H.ri_max, H.sc_rows, meta, H.nbuf)
               : panel_smem_bytes<float>(H.ds_rows, RC, H.kc_cap, H.ri_max, H.sc_rows, meta, H.nbuf);
  const size_t warp_smem = wk == 0 ? 0 : kWarpNodesPerCta * warp_bytes(wk, wr);
  H.smem = std::max(tile_smem, warp_smem);
  H.ok = H.smem <= kPanelSmem;
  return H;
}

BankView FactorBank::view() const {
  BankView v;
  v.own_idx = own_idx_.p;
  v.upd_idx = upd_idx_.p;
  v.cmap_ptr = cmap_ptr_.p;
  v.cmap_idx = cmap_idx_.p;
  v.G = G_.p();
  v.H = H_.p();
  return v;
}

TilesView FactorBank::tiles_view(int d, const PanelPlan& L) const {
  return TilesView{tiles_[d].p, L.val.p(), L.val0, tidx_[d].p, rec_.p, more_.p};
}

long long FactorBank::bytes() const {
  if (!panel_) return rows_.bytes();
  long long n = G_.bytes() + H_.bytes();
  for (auto* plans : {&pfwd_, &pbwd_})
    for (const PanelPlan& L : *plans) n += L.val.bytes() + L.warp_val.bytes();
  return n;
}

long long FactorBank::sweep_bytes() const {
  if (!panel_) return rows_.bytes();
  const int top = flow_sel_ < 0 ? 0 : flow_cfg_[flow_sel_].top;
  long long n = flow_sel_ < 0 ? 0 : flow_cfg_[flow_sel_].values;
  for (int d = 0; d < 2; ++d) {
    const std::vector<PanelPlan>& plans = d == 0 ? pfwd_ : pbwd_;
    for (size_t l = 0; l < plans.size(); ++l) {
      if (d == 0 ? l + top >= plans.size() : (int)l < top) continue;  // in the flow sweep
      const PanelPlan& L = plans[l];
      // untuned levels take leaf warps where they have them
      n += L.tuned.kind == 2 || (L.tuned.kind < 0 && L.warp.n > 0) ? L.n_warp_val : L.n_val;
    }
  }
  return n * (prec_ == PECS_PREC_FP64 ? 8 : 4);
}

int FactorBank::kernel_launches_per_solve() const {
  if (!panel_) return rows_.launches_per_solve(max_nrhs_);
  if (flow_sel_ >= 0) {
    const int top = flow_cfg_[flow_sel_].top;
    int n = 2;
    for (size_t l = 0; l + top < pfwd_.size(); ++l) n += pfwd_[l].launches();
    for (size_t l = top; l < pbwd_.size(); ++l) n += pbwd_[l].launches();
    return n;
  }
  int n = 0;
  for (auto& l : pfwd_) n += l.launches();
  for (auto& l : pbwd_) n += l.launches();
  return n;
}

void FactorBank::build(const std::vector<const MfFactor*>& factors, int precision, bool panel,
                       PanelTuning tuning, int max_nrhs) {
  if (factors.empty() || (int)factors.size() > kMaxSets)
    throw PecsError(PECS_E_ARG, "factor bank needs 1..4 factors");
  prec_ = precision;
  panel_ = panel;
  tune_ = tuning;
  if (tune_.chunk < 0 || tune_.chunk > 128 || tune_.min_ctas < 0)
    throw PecsError(PECS_E_ARG, "panel tuning out of range");
  if (tune_.min_ctas == 0) tune_.min_ctas = kTargetCtas;
  n_sets_ = (int)factors.size();
  max_nrhs_ = max_nrhs;
  if (!panel) {
    rows_.build(factors, precision, max_nrhs);
    entries_ = rows_.entries();
    for (int si = 0; si < n_sets_; ++si) set_wtotal_[si] = rows_.set_wtotal(si);
    return;
  }
  std::vector<int> hs, hm, own_off, upd_off, w_off, cm_off, own_idx, upd_idx, cmap_ptr, cmap_idx,
      node_set;
  std::vector<long long> goff, hoff;
  std::vector<int> node_at;  // of its factor
  long long go = 0, ho = 0;
  int wtot = 0;
  struct LevelNodes {
    std::vector<int> nodes;
  };
  std::vector<LevelNodes> fl, bl;
  int base = 0;
  for (int fi = 0; fi < n_sets_; ++fi) {
    const MfFactor& F = *factors[fi];
    const int N = (int)F.nodes.size();
    if ((int)F.Gf.size() != N) throw PecsError(PECS_E_STATE, "factor not factorised");
    // update-vector offsets are local to the factor: each RHS owns a buffer of
    // set_wtotal(set) doubles
    std::vector<int> wbase(N);
    wtot = 0;
    for (int j = 0; j < N; ++j) {
      wbase[j] = wtot;
      wtot += F.nodes[j].m;
    }
    set_wtotal_[fi] = std::max(1, wtot);
    std::vector<int> fpos(F.n, -1);
    for (int j = 0; j < N; ++j) {
      const MfNode& nd = F.nodes[j];
      hs.push_back(nd.s);
      hm.push_back(nd.m);
      own_off.push_back((int)own_idx.size());
      upd_off.push_back((int)upd_idx.size());
      own_idx.insert(own_idx.end(), nd.own.begin(), nd.own.end());
      upd_idx.insert(upd_idx.end(), nd.upd.begin(), nd.upd.end());
      w_off.push_back(wbase[j]);
      node_set.push_back(fi);
      goff.push_back(go);
      hoff.push_back(ho);
      node_at.push_back(j);
      go += (long long)F.Gf[j].size();
      ho += (long long)F.Hb[j].size();
      // extend-add gather lists per front position
      const int f = nd.s + nd.m;
      for (int t = 0; t < nd.s; ++t) fpos[nd.own[t]] = t;
      for (int t = 0; t < nd.m; ++t) fpos[nd.upd[t]] = nd.s + t;
      std::vector<std::vector<int>> lists(f);
      for (int c : nd.children) {
        const MfNode& ch = F.nodes[c];
        for (int a = 0; a < ch.m; ++a) {
          int p = fpos[ch.upd[a]];
          if (p < 0) throw PecsError(PECS_E_STATE, "extend-add map mismatch");
          lists[p].push_back(wbase[c] + a);
        }
      }
      for (int t = 0; t < nd.s; ++t) fpos[nd.own[t]] = -1;
      for (int t = 0; t < nd.m; ++t) fpos[nd.upd[t]] = -1;
      cm_off.push_back((int)cmap_ptr.size());
      for (int p = 0; p < f; ++p) {
        cmap_ptr.push_back((int)cmap_idx.size());
        cmap_idx.insert(cmap_idx.end(), lists[p].begin(), lists[p].end());
      }
      cmap_ptr.push_back((int)cmap_idx.size());
      if ((int)fl.size() <= nd.height) fl.resize(nd.height + 1);
      fl[nd.height].nodes.push_back(base + j);
    }
    base += N;
  }
  // backward: from the greatest height down (a parent is higher than its children).
  // Levels by depth mix cell blocks of 8 rows with separators of hundreds.
  bl.assign(fl.rbegin(), fl.rend());
  entries_ = go + ho;
  own_idx_.upload(own_idx);
  upd_idx_.upload(upd_idx);
  cmap_ptr_.upload(cmap_ptr);
  cmap_idx_.upload(cmap_idx);
  // blocks of these nodes (forward Gf, backward Hb), column-major, one after another
  auto column_major = [&](const std::vector<int>& nodes, bool forward, BankValues& out) {
    size_t n = 0;
    for (int g : nodes) n += (size_t)hs[g] * (hs[g] + hm[g]);
    auto fill = [&](auto* o) {
      using T = typename std::remove_pointer<decltype(o)>::type;
      for (int g : nodes) {
        const MfFactor& F = *factors[node_set[g]];
        const int f = hs[g] + hm[g], rows = forward ? f : hs[g], cols = forward ? hs[g] : f;
        const std::vector<double>& v = forward ? F.Gf[node_at[g]] : F.Hb[node_at[g]];
        for (int c = 0; c < cols; ++c)
          for (int r = 0; r < rows; ++r) *o++ = (T)v[(size_t)r * cols + c];
      }
    };
    if (prec_ == PECS_PREC_FP64) {
      std::vector<double> v(n);
      fill(v.data());
      out.f64.upload(v);
    } else {
      std::vector<float> v(n);
      fill(v.data());
      out.f32.upload(v);
    }
  };
  if (tune_.flow) {
    std::vector<int> all(hs.size());
    std::iota(all.begin(), all.end(), 0);
    column_major(all, true, G_);
    column_major(all, false, H_);
  }
  {
    // level plans: tiles of packed values (panel_plan.hpp), and leaf warps
    const PanelTilesPlan H = plan_panel(factors, (std::max(1, max_nrhs) + 31) / 32, tune_.min_ctas,
                                        prec_ == PECS_PREC_FP64 ? kPanelRowsF64 : kPanelRowsF32);
    const int esz = prec_ == PECS_PREC_FP64 ? 8 : 4;
    rec_.upload(H.rec);
    more_.upload(H.more);
    for (int d = 0; d < 2; ++d) {
      const bool forward = d == 0;
      const PanelTilesPlan::Dir& D = H.dir[d];
      tiles_[d].upload(D.tiles);
      tidx_[d].upload(D.idx);
      std::unique_ptr<double[]> v64(prec_ == PECS_PREC_FP64 ? new double[D.n_values] : nullptr);
      std::unique_ptr<float[]> v32(prec_ == PECS_PREC_FP64 ? nullptr : new float[D.n_values]);
      if (v64)
        pack_panel(H, factors, d, v64.get());
      else
        pack_panel(H, factors, d, v32.get());
      std::vector<PanelPlan>& out = forward ? pfwd_ : pbwd_;
      const std::vector<LevelNodes>& lv = forward ? fl : bl;
      out.clear();
      out.resize(lv.size());
      for (size_t l = 0; l < lv.size(); ++l) {
        PanelPlan& L = out[l];
        L.tiles = D.levels[l];
        for (int q = 0; q < n_sets_; ++q) L.assembled = L.assembled || (forward && L.tiles.n_rec[q] > 0);
        const size_t end = (size_t)L.tiles.first + L.tiles.n;
        L.val0 = L.tiles.n > 0 ? D.tiles[L.tiles.first].off : 0;
        L.n_val = L.tiles.n > 0 ? (end < D.tiles.size() ? D.tiles[end].off : D.n_values) - L.val0 : 0;
        auto upload_tiles = [&] {
          if (v64)
            L.val.f64.upload(v64.get() + L.val0, (size_t)L.n_val);
          else
            L.val.f32.upload(v32.get() + L.val0, (size_t)L.n_val);
        };
        // leaf level: every node small and, forward, without children
        bool leaf = true;
        for (int g : lv[l].nodes) {
          const int f = hs[g] + hm[g];
          const int rows = forward ? f : hs[g];
          const int k = forward ? hs[g] : f;
          const bool kids = cmap_ptr[cm_off[g] + f] > cmap_ptr[cm_off[g]];
          if (k > kWarpMaxK || rows > kWarpMaxRows || (forward && kids)) leaf = false;
          L.max_k = std::max(L.max_k, k);
          L.warp_rows = std::max(L.warp_rows, rows);
        }
        const size_t rows_pad = (size_t)((L.warp_rows + 3) & ~3);
        const size_t wb = (((size_t)L.max_k * 32 + (size_t)L.max_k * rows_pad) * esz + (size_t)L.max_k * 4 + 15) & ~(size_t)15;
        const bool warps = leaf && kWarpNodesPerCta * wb <= kWarpSmem;
        if (!warps || tune_.options) upload_tiles();  // untuned, leaf levels take the warps
        if (!warps) continue;
        column_major(lv[l].nodes, forward, L.warp_val);
        std::vector<PanelItem> items;
        for (int g : lv[l].nodes) {
          const long long off = L.n_warp_val;
          L.n_warp_val += (long long)hs[g] * (hs[g] + hm[g]);
          PanelItem it;
          it.a = make_int4(g, 0, forward ? hs[g] + hm[g] : hs[g], 32);
          it.b = make_int4(hs[g], hm[g], node_set[g], w_off[g]);
          it.c = make_int4((int)(off & 0xffffffffll), (int)(off >> 32), own_off[g], upd_off[g]);
          it.d = make_int4(cm_off[g], cmap_ptr[cm_off[g]], 0, 0);
          items.push_back(it);
        }
        L.warp.upload(items);
      }
    }
    if (prec_ == PECS_PREC_FP64)
      set_panel_smem_limit<double, IlSetsView>();
    else
      set_panel_smem_limit<float, IlSetsViewF>();
    // flow plans: both directions, 1, 2 and 4 right-hand sides per lane
    n_nodes_ = (int)hs.size();
    std::vector<int> parent(n_nodes_, -1);
    {
      int b0 = 0;
      for (int fi = 0; fi < n_sets_; ++fi) {
        const MfFactor& F = *factors[fi];
        for (int j = 0; j < (int)F.nodes.size(); ++j)
          for (int c : F.nodes[j].children) parent[b0 + c] = b0 + j;
        b0 += (int)F.nodes.size();
      }
    }
    flow_state_.alloc(2 * (size_t)n_nodes_ + 3);
    flow_state_.zero();
    stall_node_ = -1;
    for (int g = 0; g < (int)factors[0]->nodes.size() && stall_node_ < 0; ++g)
      if (parent[g] < 0 && !factors[0]->nodes[g].children.empty()) stall_node_ = g;
    int n_sm = 0, dev = 0;
    PECS_CUDA(cudaGetDevice(&dev));
    PECS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    FlowNodes nodes{hs, hm, node_set, w_off, own_off, upd_off, cm_off, cmap_ptr, goff, hoff, parent, {}, {}};
    for (auto& l : fl) nodes.up.push_back(l.nodes);
    for (auto& l : bl) nodes.down.push_back(l.nodes);
    flow_cfg_.clear();
    flow_sel_ = -1;
    const int n_levels = (int)std::max(fl.size(), bl.size());
    std::vector<int> tops{n_levels};
    for (int t : {7, 5, 3})
      if (t < n_levels) tops.push_back(t);
    for (int top : tops) {
      if (!tune_.flow) break;
      long long values = 0;  // bl is fl from the root down
      for (size_t l = 0; l < std::min((size_t)top, bl.size()); ++l)
        for (int g : bl[l].nodes) values += 2ll * hs[g] * (hs[g] + hm[g]);
      for (int kc : {64, 32}) {
        for (int rpl : {1, 2, 4}) {
          FlowConfig cfg;
          cfg.top = top;
          cfg.values = values;
          cfg.kc = tune_.chunk > 0 ? std::min(kc, tune_.chunk) : kc;
          cfg.rpl = rpl;
          bool ok = true;
          for (int d = 0; d < 2 && ok; ++d) {
            FlowPlan& FP = cfg.plan[d];
            FlowPlanHost H = plan_flow(nodes, d == 0, top, rpl, max_nrhs, cfg.kc, esz, n_sm);
            if (!H.ok) {
              ok = false;
              break;
            }
            FP.top = top;
            FP.rpl = rpl;
            FP.n_chunks = H.n_chunks;
            FP.kc_cap = H.kc_cap;
            FP.nbuf = H.nbuf;
            FP.ds_rows = H.ds_rows;
            FP.ri_max = H.ri_max;
            FP.sc_rows = H.sc_rows;
            FP.max_s = H.max_s;
            FP.max_f = H.max_f;
            FP.cm_cap = H.cm_cap;
            FP.warp_max_k = H.warp_max_k;
            FP.warp_rows_pad = H.warp_rows_pad;
            FP.smem = H.smem;
            FP.n_entries = (int)H.entries.size();
            FP.items.upload(H.items);
            FP.sync.upload(H.sync);
            FP.entries.upload(H.entries);
            const void* fn = esz == 8 ? flow_kernel<double, IlSetsView>(rpl, d == 0)
                                      : flow_kernel<float, IlSetsViewF>(rpl, d == 0);
            PECS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem));
            int per_sm = 0;
            PECS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSolveThreads, FP.smem));
            FP.grid = std::max(1, std::min(FP.n_entries, std::max(1, per_sm) * n_sm));
          }
          if (ok) flow_cfg_.push_back(std::move(cfg));
        }
      }
    }
  }
}

void FactorBank::tune_rows_flow(const IlSetsView& sets, int max_nrhs, cudaStream_t st, int flow_mode, int reps) {
  if (!panel_) rows_.tune_flow(row_sets(sets), max_nrhs, st, flow_mode, reps);
}

RowSets FactorBank::row_sets(const IlSetsView& sets) const {
  RowSets v;
  for (int si = 0; si < n_sets_; ++si) {
    const IlSetView& a = sets.set[si];
    RowSet& r = v.set[si];
    r.nrhs = r.sd = a.nrhs;
    r.n = rows_.dofs(si);
    r.sr = 1;
    r.b = a.b, r.x = a.x, r.y = a.y, r.w = a.w;
    r.d = a.x;  // free until the backward sweep writes the solutions
  }
  return v;
}

void FactorBank::solve(const RowSets& sets, int max_nrhs, cudaStream_t st) const {
  if (panel_) throw PecsError(PECS_E_STATE, "panel factor bank needs the interleaved layout");
  rows_.solve(sets, max_nrhs, st);
}

void FactorBank::solve(const IlSetsView& sets, int max_nrhs, cudaStream_t st) const {
  if (panel_ && prec_ != PECS_PREC_FP64)
    throw PecsError(PECS_E_STATE, "FP32 panel banks take float sweep vectors");
  if (panel_)
    solve_panel(sets, max_nrhs, st);
  else
    rows_.solve(row_sets(sets), max_nrhs, st);
}

template <typename SVT>
int FactorBank::panel_rpl(const SVT& sets, int max_nrhs) const {
  // right-hand sides per lane: at most as many as fill the lanes, dividing every set's count
  int rpl = max_nrhs >= 96 ? 4 : (max_nrhs >= 48 ? 2 : 1);
  for (int si = 0; si < n_sets_; ++si)
    while (rpl > 1 && sets.set[si].nrhs % rpl != 0) rpl /= 2;
  return rpl;
}

int FactorBank::flow_error(bool clear) const {
  if (!panel_) return rows_.flow_error(clear);
  if (flow_state_.n == 0) return 0;
  int e = 0;
  int* p = flow_state_.p + 2 * (size_t)n_nodes_ + 2;
  PECS_CUDA(cudaMemcpy(&e, p, sizeof(int), cudaMemcpyDeviceToHost));
  if (clear) PECS_CUDA(cudaMemset(p, 0, sizeof(int)));
  return e;
}

void FactorBank::debug_arm_flow_stall() const {
  if (!panel_) return rows_.debug_arm_flow_stall();
  if (flow_state_.n == 0 || stall_node_ < 0) throw PecsError(PECS_E_STATE, "no flow sweep to stall");
  PECS_CUDA(cudaDeviceSynchronize());
  const int v = -(1 << 30);
  PECS_CUDA(cudaMemcpy(flow_state_.p + stall_node_, &v, sizeof(int), cudaMemcpyHostToDevice));
}

// A flow configuration applies when its plans cover these right-hand sides
// and every sweep vector row is a whole number of 128-byte lines at a 128-byte
// aligned address (rows written inside the launch never share a line with
// another).
template <typename SVT>
bool FactorBank::flow_ok(const SVT& sets, int max_nrhs, int cfg) const {
  using T = typename std::conditional<std::is_same<SVT, IlSetsViewF>::value, float, double>::type;
  if (!panel_ || cfg < 0 || cfg >= (int)flow_cfg_.size()) return false;
  if ((prec_ == PECS_PREC_FP64) != (sizeof(T) == 8)) return false;
  const FlowConfig& C = flow_cfg_[cfg];
  const int rpl = C.rpl;
  if (C.plan[0].n_entries == 0 || C.plan[1].n_entries == 0) return false;
  if ((max_nrhs + 32 * rpl - 1) / (32 * rpl) != C.plan[0].n_chunks) return false;
  if (panel_rpl(sets, max_nrhs) < rpl) return false;
  auto al = [](const void* p) { return ((uintptr_t)p & 127u) == 0; };
  for (int si = 0; si < n_sets_; ++si) {
    const auto& v = sets.set[si];
    if (v.nrhs > max_nrhs || v.nrhs % rpl != 0 || ((size_t)v.nrhs * sizeof(T)) % 128 != 0) return false;
    if (!al(v.b) || !al(v.y) || !al(v.w) || !al(v.x)) return false;
  }
  return true;
}

// Hybrid sweep: level launches for the levels below the configuration's top
// levels, then one flow launch per direction over those, then level launches
// again (backward) for the rest.
template <typename SVT>
void FactorBank::solve_flow(const SVT& sets, int max_nrhs, int cfg, cudaStream_t st) const {
  using T = typename std::conditional<std::is_same<SVT, IlSetsViewF>::value, float, double>::type;
  const BankView B = view();
  const FlowConfig& C = flow_cfg_[cfg];
  const int lrpl = panel_rpl(sets, max_nrhs);
  int* base = flow_state_.p;
  int* ctr[2] = {base, base + n_nodes_};
  int* queue[2] = {base + 2 * (size_t)n_nodes_, base + 2 * (size_t)n_nodes_ + 1};
  int* err = base + 2 * (size_t)n_nodes_ + 2;
  for (size_t l = 0; l + C.top < pfwd_.size(); ++l)
    launch_panel_level<T, SVT>(true, B, tiles_view(0, pfwd_[l]), sets, n_sets_, pfwd_[l], max_nrhs, lrpl, tune_, st);
  for (int d = 0; d < 2; ++d) {
    const FlowPlan& FP = C.plan[d];
    const FlowView F{FP.entries.p, FP.items.p, FP.sync.p, ctr[d], ctr[1 - d], n_nodes_,
                     queue[d],     queue[1 - d], err,     FP.n_entries};
    switch (C.rpl) {
      case 1: launch_flow<T, 1, SVT>(d == 0, B, sets, FP, F, st); break;
      case 2: launch_flow<T, 2, SVT>(d == 0, B, sets, FP, F, st); break;
      default: launch_flow<T, 4, SVT>(d == 0, B, sets, FP, F, st); break;
    }
  }
  for (size_t l = C.top; l < pbwd_.size(); ++l)
    launch_panel_level<T, SVT>(false, B, tiles_view(1, pbwd_[l]), sets, n_sets_, pbwd_[l], max_nrhs, lrpl, tune_, st);
}

template <typename SVT>
void FactorBank::solve_panel(const SVT& sets, int max_nrhs, cudaStream_t st) const {
  if (flow_sel_ >= 0 && flow_ok(sets, max_nrhs, flow_sel_)) {
    solve_flow(sets, max_nrhs, flow_sel_, st);
    return;
  }
  const int rpl = panel_rpl(sets, max_nrhs);
  const BankView B = view();
  for (int pass = 0; pass < 2; ++pass) {
    const bool fwd = pass == 0;
    for (const PanelPlan& L : fwd ? pfwd_ : pbwd_) {
      if constexpr (std::is_same<SVT, IlSetsViewF>::value)
        launch_panel_level<float, SVT>(fwd, B, tiles_view(pass, L), sets, n_sets_, L, max_nrhs, rpl, tune_, st);
      else
        launch_panel_level<double, SVT>(fwd, B, tiles_view(pass, L), sets, n_sets_, L, max_nrhs, rpl, tune_, st);
    }
  }
}

// Per level, choose the tiling option that gives the fastest whole sweep:
// starting from the heuristic choice everywhere, each level in turn tries all
// of its valid options with the other levels fixed, timing complete sweeps
// (minimum of `reps` after one warm-up), so every level is measured with the
// cache state the real sweep gives it.  The sweep's values are meaningless
// while tuning; callers solve again before using any result.
template <typename SVT>
void FactorBank::force_flow_impl(const SVT& sets, int max_nrhs) {
  // every level in the flow launch, the widest chunks and the most
  // right-hand sides per lane that apply
  int best = -1;
  for (int c = 0; c < (int)flow_cfg_.size(); ++c) {
    const FlowConfig& C = flow_cfg_[c];
    if (!flow_ok(sets, max_nrhs, c) || C.top != flow_cfg_[0].top) continue;
    if (best < 0 || C.kc > flow_cfg_[best].kc || (C.kc == flow_cfg_[best].kc && C.rpl > flow_cfg_[best].rpl))
      best = c;
  }
  flow_sel_ = best;
}

void FactorBank::force_flow(const IlSetsViewF& sets, int max_nrhs) {
  force_flow_impl(sets, max_nrhs);
  release_unused();
}
void FactorBank::force_flow(const IlSetsView& sets, int max_nrhs) {
  force_flow_impl(sets, max_nrhs);
  release_unused();
}

// Once the kernels are chosen: the flow plans and the forms of the blocks that none of them
// reads.  (A chosen flow sweep keeps the levels' too: they are timed on request.)
void FactorBank::release_unused() {
  for (int c = 0; c < (int)flow_cfg_.size(); ++c) {
    if (c == flow_sel_) continue;
    for (FlowPlan& P : flow_cfg_[c].plan) {
      P.items.release();
      P.sync.release();
      P.entries.release();
      P.n_entries = 0;
    }
  }
  if (flow_sel_ >= 0) return;
  G_.release();
  H_.release();
  for (auto* plans : {&pfwd_, &pbwd_})
    for (PanelPlan& L : *plans) {
      if (L.tuned.kind == 2) L.val.release();
      if (L.tuned.kind == 0) L.warp.release(), L.warp_val.release();
    }
}

template <typename SVT>
void FactorBank::autotune_panel(const SVT& sets, int max_nrhs, cudaStream_t st, int reps, int flow_mode) {
  using T = typename std::conditional<std::is_same<SVT, IlSetsViewF>::value, float, double>::type;
  if (!tune_.flow && flow_mode >= 0) throw PecsError(PECS_E_STATE, "bank built without flow sweeps");
  if (!tune_.options) throw PecsError(PECS_E_STATE, "bank built for the untuned kernels only");
  const int rpl = panel_rpl(sets, max_nrhs);
  cudaEvent_t e0, e1;
  PECS_CUDA(cudaEventCreate(&e0));
  PECS_CUDA(cudaEventCreate(&e1));
  for (int pass = 0; pass < 2; ++pass)
    for (PanelPlan& L : pass == 0 ? pfwd_ : pbwd_)
      L.tuned = panel_default_option<T>(L, max_nrhs, rpl, tune_);
  auto time_sweep = [&]() {
    const int per_sweep = kernel_launches_per_solve();
    float best = 1e30f;
    solve_panel(sets, max_nrhs, st);  // warm-up
    tune_launches_ += per_sweep;
    for (int r = 0; r < reps; ++r) {
      PECS_CUDA(cudaEventRecord(e0, st));
      solve_panel(sets, max_nrhs, st);
      PECS_CUDA(cudaEventRecord(e1, st));
      PECS_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      PECS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best = std::min(best, ms);
      tune_launches_ += per_sweep;
    }
    return best;
  };
  float best_sweep = time_sweep();
  for (int pass = 0; pass < 2; ++pass) {
    for (PanelPlan& L : pass == 0 ? pfwd_ : pbwd_) {
      const PanelOption keep = L.tuned;
      PanelOption best = keep;
      for (const PanelOption& o : panel_options<T>(L, max_nrhs, rpl)) {
        if (o.kind == keep.kind && o.warps == keep.warps && o.n == keep.n) continue;
        L.tuned = o;
        float ms;
        try {
          ms = time_sweep();
        } catch (const PecsError& err) {
          if (err.code != PECS_E_ARG) throw;
          continue;  // the option's staging does not fit in shared memory
        }
        if (ms < best_sweep) {
          best_sweep = ms;
          best = o;
        }
      }
      L.tuned = best;
    }
  }
  // the flow sweep (one persistent launch per direction) at each valid
  // right-hand-sides-per-lane count, against the tuned level sweep
  int best_flow = -1;
  float best_flow_ms = 1e30f;
  for (int c = 0; c < (int)flow_cfg_.size() && flow_mode >= 0; ++c) {
    if (!flow_ok(sets, max_nrhs, c)) continue;
    flow_sel_ = c;
    const float ms = time_sweep();
    flow_sel_ = -1;
    if (std::getenv("PECS_TUNE_LOG"))  // diagnostic: every flow configuration's sweep time
      std::fprintf(stderr, "flow top %d kc %d rpl %d: %.4f ms (levels %.4f ms)\n", flow_cfg_[c].top,
                   flow_cfg_[c].kc, flow_cfg_[c].rpl, ms, best_sweep);
    if (flow_error() != 0)
      throw PecsError(PECS_E_CUDA, "flow sweep: a wait for a node's inputs ran out");
    if (ms < best_flow_ms) {
      best_flow_ms = ms;
      best_flow = c;
    }
  }
  if (best_flow >= 0 && (flow_mode > 0 || best_flow_ms < best_sweep)) {
    best_sweep = best_flow_ms;
    flow_sel_ = best_flow;
  }
  release_unused();
  tuned_ms_ = best_sweep;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
}

std::vector<double> FactorBank::time_levels(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st,
                                            int reps) const {
  if (!panel_ || prec_ == PECS_PREC_FP64) throw PecsError(PECS_E_STATE, "level timing needs an FP32 panel bank");
  const int rpl = panel_rpl(sets, max_nrhs);
  const BankView B = view();
  const int nl = (int)(pfwd_.size() + pbwd_.size());
  std::vector<cudaEvent_t> ev(nl + 1);
  for (auto& e : ev) PECS_CUDA(cudaEventCreate(&e));
  std::vector<double> ms(nl, 0.0);
  for (int r = 0; r <= reps; ++r) {
    int l = 0;
    PECS_CUDA(cudaEventRecord(ev[0], st));
    for (int pass = 0; pass < 2; ++pass)
      for (const PanelPlan& L : pass == 0 ? pfwd_ : pbwd_) {
        launch_panel_level<float, IlSetsViewF>(pass == 0, B, tiles_view(pass, L), sets, n_sets_, L, max_nrhs, rpl, tune_, st);
        PECS_CUDA(cudaEventRecord(ev[++l], st));
      }
    PECS_CUDA(cudaEventSynchronize(ev[nl]));
    if (r == 0) continue;
    for (int k = 0; k < nl; ++k) {
      float t = 0.f;
      PECS_CUDA(cudaEventElapsedTime(&t, ev[k], ev[k + 1]));
      ms[k] += t / reps;
    }
  }
  for (auto& e : ev) cudaEventDestroy(e);
  return ms;
}

void FactorBank::autotune(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st, int reps, int flow_mode) {
  if (!panel_ || prec_ == PECS_PREC_FP64) throw PecsError(PECS_E_STATE, "autotune needs an FP32 panel bank");
  autotune_panel(sets, max_nrhs, st, reps, flow_mode);
}

void FactorBank::autotune(const IlSetsView& sets, int max_nrhs, cudaStream_t st, int reps, int flow_mode) {
  if (!panel_ || prec_ != PECS_PREC_FP64) throw PecsError(PECS_E_STATE, "autotune needs an FP64 panel bank");
  autotune_panel(sets, max_nrhs, st, reps, flow_mode);
}

void FactorBank::solve(const IlSetsViewF& sets, int max_nrhs, cudaStream_t st) const {
  if (!panel_ || prec_ == PECS_PREC_FP64)
    throw PecsError(PECS_E_STATE, "float solve vectors need a panel bank with FP32 factors");
  solve_panel(sets, max_nrhs, st);
}

}  // namespace pecs
