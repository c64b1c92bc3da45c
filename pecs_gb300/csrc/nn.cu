// Neural operator for the learned warm start: a small MLP mapping the six
// physical parameters of an instance (bias, generation amplitude, absorption
// coefficient, doping, lifetime, interface rate) to the coefficients of a
// fixed low-rank (POD) basis of the steady-state fields.  No counterpart in
// the reference: it is the warm-start component the benchmark adds.
//
// Arithmetic: GEMM operands are BF16 (weights stored in BF16, activations
// rounded to BF16 when staged), accumulation FP32 on the tensor cores
// (tcgen05.mma into TMEM); FP32 master weights and Adam moments.  Layers: z = x W^T + b, y = tanh(z) for hidden layers, linear
// output; loss = mean squared error.  The decoder (mean + V c) is an FP32 GEMM.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include "bulk_copy.cuh"
#include "common.hpp"
#include "fp_bits.cuh"
#include "sweep_sync.cuh"

namespace pecs {
namespace {

constexpr int kBM = 64, kBN = 64, kBK = 16, kGemmThreads = 256;

// The decoder's GEMM in FP32: C[M,N] = A[M,K] B[N,K]^T + mean[n].
__global__ void __launch_bounds__(kGemmThreads)
    k_decode(int M, int N, int K, const float* __restrict__ A, const float* __restrict__ B,
             const float* __restrict__ mean, float* __restrict__ C) {
  __shared__ float As[kBK][kBM + 1];
  __shared__ float Bs[kBK][kBN + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += kBK) {
    for (int t = threadIdx.x; t < kBK * kBM; t += kGemmThreads) {
      const int kk = t % kBK, mm = t / kBK, m = m0 + mm, k = k0 + kk;
      As[kk][mm] = m < M && k < K ? A[(size_t)m * K + k] : 0.f;
    }
    for (int t = threadIdx.x; t < kBK * kBN; t += kGemmThreads) {
      const int nn = t % kBN, kk = t / kBN, n = n0 + nn, k = k0 + kk;
      Bs[kk][nn] = n < N && k < K ? B[(size_t)n * K + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kBK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * N + n] = acc[i][j] + mean[n];
    }
  }
}

// ---- tensor-core GEMM: tcgen05.mma, BF16 operands, FP32 accumulator in TMEM ----
// The layers' GEMMs op(A) op(B) with BF16-rounded operands run on the
// 5th-generation tensor cores.  Most are small (batch 256 x 704 x 704), so the latency
// of one tile and the number of SMs that have one decide: a CTA owns a 128 x 32 tile
// of C (32 TMEM columns; 88 tiles of a 256 x 704 layer, where 128 columns gave 12), and
// forward, where those are more than the SMs, 64 or 128 columns (Mlp::forward).  Per K
// chunk of 64 its 256 threads convert op(A) (128 x 64) and op(B)^T (a row per column) to
// BF16, eight K values per 16-byte store, into the canonical K-major layout without
// swizzle (8-row x 16-byte core matrices; K-adjacent core matrices 128 B apart, 8-row
// groups 1024 B apart), one thread issues four tcgen05.mma (K = 16 each) and commits
// them to the buffer's mbarrier, and the loads of the next two chunks run under them
// (two buffers, three register sets).  Waits poll a bounded number of times: one that
// runs out sets the error flag, the tile is skipped and the TMEM is still freed.  The
// epilogue reads the accumulator with tcgen05.ld (warp w: TMEM lanes 32 (w % 4).. =
// rows, 16 of each 32 columns).  Measured at batch 256 with 6-704-704-704-64 layers
// against 128 x 128 tiles staged value by value: the forward pass and its call 488 -> 91
// us, loss and gradients without their copy to the host 1,025 -> 161 us; the sums are
// the same bits.
constexpr int kTcM = 128, kTcN = 32, kTcK = 64, kTcThreads = 256;
constexpr int kTcSms = 152;  // multiprocessors of a GB300
constexpr long long kTcPollLimit = 1LL << 24;

// shared-memory matrix descriptor: start address, leading-dimension byte
// offset (K direction, 128 B), stride byte offset (8-row groups, 1024 B),
// descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
         ((uint64_t)(1024u >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity) {
  for (long long i = 0; i < kTcPollLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Eight K-consecutive values of one row (or column) of an operand, as loaded.
// CONTIGUOUS: they follow one another in memory (16-byte loads where `vec` says that
// the rows are aligned); else `ld` apart.  pack: as BF16, K ascending.
struct Raw8F {
  float v[8];
  __device__ __forceinline__ uint4 pack() const {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  template <bool CONTIGUOUS>
  __device__ __forceinline__ void load(const float* p, int ld, int n, bool vec) {
    if (CONTIGUOUS && vec && n == 8) {
      const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = j < n ? p[CONTIGUOUS ? (size_t)j : (size_t)j * ld] : 0.f;
    }
  }
};
struct Raw8H {
  uint16_t v[8];
  __device__ __forceinline__ uint4 pack() const {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = (uint32_t)v[2 * j] | (uint32_t)v[2 * j + 1] << 16;
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  template <bool CONTIGUOUS>
  __device__ __forceinline__ void load(const __nv_bfloat16* q, int ld, int n, bool vec) {
    const uint16_t* p = reinterpret_cast<const uint16_t*>(q);
    if (CONTIGUOUS && vec && n == 8) {
      const uint4 a = *reinterpret_cast<const uint4*>(p);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (uint16_t)(w[j / 2] >> (j % 2 * 16));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = j < n ? p[CONTIGUOUS ? (size_t)j : (size_t)j * ld] : (uint16_t)0;
    }
  }
};
template <typename T>
struct Raw8Of {
  using type = Raw8F;
};
template <>
struct Raw8Of<__nv_bfloat16> {
  using type = Raw8H;
};

template <int TN>
struct GemmSmem {
  __align__(1024) unsigned char a[2][kTcM * kTcK * 2];
  __align__(1024) unsigned char b[2][TN * kTcK * 2];
  __align__(8) unsigned long long mbar[2];
  uint32_t tmem;
};

// One 128 x TN tile at (m0, n0) of op(A)[M,K] op(B)[K,N]: op(A)(m,k) = TA ?
// A[k*lda+m] : A[m*lda+k]; op(B)(k,n) = TB ? B[n*ldb+k] : B[k*ldb+n].  wait() is
// called before the first operand is read.  epilogue(row, column, values[16]) gets
// the sums of one row's columns [column, column + 16).
template <typename TAe, typename TBe, bool TA, bool TB, int TN, typename Wait, typename Epi>
__device__ __forceinline__ void gemm_tile(GemmSmem<TN>& s, int M, int N, int K, const TAe* __restrict__ A, int lda,
                                          const TBe* __restrict__ B, int ldb, int m0, int n0, int* err, Wait wait,
                                          Epi epilogue) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s.tmem)),
                 "r"((uint32_t)TN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  const uint32_t bar[2] = {smem_u32(&s.mbar[0]), smem_u32(&s.mbar[1])};
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar[0]) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar[1]) : "memory");
  }
  // this thread's 16-byte pieces: four of A, one of B per 32 columns.  Along K-contiguous
  // operands lanes take 8 rows x 4 pieces (whole sectors, and shared-memory stores
  // without bank conflicts), else consecutive rows.
  const bool va = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  const bool vb = ldb % (16 / (int)sizeof(TBe)) == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0;
  auto place = [&](bool contiguous, int idx, int rows, int& row, int& k8) {
    if (contiguous) {
      row = (idx >> 6) * 8 + (idx & 7);
      k8 = (idx >> 5 & 1) * 4 + (idx >> 3 & 3);
    } else {
      row = idx % rows;
      k8 = idx / rows;
    }
  };
  constexpr int NB = TN / 32;
  struct Set {
    typename Raw8Of<TAe>::type a[4];
    typename Raw8Of<TBe>::type b[NB];
  } set[3];
  auto load = [&](Set& r, int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int row, k8;
      place(!TA, tid + q * kTcThreads, kTcM, row, k8);
      const int m = m0 + row, k = k0 + k8 * 8, n = m < M ? min(8, K - k) : 0;
      r.a[q].template load<!TA>(TA ? A + (size_t)k * lda + m : A + (size_t)m * lda + k, lda, n, va);
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      int row, k8;
      place(TB, tid + q * kTcThreads, TN, row, k8);
      const int c = n0 + row, k = k0 + k8 * 8, n = c < N ? min(8, K - k) : 0;
      r.b[q].template load<TB>(TB ? B + (size_t)c * ldb + k : B + (size_t)k * ldb + c, ldb, n, vb);
    }
  };
  auto piece = [](int row, int k8) { return (row >> 3) * 1024 + k8 * 128 + (row & 7) * 16; };
  const int nk = (K + kTcK - 1) / kTcK;
  wait();
  load(set[0], 0);
  if (nk > 1) load(set[1], kTcK);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = s.tmem;
  // instruction descriptor (kind::f16): FP32 accumulator, BF16 A and B, both
  // K-major, N = TN, M = 128
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) |
                         ((uint32_t)(kTcM >> 4) << 24);
  bool ok = true;
  // chunk kc from registers `cur` into shared memory and multiplied, while the
  // loads of chunk kc + 2 (into `far`) and kc + 1 are in flight
  auto step = [&](int kc, const Set& cur, Set& far) {
    const int buf = kc & 1;
    if (kc + 2 < nk) load(far, (kc + 2) * kTcK);
    if (kc >= 2) ok = tc_wait(bar[buf], ((kc >> 1) - 1) & 1) && ok;  // the chunk before last has been multiplied
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int row, k8;
      place(!TA, tid + q * kTcThreads, kTcM, row, k8);
      *reinterpret_cast<uint4*>(s.a[buf] + piece(row, k8)) = cur.a[q].pack();
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      int row, k8;
      place(TB, tid + q * kTcThreads, TN, row, k8);
      *reinterpret_cast<uint4*>(s.b[buf] + piece(row, k8)) = cur.b[q].pack();
    }
    // the staged tiles are read by the tensor cores (async proxy)
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (tid == 0) {
#pragma unroll
      for (int q = 0; q < kTcK / 16; ++q) {
        const uint64_t ad = tc_desc(smem_u32(s.a[buf]) + q * 256);
        const uint64_t bd = tc_desc(smem_u32(s.b[buf]) + q * 256);
        const uint32_t accumulate = (kc > 0 || q > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar[buf])
                   : "memory");
    }
  };
  for (int kc = 0; kc < nk; kc += 3) {
    step(kc, set[0], set[2]);
    if (kc + 1 < nk) step(kc + 1, set[1], set[0]);
    if (kc + 2 < nk) step(kc + 2, set[2], set[1]);
  }
  // the last commit covers every MMA before it
  ok = tc_wait(bar[(nk - 1) & 1], ((nk - 1) >> 1) & 1) && ok;
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (__syncthreads_or(!ok)) {
    if (tid == 0) atomicExch(err, 1);
    tc_wait(bar[(nk - 1) & 1], ((nk - 1) >> 1) & 1);  // MMAs still in flight (bounded) before the TMEM is freed
  } else {
    const int row = m0 + (warp & 3) * 32 + lane;
#pragma unroll 1
    for (int c0 = (warp >> 2) * 16; c0 < TN; c0 += 32) {
      uint32_t v[16];
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                   : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                     "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                   : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0)
                   : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      float f[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(v[j]);
      if (row < M) epilogue(row, n0 + c0, f);
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)TN) : "memory");
}

// 16 consecutive values of one row, those below column N
__device__ __forceinline__ void store16(float* __restrict__ C, int ldc, int N, int row, int n, const float (&f)[16]) {
  float* p = C + (size_t)row * ldc + n;
  if (n + 16 <= N && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) reinterpret_cast<float4*>(p)[j / 4] = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (n + j < N) p[j] = f[j];
  }
}

// Y (B x N) = X (B x K) W^T + bias, W stored N x K; act: tanh.
template <int TN>
__global__ void __launch_bounds__(kTcThreads)
    k_mlp_layer(int B, int N, int K, const float* __restrict__ X, const __nv_bfloat16* __restrict__ W,
                const float* __restrict__ bias, int act, float* __restrict__ Y, int* err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  GemmSmem<TN>& s = *reinterpret_cast<GemmSmem<TN>*>(smem_raw);
  pdl_trigger();
  gemm_tile<float, __nv_bfloat16, false, true>(s, B, N, K, X, K, W, K, (int)blockIdx.y * kTcM, (int)blockIdx.x * TN,
                                               err, [] { pdl_wait(); }, [&](int row, int n, float (&f)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (n + j < N) f[j] += bias[n + j];
      if (act) f[j] = tanhf(f[j]);
    }
    store16(Y, N, N, row, n, f);
  });
}

// Backward of one layer in one launch, by block: dW (N x K) = dZ^T X tiles; dX (B x
// K) = (dZ W) (1 - X^2) tiles (null: first layer; X is the previous layer's tanh);
// db (N) = column sums of dZ, in batch order.
__global__ void __launch_bounds__(kTcThreads)
    k_mlp_layer_bwd(int B, int N, int K, const float* __restrict__ dZ, const float* __restrict__ X,
                    const __nv_bfloat16* __restrict__ W, float* __restrict__ dW, float* __restrict__ db,
                    float* __restrict__ dX, int w_blocks, int x_blocks, int* err) {
  __shared__ GemmSmem<kTcN> s;
  pdl_trigger();
  const int nk = (K + kTcN - 1) / kTcN;  // column tiles of both products
  int q = blockIdx.x;
  if (q < w_blocks) {
    gemm_tile<float, float, true, false>(s, N, K, B, dZ, N, X, K, q / nk * kTcM, q % nk * kTcN, err,
                                         [] { pdl_wait(); },
                                         [&](int row, int n, float (&f)[16]) { store16(dW, K, K, row, n, f); });
    return;
  }
  q -= w_blocks;
  if (q < x_blocks) {
    gemm_tile<float, __nv_bfloat16, false, false>(s, B, K, N, dZ, N, W, K, q / nk * kTcM, q % nk * kTcN, err,
                                                  [] { pdl_wait(); }, [&](int row, int n, float (&f)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (n + j < K) {
          const float x = X[(size_t)row * K + n + j];
          f[j] *= (1.f - x * x);
        }
      store16(dX, K, K, row, n, f);
    });
    return;
  }
  q -= x_blocks;
  pdl_wait();
  const int n = q * kTcThreads + threadIdx.x;
  if (n >= N) return;
  float t = 0.f;
  for (int b0 = 0; b0 < B; b0 += 16) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = b0 + j < B ? dZ[(size_t)(b0 + j) * N + n] : 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (b0 + j < B) t += v[j];
  }
  db[n] = t;
}

// dy = 2 (y - t) / (B N); per-block partial loss sums
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ t, float* __restrict__ dy,
                      size_t n, float* __restrict__ loss_partial) {
  __shared__ float s[256];
  float acc = 0.f;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float d = y[i] - t[i];
    dy[i] = 2.f * d / (float)n;
    acc += d * d;
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) loss_partial[blockIdx.x] = s[0];
}

// Adam on FP32 masters, refreshes the BF16 copy
__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, __nv_bfloat16* __restrict__ wb, size_t n, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  wb[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb, size_t n) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) wb[i] = __float2bfloat16_rn(w[i]);
}

}  // namespace

constexpr int kLossParts = 64;

struct Mlp {
  std::vector<int> w;          // widths, layers = w.size()-1
  size_t n_params = 0;
  std::vector<size_t> woff, boff;  // offsets of W_l (out x in) and b_l in the packed vector
  DBuf<float> P, G, Mo, Vo;    // masters, grads, Adam moments
  DBuf<__nv_bfloat16> Pb;      // BF16 copy
  int max_batch = 0;
  std::vector<DBuf<float>> act;  // act[l]: batch x w[l] (hidden layers and the output)
  std::vector<DBuf<float>> dact;
  // pinned, written by the kernels, read after a synchronisation: the loss's
  // partial sums, and a flag set by a GEMM whose MMA-completion wait ran out
  struct Host {
    float loss[kLossParts];
    int err;
  };
  Host* host = nullptr;
  int adam_t = 0;
  cudaStream_t st = nullptr;
  ~Mlp() {
    if (st) cudaStreamDestroy(st);
    if (host) cudaFreeHost(host);
  }

  void ensure_batch(int B) {
    if (B <= max_batch) return;
    act.clear();
    dact.clear();
    act.resize(w.size());
    dact.resize(w.size());
    for (size_t l = 1; l < w.size(); ++l) {
      act[l].alloc((size_t)B * w[l]);
      dact[l].alloc((size_t)B * w[l]);
    }
    max_batch = B;
  }

  const __nv_bfloat16* Wb(int l) const { return Pb.p + woff[l]; }
  const float* bias(int l) const { return P.p + boff[l]; }

  static int tiles(int n, int t) { return (n + t - 1) / t; }

  // Activations of every layer; the output into y (null: act.back()).  x and y may
  // overlap: the first layer has read x when the last one writes y, and a network of one
  // layer, whose tiles read and write the same rows at the same time, then goes through
  // act.back().
  void forward(int B, const float* x, float* y, cudaStream_t s) {
    ensure_batch(B);
    const int L = (int)w.size() - 1;
    const size_t ny = (size_t)B * w[L] * sizeof(float);
    const uintptr_t px = reinterpret_cast<uintptr_t>(x), py = reinterpret_cast<uintptr_t>(y);
    if (L == 1 && y && px < py + ny && py < px + (size_t)B * w[0] * sizeof(float)) {
      forward(B, x, nullptr, s);
      PECS_CUDA(cudaMemcpyAsync(y, act.back().p, ny, cudaMemcpyDeviceToDevice, s));
      return;
    }
    for (int l = 0; l < L; ++l) {
      // act[l+1] = act(act[l] W_l^T + b_l); W_l stored out x in (row-major)
      auto go = [&](auto tn) {
        constexpr int TN = decltype(tn)::value;
        constexpr size_t smem = sizeof(GemmSmem<TN>);
        if (smem > 48 * 1024)
          PECS_CUDA(cudaFuncSetAttribute(k_mlp_layer<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        launch_pdl(k_mlp_layer<TN>, dim3(tiles(w[l + 1], TN), tiles(B, kTcM)), kTcThreads, smem, s, B, w[l + 1], w[l],
                     l == 0 ? x : (const float*)act[l].p, Wb(l), bias(l), l < L - 1 ? 1 : 0,
                     l == L - 1 && y ? y : act[l + 1].p, &host->err);
      };
      // The narrowest tile that leaves no more tiles than SMs (none wider than the layer):
      // with fewer tiles SMs idle, with more the activations are converted again for every
      // tile of a row.  us per forward pass for 32 / 64 / 128 columns: 6-704-704-704-64,
      // batch 256 90 / 108 / 134, 1,000 134 / 108 / 134, 4,096 287 / 231 / 217;
      // 64-2048-2048-64, batch 256 140 / 165 / 194, 512 204 / 165 / 195, 4,096 968 / 630 / 498.
      auto fits = [&](int tn) { return w[l + 1] <= tn || tiles(w[l + 1], tn) * (long long)tiles(B, kTcM) <= kTcSms; };
      if (fits(32))
        go(std::integral_constant<int, 32>());
      else if (fits(64))
        go(std::integral_constant<int, 64>());
      else
        go(std::integral_constant<int, 128>());
    }
  }

  // gradients of mean((y - t)^2) into G; the loss's partial sums into host->loss
  void backward(int B, const float* x, const float* target, cudaStream_t s) {
    const int L = (int)w.size() - 1;
    const size_t nout = (size_t)B * w[L];
    k_mse<<<kLossParts, 256, 0, s>>>(act[L].p, target, dact[L].p, nout, host->loss);
    PECS_CUDA(cudaGetLastError());
    for (int l = L - 1; l >= 0; --l) {
      const int N = w[l + 1], K = w[l], wb = tiles(N, kTcM) * tiles(K, kTcN),
                xb = l > 0 ? tiles(B, kTcM) * tiles(K, kTcN) : 0;
      launch_pdl(k_mlp_layer_bwd, dim3(wb + xb + tiles(N, kTcThreads)), kTcThreads, 0, s, B, N, K, (const float*)dact[l + 1].p,
                   l == 0 ? x : (const float*)act[l].p, Wb(l), G.p + woff[l], G.p + boff[l],
                   l > 0 ? dact[l].p : nullptr, wb, xb, &host->err);
    }
  }

  // after the stream has synchronised: report (and clear) a GEMM that gave up
  void check_err() {
    if (host->err) {
      host->err = 0;
      throw PecsError(PECS_E_CUDA, "a tensor-core GEMM gave up waiting for its MMAs; outputs are invalid");
    }
  }

  // after the stream has synchronised
  float read_loss(int B) const {
    double t = 0;
    for (float v : host->loss) t += v;
    return (float)(t / ((double)B * w.back()));
  }

  void adam(float lr, cudaStream_t s) {
    ++adam_t;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)adam_t), c2 = 1.f - std::pow(b2, (float)adam_t);
    k_adam<<<(unsigned)((n_params + 255) / 256), 256, 0, s>>>(P.p, Mo.p, Vo.p, G.p, Pb.p, n_params, lr,
                                                              b1, b2, 1e-8f, c1, c2);
    PECS_CUDA(cudaGetLastError());
  }

  void sync_bf16(cudaStream_t s) {
    k_to_bf16<<<(unsigned)((n_params + 255) / 256), 256, 0, s>>>(P.p, Pb.p, n_params);
    PECS_CUDA(cudaGetLastError());
  }
};

}  // namespace pecs

using namespace pecs;

struct pecs_mlp {
  Mlp m;
};

namespace pecs {
void set_error_external(const std::string& m);
}

#define NN_TRY(...)                                     \
  try {                                                 \
    __VA_ARGS__;                                        \
    return PECS_OK;                                     \
  } catch (const PecsError& ex) {                       \
    pecs::set_error_external(ex.what());                \
    return ex.code;                                     \
  } catch (const std::exception& ex) {                  \
    pecs::set_error_external(ex.what());                \
    return PECS_E_ARG;                                  \
  }

extern "C" {

int pecs_mlp_create(int n_layers, const int* widths, unsigned long long seed, pecs_mlp** out) {
  NN_TRY({
    if (!out || !widths || n_layers < 1 || n_layers > 16) throw PecsError(PECS_E_ARG, "bad layers");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0)
      throw PecsError(PECS_E_NODEVICE, "no CUDA device available");
    std::unique_ptr<pecs_mlp> h(new pecs_mlp());
    Mlp& m = h->m;
    m.w.assign(widths, widths + n_layers + 1);
    for (int x : m.w)
      if (x < 1 || x > 65536) throw PecsError(PECS_E_ARG, "bad width");
    size_t off = 0;
    for (int l = 0; l < n_layers; ++l) {
      m.woff.push_back(off);
      off += (size_t)m.w[l] * m.w[l + 1];
      m.boff.push_back(off);
      off += m.w[l + 1];
    }
    m.n_params = off;
    std::vector<float> init(off, 0.f);
    std::mt19937_64 g(seed);
    for (int l = 0; l < n_layers; ++l) {
      const float sc = std::sqrt(1.0f / m.w[l]);  // LeCun-uniform-like for tanh
      std::uniform_real_distribution<float> U(-sc * std::sqrt(3.f), sc * std::sqrt(3.f));
      for (size_t t = 0; t < (size_t)m.w[l] * m.w[l + 1]; ++t) init[m.woff[l] + t] = U(g);
    }
    PECS_CUDA(cudaStreamCreateWithFlags(&m.st, cudaStreamNonBlocking));
    m.P.upload(init);
    m.G.alloc(off);
    m.G.zero();
    PECS_CUDA(cudaHostAlloc((void**)&m.host, sizeof(Mlp::Host), cudaHostAllocDefault));
    m.host->err = 0;
    m.Mo.alloc(off);
    m.Mo.zero();
    m.Vo.alloc(off);
    m.Vo.zero();
    m.Pb.alloc(off);
    m.sync_bf16(m.st);
    PECS_CUDA(cudaStreamSynchronize(m.st));
    *out = h.release();
  })
}

void pecs_mlp_destroy(pecs_mlp* m) { delete m; }

int pecs_mlp_n_params(pecs_mlp* h, long long* n) {
  NN_TRY({
    if (!h || !n) throw PecsError(PECS_E_ARG, "NULL argument");
    *n = (long long)h->m.n_params;
  })
}

int pecs_mlp_get_params(pecs_mlp* h, float* host) {
  NN_TRY({
    if (!h || !host) throw PecsError(PECS_E_ARG, "NULL argument");
    PECS_CUDA(cudaMemcpy(host, h->m.P.p, h->m.n_params * 4, cudaMemcpyDeviceToHost));
  })
}

int pecs_mlp_set_params(pecs_mlp* h, const float* host) {
  NN_TRY({
    if (!h || !host) throw PecsError(PECS_E_ARG, "NULL argument");
    Mlp& m = h->m;
    PECS_CUDA(cudaMemcpy(m.P.p, host, m.n_params * 4, cudaMemcpyHostToDevice));
    m.sync_bf16(m.st);
    m.Mo.zero();
    m.Vo.zero();
    m.adam_t = 0;
    PECS_CUDA(cudaStreamSynchronize(m.st));
  })
}

// y (batch x out) = network(x (batch x in)); device pointers
int pecs_mlp_forward(pecs_mlp* h, int batch, const float* x_dev, float* y_dev, void* stream) {
  NN_TRY({
    if (!h || batch < 1 || !x_dev || !y_dev) throw PecsError(PECS_E_ARG, "invalid arguments");
    Mlp& m = h->m;
    cudaStream_t s = stream ? (cudaStream_t)stream : m.st;
    m.forward(batch, x_dev, y_dev, s);
    PECS_CUDA(cudaStreamSynchronize(s));
    m.check_err();
  })
}

// gradients of the MSE loss (no update); grad_host receives n_params floats
int pecs_mlp_gradients(pecs_mlp* h, int batch, const float* x_dev, const float* t_dev, float* grad_host,
                       float* loss) {
  NN_TRY({
    if (!h || batch < 1 || !x_dev || !t_dev) throw PecsError(PECS_E_ARG, "invalid arguments");
    Mlp& m = h->m;
    m.forward(batch, x_dev, nullptr, m.st);
    m.backward(batch, x_dev, t_dev, m.st);
    if (grad_host)
      PECS_CUDA(cudaMemcpyAsync(grad_host, m.G.p, m.n_params * 4, cudaMemcpyDeviceToHost, m.st));
    PECS_CUDA(cudaStreamSynchronize(m.st));
    if (loss) *loss = m.read_loss(batch);
    m.check_err();
  })
}

// one Adam step on the MSE loss of (x, t); loss (may be NULL) returns the pre-update loss
int pecs_mlp_train_step(pecs_mlp* h, int batch, const float* x_dev, const float* t_dev, float lr,
                        float* loss) {
  NN_TRY({
    if (!h || batch < 1 || !x_dev || !t_dev || !(lr > 0)) throw PecsError(PECS_E_ARG, "invalid arguments");
    Mlp& m = h->m;
    m.forward(batch, x_dev, nullptr, m.st);
    m.backward(batch, x_dev, t_dev, m.st);
    m.adam(lr, m.st);
    PECS_CUDA(cudaStreamSynchronize(m.st));
    if (loss) *loss = m.read_loss(batch);
    m.check_err();
  })
}

// Warm-start carrier vectors straight from the network's coefficients: for
// each row b, y_i = mean_i + sum_j V_ij c_bj (FP32, j ascending) over the 2 n_u
// density outputs, and the full carrier vectors (nd doubles, currents zero) get
// exp(y) in their density block at u_off: electrons from y_0..y_{n_u-1},
// holes from y_{n_u}..y_{2 n_u - 1}.
//
// Blocks below n_tiles * b_tiles: a 128-output x 64-row tile, V and c staged in
// shared memory 32 coefficients at a time, a thread 4 outputs x 8 rows -- so V is
// read once per 64 rows where a thread per (row, output) read it again for each.  The
// other blocks write the zeros (two thirds of the result).  Bound by its writes:
// 201 MB at batch 256, n_u = 16,384; measured there 1,920 -> 84 us.
constexpr int kWsOut = 128, kWsRows = 64, kWsK = 32, kWsZeros = 4096;

__global__ void __launch_bounds__(256, 4)
    k_warm_start(int batch, int r, int n_u, const float* __restrict__ c, const float* __restrict__ V,
                 const float* __restrict__ mean, int nd, int u_off, double* __restrict__ vn,
                 double* __restrict__ vp, int n_tiles, int b_tiles) {
  __shared__ float Vs[kWsK][kWsOut + 1];
  __shared__ __align__(16) float Cs[kWsK][kWsRows + 4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((int)blockIdx.x >= n_tiles * b_tiles) {  // kWsZeros of one vector's zeros
    const int q = (int)blockIdx.x - n_tiles * b_tiles, row = q % (2 * batch), nz = nd - n_u;
    double* out = row < batch ? vn + (size_t)row * nd : vp + (size_t)(row - batch) * nd;
    const int i0 = q / (2 * batch) * kWsZeros, i1 = min(nz, i0 + kWsZeros);
    for (int i = i0 + tid; i < i1; i += 256) out[i < u_off ? i : i + n_u] = 0.0;
    return;
  }
  const int o0 = (int)blockIdx.x % n_tiles * kWsOut, b0 = (int)blockIdx.x / n_tiles * kWsRows;
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int o = o0 + lane + 32 * i;
    const float m = o < 2 * n_u ? mean[o] : 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[i][b] = m;
  }
  for (int k0 = 0; k0 < r; k0 += kWsK) {
    const int kc = min(kWsK, r - k0);
    __syncthreads();
    for (int e = tid; e < kWsOut * kWsK; e += 256) {
      const int k = e % kWsK, o = e / kWsK;
      Vs[k][o] = k < kc && o0 + o < 2 * n_u ? V[(size_t)(o0 + o) * r + k0 + k] : 0.f;
    }
    for (int e = tid; e < kWsRows * kWsK; e += 256) {
      const int k = e % kWsK, b = e / kWsK;
      Cs[k][b] = k < kc && b0 + b < batch ? c[(size_t)(b0 + b) * r + k0 + k] : 0.f;
    }
    __syncthreads();
    if (b0 + warp * 8 < batch) {
#pragma unroll 4
      for (int k = 0; k < kc; ++k) {
        const float4 c0 = *reinterpret_cast<const float4*>(&Cs[k][warp * 8]);
        const float4 c1 = *reinterpret_cast<const float4*>(&Cs[k][warp * 8 + 4]);
        const float cv[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float v = Vs[k][lane + 32 * i];
#pragma unroll
          for (int b = 0; b < 8; ++b) acc[i][b] = fmaf(v, cv[b], acc[i][b]);
        }
      }
    }
  }
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int row = b0 + warp * 8 + b;
    if (row >= batch) break;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int o = o0 + lane + 32 * i;
      if (o >= 2 * n_u) continue;
      const bool hole = o >= n_u;
      (hole ? vp : vn)[(size_t)row * nd + u_off + (hole ? o - n_u : o)] = f2d_exact(expf(acc[i][b]));
    }
  }
}

// Few outputs of few coefficients: a thread per value.  Bound by its launch; the tiles'
// staging and their 32 values per thread take 2 to 6 us more: n_u = 64, r = 3, batch 256 25.2
// -> 19.0 us the call, n_u = 1,000, r = 17, batch 16 24.7 -> 19.1.  The tiles are faster from
// kWsFew densities on (n_u = 1,000, batch 256: 25.0 against 26.6), and where a thread's
// coefficients are more than a stage (n_u = 16,384, r = 64, batch 1: 25.3 against 35.2: its
// loads of V are not coalesced).  The same sums in the same order.
constexpr long long kWsFew = 1 << 18;

__global__ void __launch_bounds__(256)
    k_warm_start_few(int r, int n_u, const float* __restrict__ c, const float* __restrict__ V,
                     const float* __restrict__ mean, int nd, int u_off, double* __restrict__ vn,
                     double* __restrict__ vp) {
  __shared__ float cs[kWsK];
  const size_t row = blockIdx.y;
  if ((int)threadIdx.x < r) cs[threadIdx.x] = c[row * r + threadIdx.x];
  __syncthreads();
  for (long long t = blockIdx.x * 256 + threadIdx.x; t < 2LL * nd; t += (long long)gridDim.x * 256) {
    const bool hole = t >= nd;
    const int d = (int)(hole ? t - nd : t), i = d - u_off;
    double x = 0.0;
    if (i >= 0 && i < n_u) {
      const int o = hole ? n_u + i : i;
      const float* v = V + (size_t)o * r;
      float y = mean[o];
      for (int j = 0; j < r; ++j) y = fmaf(v[j], cs[j], y);
      x = f2d_exact(expf(y));
    }
    (hole ? vp : vn)[row * nd + d] = x;
  }
}

// FP32 decoder: y (batch x n) = mean (n) + c (batch x r) V^T, V stored n x r (row-major)
int pecs_decode(int batch, int r, int n, const float* c_dev, const float* V_dev, const float* mean_dev,
                float* y_dev, void* stream) {
  NN_TRY({
    if (batch < 1 || r < 1 || n < 1 || !c_dev || !V_dev || !mean_dev || !y_dev)
      throw PecsError(PECS_E_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    k_decode<<<dim3((n + kBN - 1) / kBN, (batch + kBM - 1) / kBM), kGemmThreads, 0, s>>>(batch, n, r, c_dev, V_dev,
                                                                                         mean_dev, y_dev);
    PECS_CUDA(cudaGetLastError());
    PECS_CUDA(cudaStreamSynchronize(s));
  })
}

int pecs_warm_start_vectors(int batch, int r, int n_u, const float* c_dev, const float* V_dev,
                            const float* mean_dev, int nd, int u_off, double* vn_dev, double* vp_dev,
                            void* stream) {
  NN_TRY({
    if (batch < 1 || r < 1 || n_u < 1 || nd < 1 || u_off < 0 || u_off + n_u > nd || !c_dev || !V_dev ||
        !mean_dev || !vn_dev || !vp_dev)
      throw PecsError(PECS_E_ARG, "invalid arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (r <= kWsK && batch <= 65535 && 2LL * n_u * batch <= kWsFew) {
      const unsigned nx = (unsigned)std::min<long long>((2LL * nd + 255) / 256, 1024);
      k_warm_start_few<<<dim3(nx, batch), 256, 0, s>>>(r, n_u, c_dev, V_dev, mean_dev, nd, u_off, vn_dev, vp_dev);
      PECS_CUDA(cudaGetLastError());
      PECS_CUDA(cudaStreamSynchronize(s));
      return PECS_OK;
    }
    const long long n_tiles = (2LL * n_u + kWsOut - 1) / kWsOut, b_tiles = (batch + kWsRows - 1) / kWsRows;
    const long long z_parts = ((long long)(nd - n_u) + kWsZeros - 1) / kWsZeros;
    const long long blocks = n_tiles * b_tiles + 2LL * batch * z_parts;
    if (blocks > INT_MAX) throw PecsError(PECS_E_ARG, "batch too large");
    k_warm_start<<<(unsigned)blocks, 256, 0, s>>>(batch, r, n_u, c_dev, V_dev, mean_dev, nd, u_off, vn_dev, vp_dev,
                                                  (int)n_tiles, (int)b_tiles);
    PECS_CUDA(cudaGetLastError());
    PECS_CUDA(cudaStreamSynchronize(s));
  })
}

}  // extern "C"
