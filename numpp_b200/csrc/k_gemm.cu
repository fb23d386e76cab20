// Row-major GEMM for the GpuVTable::gemm slot (include/numpp/backend/gpu_vtable.hpp
// in NumPP: C[m,n] = A[m,k] B[k,n], accumulated in k order per output element).
//
// FP64: 128x64 CTA tile, 8 warps of 32x32, DMMA m16n8k8; K is staged 16 deep in
// shared memory through a ring of three slabs (cp.async: global -> shared without
// a register round trip), so two slabs are on their way while the tensor pipe
// works on the current one.
// FP32: SIMT 64x64 tile, 4x4 outputs per thread (the float32 form of the slot).
#include <algorithm>

#include "dmma.cuh"
#include "nppb_internal.hpp"

namespace nppb {
namespace {

constexpr int BM = 128, BN = 64, BK = 16, STAGES = 3;
constexpr int NT = 256;
constexpr int BS = BN + 2;  // row stride of a B slab (8-byte reads down a column: banks 4t + g)
constexpr int SLAB = BM * BK + BK * BS;
constexpr int kGemmSmem = 8 * STAGES * SLAB;

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool pred) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = pred ? 8 : 0;  // 0 source bytes = zero fill
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async16(double* smem, const double* gmem, bool pred) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// blockIdx.z walks a strided batch (sA, sB, sC elements apart; 0 for one GEMM).
// Bound: the FP64 tensor pipe (a tile's eight warps hold it 0.52 us per slab of an
// SM). m16n8k8 holds the pipe as long as its four m8n8k4 and takes half the
// operand reads; slabs of 16 leave a barrier per 16 products of a warp instead of
// per 32 small ones, and two slabs are in flight behind the one in use. 1024
// products of 128 x 128 x 128: 200 us with m8n8k4 and
// slabs of 8, 150 us so (28.7 TFLOP/s).
// VEC: every row start, and so every pair of columns, is 16-byte aligned, and K
// and N are even (a pair is in or out as one): copies of 16 bytes, half the copies
// of the 8-byte form that serves everything else.
// Warps whose 32 x 32 part lies outside C only copy.
template <bool VEC>
__global__ void __launch_bounds__(NT, 2)
k_gemm_f64(int64_t M, int64_t N, int64_t K, const double* __restrict__ A, int64_t lda,
           const double* __restrict__ B, int64_t ldb, double* __restrict__ C, int64_t ldc, int64_t sA,
           int64_t sB, int64_t sC, int64_t z0) {
  extern __shared__ __align__(16) double sm[];
  {
    const int64_t z = z0 + blockIdx.z;
    A += z * sA;
    B += z * sB;
    C += z * sC;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t bm = (int64_t)blockIdx.y * BM, bn = (int64_t)blockIdx.x * BN;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;  // 4 x 2 warps
  const bool live = bm + wm < M && bn + wn < N;

  // A slab: 16-byte piece c of row r at piece c ^ 4 (r & 1), so that two neighbouring
  // rows fall into the two halves of the banks
  auto load = [&](int64_t slab) {
    double* a = sm + slab % STAGES * SLAB;
    double* b = a + BM * BK;
    const int64_t k0 = slab * BK;
#pragma unroll
    for (int i = 0; i < (BM * BK) / (2 * NT); ++i) {
      const int idx = tid + i * NT, r = idx >> 3, c = idx & 7;
      const int64_t gr = bm + r, gc = k0 + 2 * c;
      double* dst = a + r * BK + 2 * (c ^ 4 * (r & 1));
      const double* src = A + gr * lda + gc;
      if constexpr (VEC) {
        const bool ok = gr < M && gc < K;
        cp_async16(dst, ok ? src : A, ok);
      } else {
        const bool ok0 = gr < M && gc < K, ok1 = gr < M && gc + 1 < K;
        cp_async8(dst, ok0 ? src : A, ok0);
        cp_async8(dst + 1, ok1 ? src + 1 : A, ok1);
      }
    }
#pragma unroll
    for (int i = 0; i < (BK * BN) / (2 * NT); ++i) {
      const int idx = tid + i * NT, r = idx >> 5, c = (idx & 31) * 2;
      const int64_t gr = k0 + r, gc = bn + c;
      double* dst = b + r * BS + c;
      const double* src = B + gr * ldb + gc;
      if constexpr (VEC) {
        const bool ok = gr < K && gc < N;
        cp_async16(dst, ok ? src : B, ok);
      } else {
        const bool ok0 = gr < K && gc < N, ok1 = gr < K && gc + 1 < N;
        cp_async8(dst, ok0 ? src : B, ok0);
        cp_async8(dst + 1, ok1 ? src + 1 : B, ok1);
      }
    }
    cp_async_commit();
  };

  double acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][ni][e] = 0.0;

  const int64_t nk = (K + BK - 1) / BK;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (i < nk) load(i);
    else cp_async_commit();
  }
  for (int64_t k = 0; k < nk; ++k) {
    cp_async_wait<1>();
    __syncthreads();  // slab k is here, and slab k - 1 has been read
    if (k + 2 < nk) load(k + 2);
    else cp_async_commit();
    if (!live) continue;
    const double* a = sm + k % STAGES * SLAB;
    const double* b = a + BM * BK;
#pragma unroll
    for (int q = 0; q < BK / 8; ++q) {
      double2 av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = wm + 8 * i + g;
        av[i] = *reinterpret_cast<const double2*>(a + r * BK + 2 * ((4 * q + t) ^ 4 * (r & 1)));
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const double* p = b + (8 * q + 2 * t) * BS + wn + 8 * ni + g;
        bv[ni] = make_double2(p[0], p[BS]);
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma1688(acc[m][ni], av[2 * m], av[2 * m + 1], bv[ni]);
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t row = bm + wm + 16 * m + 8 * h + g;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int64_t col = bn + wn + 8 * ni + 2 * t;
        double* c = C + row * ldc + col;
        if constexpr (VEC) {
          if (row < M && col < N)
            *reinterpret_cast<double2*>(c) = make_double2(acc[m][ni][2 * h], acc[m][ni][2 * h + 1]);
        } else {
          if (row < M && col < N) c[0] = acc[m][ni][2 * h];
          if (row < M && col + 1 < N) c[1] = acc[m][ni][2 * h + 1];
        }
      }
    }
}

// Whether every row of the three operands starts on a 16-byte boundary and no
// pair of columns is cut by K or N.
bool gemm_pairs(int64_t N, int64_t K, const double* A, int64_t lda, const double* B, int64_t ldb, const double* C,
                int64_t ldc, int64_t sA, int64_t sB, int64_t sC) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C);
  return p % 16 == 0 && ((N | K | lda | ldb | ldc | sA | sB | sC) & 1) == 0;
}

constexpr int FT = 64;
__global__ void __launch_bounds__(256)
k_gemm_f32(int64_t M, int64_t N, int64_t K, const float* __restrict__ A,
           const float* __restrict__ B, float* __restrict__ C) {
  __shared__ float As[16][FT + 1];
  __shared__ float Bs[16][FT + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t bm = (int64_t)blockIdx.y * FT, bn = (int64_t)blockIdx.x * FT;
  float acc[4][4] = {};
  for (int64_t k0 = 0; k0 < K; k0 += 16) {
    for (int i = threadIdx.x; i < FT * 16; i += 256) {
      const int r = i / 16, c = i % 16;
      const int64_t gr = bm + r, gc = k0 + c;
      As[c][r] = (gr < M && gc < K) ? A[gr * K + gc] : 0.f;
      const int rb = i / FT, cb = i % FT;
      const int64_t hr = k0 + rb, hc = bn + cb;
      Bs[rb][cb] = (hr < K && hc < N) ? B[hr * N + hc] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t r = bm + ty + 16 * i, c = bn + tx + 16 * j;
      if (r < M && c < N) C[r * N + c] = acc[i][j];
    }
}

}  // namespace

cudaError_t gemm_prepare() {
  cudaError_t e = cudaFuncSetAttribute(k_gemm_f64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_gemm_f64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
  return e;
}

cudaError_t launch_gemm_f64(int64_t m, int64_t n, int64_t k, const double* A, int64_t lda,
                            const double* B, int64_t ldb, double* C, int64_t ldc,
                            cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  dim3 grid((unsigned)((n + BN - 1) / BN), (unsigned)((m + BM - 1) / BM));
  const bool vec = gemm_pairs(n, k, A, lda, B, ldb, C, ldc, 0, 0, 0);
  const auto kernel = vec ? k_gemm_f64<true> : k_gemm_f64<false>;
  kernel<<<grid, NT, kGemmSmem, st>>>(m, n, k, A, lda, B, ldb, C, ldc, 0, 0, 0, 0);
  return cudaGetLastError();
}

cudaError_t launch_gemm_f64_batched(int64_t batch, int64_t m, int64_t n, int64_t k, const double* A,
                                    const double* B, double* C, cudaStream_t st) {
  if (m <= 0 || n <= 0 || batch <= 0) return cudaSuccess;
  const unsigned gx = (unsigned)((n + BN - 1) / BN), gy = (unsigned)((m + BM - 1) / BM);
  const bool vec = gemm_pairs(n, k, A, k, B, n, C, n, m * k, k * n, m * n);
  const auto kernel = vec ? k_gemm_f64<true> : k_gemm_f64<false>;
  for (int64_t z0 = 0; z0 < batch; z0 += 65535) {
    const dim3 grid(gx, gy, (unsigned)std::min<int64_t>(65535, batch - z0));
    kernel<<<grid, NT, kGemmSmem, st>>>(m, n, k, A, k, B, n, C, n, m * k, k * n, m * n, z0);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_gemm_f32(int64_t m, int64_t n, int64_t k, const float* A, const float* B,
                            float* C, cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  dim3 grid((unsigned)((n + FT - 1) / FT), (unsigned)((m + FT - 1) / FT));
  k_gemm_f32<<<grid, 256, 0, st>>>(m, n, k, A, B, C);
  return cudaGetLastError();
}

}  // namespace nppb
