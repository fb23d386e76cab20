// Batched Cholesky factor of (count, n, n) FP64 stacks. C++20.
//
// The reference factors one matrix at a time, column by column, reading only
// the lower triangle and stopping with "Matrix is not positive definite" at a
// diagonal <= 0 (src/linalg/linalg.cpp:117-136; stacks batched.cpp:77). Here one
// CTA, or a cluster of up to eight, keeps one matrix for the whole factorisation,
// left-looking by 32-column blocks like the LU of k_sys.cu: block b of 32 rows
// belongs to warp b / CS of CTA b % CS. For block column J
//  1. the warps at or below it read their rows of A, negated, into the FP64
//     tensor core's accumulators (the lower triangle once),
//  2. add L_wK L_JK^T for every earlier block K: their own rows of L_wK through
//     their operand rings, L_JK shared through two alternating tiles,
//  3. the owner of block J factors its 32 x 32 block (a lane per row, groups of
//     eight columns, the rest of the block by the tensor core) and inverts it,
//  4. the warps below multiply by that inverse and write their rows of L.
// L serves as the working storage: no workspace, and A is read before the same
// columns of L are written, so L may be A.
//
// Half the operations of an LU and none of its pivot searches; the diagonal
// blocks, 32 dependent reciprocal square roots each, bound it while few systems
// share an SM. 512 x 256, one B200: 438 us, against 1489 us as an
// unpivoted LU scaled afterwards. Orders up to 32 take a warp each (k_chol_warp), orders
// above 2048 outer blocks (k_chol_update).
#include <algorithm>
#include <cmath>
#include <new>

#include "../../include/numpp_b200.h"
#include "runtime.hpp"
#include "sys_device.cuh"

namespace nppb {
namespace {

#define NPPB_CUDA(call, what)                            \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return cuda_status(e_, what); \
  } while (0)

template <class F>
int guarded(F&& f) {
  try {
    clear_error();
    return f();
  } catch (const std::bad_alloc&) {
    set_error("host allocation failed");
    return NPPB_E_NOMEM;
  }
}

// Minus the warp's rows of a 32-column block, columns up to the diagonal, into
// accumulators: two columns per load, all loads in flight at once (addresses are
// clamped into the matrix, values past the triangle become zero).
__device__ __forceinline__ void load_block(Acc<4>& acc, const double* A, bool vec, int blk, int col0, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double* src[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) src[i] = A + (int64_t)min(32 * blk + 8 * i + g, n - 1) * n;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
      const int col = col0 + 8 * ni + 2 * t;
      double2 x;
      if (vec) {  // uniform; n is even
        x = __ldcs(reinterpret_cast<const double2*>(src[i] + min(col, n - 2)));
      } else {
        x.x = __ldcs(src[i] + min(col, n - 1));
        x.y = __ldcs(src[i] + min(col + 1, n - 1));
      }
      acc.v[i >> 1][ni][2 * (i & 1)] = x.x;
      acc.v[i >> 1][ni][2 * (i & 1) + 1] = x.y;
    }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = 32 * blk + 8 * i + g, end = p >= n ? 0 : p + 1;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        double& v = acc.v[i >> 1][ni][2 * (i & 1) + e];
        v = col0 + 8 * ni + 2 * t + e < end ? -v : 0.0;
      }
  }
}

// Shared memory, in doubles: the inversion's scratch tile, a region per warp
// (ring / staging tile), and with more than one block the inverse and two tiles
// of L_JK.
constexpr int kScratch = 32 * TS;
constexpr int chol_smem(int warps, int blocks) {
  return 8 * (kScratch + warps * kPerWarp + (blocks > 1 ? 3 * 32 * US : 0));
}

// The 32 x 32 diagonal block by one warp, in its tile (stride PS), zeros above the
// diagonal. Eight columns at a time: every lane factors the 8 x 8 block on the
// diagonal for itself (no exchange between the dependent steps), solves its own
// row with it, and the tensor core updates the columns right of the group.
// Returns 0 or the first column whose diagonal is not positive, + 1.
__device__ __forceinline__ int factor_block(double* tile, int kb) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int j0 = 0; j0 < kb; j0 += 8) {
    double a[8], d[8][8], r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c <= i; c += 2) {
        const double2 x = *reinterpret_cast<const double2*>(tile + (j0 + i) * PS + j0 + c);
        d[i][c] = x.x;
        if (c < i) d[i][c + 1] = x.y;
      }
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 x = *reinterpret_cast<const double2*>(tile + lane * PS + j0 + c);
      a[c] = x.x;
      a[c + 1] = x.y;
    }
    int bad = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      if (j0 + s < kb && !bad && !(d[s][s] > 0.0)) bad = j0 + s + 1;  // a NaN included
      r[s] = j0 + s < kb ? rsqrt(d[s][s]) : 1.0;
      a[s] *= r[s];
#pragma unroll
      for (int i = s + 1; i < 8; ++i) d[i][s] *= r[s];
#pragma unroll
      for (int k = s + 1; k < 8; ++k) {
        a[k] = fma(-a[s], d[k][s], a[k]);
#pragma unroll
        for (int i = k; i < 8; ++i) d[i][k] = fma(-d[i][s], d[k][s], d[i][k]);
      }
    }
    if (bad) return bad;  // the same in every lane
    // the lane's own diagonal: d times the reciprocal root, corrected once, so that
    // squares give their roots exactly (and an infinity stays one)
    double dd = 1.0, rr = 1.0;
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (lane == j0 + s) {
        dd = d[s][s];
        rr = r[s];
      }
    const double q = dd * rr, root = isinf(dd) ? dd : fma(0.5 * rr, fma(-q, q, dd), q);
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (lane == j0 + s) a[s] = root;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 8; c += 2)
      *reinterpret_cast<double2*>(tile + lane * PS + j0 + c) =
          make_double2(j0 + c <= lane ? a[c] : 0.0, j0 + c + 1 <= lane ? a[c + 1] : 0.0);
    __syncwarp();
    double2 l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      l[i] = *reinterpret_cast<const double2*>(tile + (8 * i + g) * PS + j0 + 2 * t);
      l[i].x = -l[i].x;
      l[i].y = -l[i].y;
    }
    for (int c0 = j0 + 8; c0 < kb; c0 += 8) {  // columns c0 .. c0 + 7: their rows are the operand
      const double2 b = *reinterpret_cast<const double2*>(tile + (c0 + g) * PS + j0 + 2 * t);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        double* o = tile + (16 * m + g) * PS + c0 + 2 * t;
        const double2 lo = *reinterpret_cast<const double2*>(o), hi = *reinterpret_cast<const double2*>(o + 8 * PS);
        double v[4] = {lo.x, lo.y, hi.x, hi.y};
        dmma1688(v, l[2 * m], l[2 * m + 1], b);
        *reinterpret_cast<double2*>(o) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(o + 8 * PS) = make_double2(v[2], v[3]);
      }
    }
    __syncwarp();
  }
  for (int c = (kb + 7) & ~7; c < 32; ++c) tile[lane * PS + c] = 0.0;  // past the last group
  __syncwarp();
  return 0;
}

// Orders up to 32: a warp per system, as many warps to a CTA (at most four) as leave
// every SM a CTA. A CTA of k_sys_chol per system instead takes 148 us for 40000 systems
// of order 4 and 209 of order 9.
__global__ void __launch_bounds__(128)
k_chol_warp(const double* A, double* L, int32_t* __restrict__ info, int count, int n) {
  extern __shared__ __align__(16) double sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, z = blockIdx.x * (blockDim.x >> 5) + warp;
  if (z >= count) return;
  double* tile = sm + warp * 32 * PS;
  A += (int64_t)z * n * n;
  L += (int64_t)z * n * n;
  {
    double x[32];
#pragma unroll
    for (int r = 0; r < 32; ++r) x[r] = r < n && lane <= r ? __ldcs(A + r * n + lane) : 0.0;
#pragma unroll
    for (int r = 0; r < 32; ++r) tile[r * PS + lane] = x[r];
  }
  __syncwarp();
  const int bad = factor_block(tile, n);
  if (lane == 0) info[z] = bad;
  if (bad || lane >= n) return;
#pragma unroll 8
  for (int r = 0; r < n; ++r) L[r * n + lane] = tile[r * PS + lane];
}

template <bool VEC, int CS>
__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_chol(const double* A, double* L, int32_t* __restrict__ info, int n, int jb, int je) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_fail;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3, nb = sys_blocks(n);
  const int rank = CS > 1 ? (int)blockIdx.x % CS : 0;
  const int64_t z = (int)blockIdx.x / CS;
  const int blk = jb + warp * CS + rank;
  if (jb > 0 && info[z]) return;  // read ahead of the barrier that a writer has passed: the same in every CTA
  double* scratch = sm;
  double* tile = sm + kScratch + warp * kPerWarp;
  double* Li = sm + kScratch + nw * kPerWarp;
  double* Bt = Li + 32 * US;
  const unsigned ring = smem(tile) + 16 * lane;
  A += z * n * n;
  L += z * n * n;
  const bool avec = n % 2 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  auto sync = [] {
    if constexpr (CS > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  // rows 32J .. 32J + 31 of L, columns of block K, into tile K & 1
  auto fetch_rows = [&](int J, int K) {
    double* b = Bt + (K & 1) * 32 * US;
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
      const int r = i >> 4, c = (i & 15) * 2, p = 32 * J + r;
      const double* src = L + (int64_t)min(p, n - 1) * n + 32 * K + c;
      const unsigned d = smem(b + r * US + c);
      if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(p < n ? 16 : 0));
      } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(p < n ? 8 : 0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8), "l"(src + 1), "r"(p < n ? 8 : 0));
      }
    }
    cp_commit();
  };
  if (threadIdx.x == 0) s_fail = 0;
  sync();

  Rows r;
  r.live = n - 32 * blk - g;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = 32 * blk + 8 * i + g;
    r.off[i] = (unsigned)(p < n ? p : 0) * n * 8;
  }
  for (int J = jb; J < je; ++J) {
    const int kb = min(32, n - 32 * J);
    const bool active = blk >= J && blk < nb;
    Acc<4> acc;
    if (active) load_block(acc, A, avec, blk, 32 * J, n);
    if (blk > J && J + 1 < nb && 32 * blk + lane < n) {  // the next column block on its way into L2
      const double* nx = A + (int64_t)(32 * blk + lane) * n + 32 * (J + 1);
      const int left = min(32 * blk + lane, n - 1) - 32 * (J + 1);  // up to the diagonal
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx));
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(16, left)));
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(31, left)));
    }
    if (J > jb) {
      fetch_rows(J, jb);
      ring_start<VEC, false>(ring, L, r, jb, n, active);
      for (int K = jb; K < J; ++K) {
        cp_wait<2>();     // L_JK; at most two operand stages stay in flight
        __syncthreads();  // and every warp is done with the other tile
        if (K + 1 < J) fetch_rows(J, K + 1);
        else cp_commit();
        if (active) {
          update<4, VEC, false>(acc, ring, L, r, smem(Bt + (K & 1) * 32 * US + g * US + 2 * t), K, K + 1, K + 1 < J, n);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) cp_commit();  // the waits count groups
        }
      }
      cp_wait<0>();
      __syncwarp();  // the ring becomes the staging tile
    }
    if (active) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          double* o = tile + (16 * m + g) * PS + 8 * ni + 2 * t;
          *reinterpret_cast<double2*>(o) = make_double2(-acc.v[m][ni][0], -acc.v[m][ni][1]);
          *reinterpret_cast<double2*>(o + 8 * PS) = make_double2(-acc.v[m][ni][2], -acc.v[m][ni][3]);
        }
      __syncwarp();
    }
    if (blk == J) {
      const int bad = factor_block(tile, kb);
      if (bad) {
        if (lane == 0) {
          info[z] = 32 * J + bad;
#pragma unroll
          for (int c = 0; c < CS; ++c) *(CS > 1 ? cg::this_cluster().map_shared_rank(&s_fail, c) : &s_fail) = 1;
        }
      } else if (J + 1 < nb) {
        tri_inverse<kLower, false>(tile, scratch, kb, [&](int row, int col, double v) {
#pragma unroll
          for (int c = 0; c < CS; ++c)
            (CS > 1 ? cg::this_cluster().map_shared_rank(Li, c) : Li)[row * US + col] = v;
        });
      }
    }
    sync();  // the inverse is everywhere
    if (s_fail) return;  // the same in every CTA of the cluster
    if (active && blk > J) {
      // rows times the inverse's transpose: L_JJ^-1 [n][k] = 0 for k > n
      Acc<4> out;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int e = 0; e < 4; ++e) out.v[m][ni][e] = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double2 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const double2*>(tile + (8 * i + g) * PS + 8 * q + 2 * t);
#pragma unroll
        for (int ni = q; ni < 4; ++ni) {
          const double2 b = *reinterpret_cast<const double2*>(Li + (8 * ni + g) * US + 8 * q + 2 * t);
#pragma unroll
          for (int m = 0; m < 2; ++m) dmma1688(out.v[m][ni], a[2 * m], a[2 * m + 1], b);
        }
      }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          double* o = tile + (16 * m + g) * PS + 8 * ni + 2 * t;
          *reinterpret_cast<double2*>(o) = make_double2(out.v[m][ni][0], out.v[m][ni][1]);
          *reinterpret_cast<double2*>(o + 8 * PS) = make_double2(out.v[m][ni][2], out.v[m][ni][3]);
        }
      __syncwarp();
    }
    if (blk < nb) {
      // the factor's rows, zeros above the diagonal
      double* o = L + (int64_t)32 * blk * n + 32 * J + lane;
      const int rows = lane < kb ? min(32, n - 32 * blk) : 0;
#pragma unroll 16
      for (int rr = 0; rr < 32; ++rr)
        if (rr < rows) o[(int64_t)rr * n] = blk >= J ? tile[rr * PS + lane] : 0.0;
    }
    if (J + 1 < je) sync();  // this column of L before the next one reads it
  }
  if (jb == 0 && threadIdx.x == 0 && rank == 0) info[z] = 0;
}

// Orders above 2048: outer blocks of 128 columns. k_sys_chol factors a block's columns
// over all rows below (left-looking inside it), k_chol_update subtracts their
// products from the rest of the lower triangle. One cluster for the whole matrix
// keeps 8 SMs busy: 24.5 ms for one matrix of order 4096, where the unpivoted LU on the step
// kernels had taken 12.
//
// Rows 32 je .. n - 1 minus L_21 L_21^T on and below the diagonal, K = 128: a CTA per
// 128 x 64 tile (grid.z = system), slabs of 16 columns of both row ranges through a
// ring of three, as in k_sys_gemm. src: A for the first block, L after it.
constexpr int CM = 128, CN = 64, CK = 16, CSTAGES = 3;
constexpr int kCholSlab = (CM + CN) * CK;
constexpr int kCholUpdateSmem = 8 * CSTAGES * kCholSlab;

template <bool VEC>
__global__ void __launch_bounds__(256, 2)
k_chol_update(const double* src, double* L, const int32_t* __restrict__ info, int n, int jb, int je) {
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int64_t z = blockIdx.z;
  const int row0 = 32 * je + CM * (int)blockIdx.y, col0 = 32 * je + CN * (int)blockIdx.x;
  if (col0 >= row0 + CM || info[z]) return;  // above the diagonal; not positive definite
  src += z * n * n;
  L += z * n * n;
  // 192 rows of a slab (128 of the tile's rows, then 64 of its columns); 16-byte piece
  // c of row r at piece c ^ 4 (r & 1): neighbouring rows fall into the two halves of the banks
  auto load = [&](int slab) {
    double* a = sm + slab % CSTAGES * kCholSlab;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int idx = tid + 256 * i, r = idx >> 3, c = idx & 7;
      const int row = r < CM ? row0 + r : col0 + r - CM;
      const double* p = L + (int64_t)min(row, n - 1) * n + 32 * jb + CK * slab + 2 * c;
      const unsigned d = smem(a + r * CK + 2 * (c ^ 4 * (r & 1)));
      if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(row < n ? 16 : 0));
      } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(p), "r"(row < n ? 8 : 0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8), "l"(p + 1), "r"(row < n ? 8 : 0));
      }
    }
    cp_commit();
  };
  constexpr int kSlabs = 128 / CK;
  load(0);
  load(1);
  const int wm = 32 * (warp >> 1), wn = 32 * (warp & 1);
  double acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + wm + 16 * m + 8 * (e >> 1) + g, col = col0 + wn + 8 * ni + 2 * t + (e & 1);
        acc[m][ni][e] = row < n && col <= row ? -src[(int64_t)row * n + col] : 0.0;
      }
  for (int k = 0; k < kSlabs; ++k) {
    cp_wait<1>();
    __syncthreads();  // slab k is here, and slab k - 1 has been read
    if (k + 2 < kSlabs) load(k + 2);
    else cp_commit();
    const double* a = sm + k % CSTAGES * kCholSlab;
    const double* b = a + CM * CK;
#pragma unroll
    for (int q = 0; q < CK / 8; ++q) {
      double2 av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = wm + 8 * i + g, c = wn + 8 * i + g;
        av[i] = *reinterpret_cast<const double2*>(a + r * CK + 2 * ((4 * q + t) ^ 4 * (r & 1)));
        bv[i] = *reinterpret_cast<const double2*>(b + c * CK + 2 * ((4 * q + t) ^ 4 * (c & 1)));
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
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + wm + 16 * m + 8 * (e >> 1) + g, col = col0 + wn + 8 * ni + 2 * t + (e & 1);
        if (row < n && col <= row) L[(int64_t)row * n + col] = -acc[m][ni][e];
      }
}

// Zeros right of each row's 128-column diagonal block (the outer blocks write the rest).
__global__ void __launch_bounds__(256) k_chol_zeros(double* L, int n) {
  const int row = blockIdx.x, end = min(n, (row / 128 + 1) * 128);
  double* o = L + ((int64_t)blockIdx.y * n + row) * n;
  for (int c = end + threadIdx.x; c < n; c += 256) o[c] = 0.0;
}

template <bool VEC, int CS>
cudaError_t chol_prepare1() {
  return cudaFuncSetAttribute(k_sys_chol<VEC, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              chol_smem(kMaxWarps, 2));
}

// Columns of the blocks [jb, je).
template <bool VEC, int CS>
cudaError_t launch_chol(const double* A, double* L, int32_t* info, int64_t count, int n, int jb, int je,
                        cudaStream_t st) {
  const int nb = sys_blocks(n) - jb, nw = (nb + CS - 1) / CS;
  cudaError_t e = chol_prepare1<VEC, CS>();
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * CS));
  cfg.blockDim = dim3(32 * nw);
  cfg.dynamicSmemBytes = chol_smem(nw, nb);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_sys_chol<VEC, CS>, A, L, info, n, jb, je);
}

template <bool VEC>
cudaError_t launch_chol(const double* A, double* L, int32_t* info, int64_t count, int n, int jb, int je,
                        cudaStream_t st) {
  switch (sys_cluster(n - 32 * jb, count)) {
    case 1: return launch_chol<VEC, 1>(A, L, info, count, n, jb, je, st);
    case 2: return launch_chol<VEC, 2>(A, L, info, count, n, jb, je, st);
    case 4: return launch_chol<VEC, 4>(A, L, info, count, n, jb, je, st);
    default: return launch_chol<VEC, 8>(A, L, info, count, n, jb, je, st);
  }
}

template <bool VEC>
cudaError_t run_chol_outer(const double* A, double* L, int32_t* info, int64_t count, int n, cudaStream_t st) {
  constexpr int kOuter = 4;
  const int nb = sys_blocks(n);
  cudaError_t e = cudaFuncSetAttribute(k_chol_update<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kCholUpdateSmem);
  for (int jb = 0; jb < nb && e == cudaSuccess; jb += kOuter) {
    const int je = std::min(nb, jb + kOuter), rest = n - 32 * je;
    const double* src = jb ? L : A;
    e = launch_chol<VEC>(src, L, info, count, n, jb, je, st);
    if (e != cudaSuccess || rest <= 0) break;
    const dim3 grid((unsigned)(rest + CN - 1) / CN, (unsigned)(rest + CM - 1) / CM, (unsigned)count);
    k_chol_update<VEC><<<grid, 256, kCholUpdateSmem, st>>>(src, L, info, n, jb, je);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  // behind every reader of A, which may be L
  k_chol_zeros<<<dim3((unsigned)n, (unsigned)count), 256, 0, st>>>(L, n);
  return cudaGetLastError();
}

int cholesky_device(int64_t count, int32_t n, const double* dA, double* dL, int32_t* dinfo, cudaStream_t st) {
  if (count * sys_cluster(n, count) > INT32_MAX) {
    set_error("batch count above 2^31-1");
    return NPPB_E_RANGE;
  }
  const bool vec = n % 2 == 0 && (reinterpret_cast<uintptr_t>(dL) & 15) == 0;
  const int nb = sys_blocks(n);
  if (n <= 32) {
    const int w = (int)std::min<int64_t>(4, (count + 147) / 148);
    k_chol_warp<<<(unsigned)((count + w - 1) / w), 32 * w, w * 32 * PS * (int)sizeof(double), st>>>(dA, dL, dinfo,
                                                                                                  (int)count, n);
    NPPB_CUDA(cudaGetLastError(), "factorisation");
  } else if (n > 2048 && count <= 65535)
    NPPB_CUDA((vec ? run_chol_outer<true>(dA, dL, dinfo, count, n, st)
                   : run_chol_outer<false>(dA, dL, dinfo, count, n, st)),
              "factorisation");
  else
    NPPB_CUDA((vec ? launch_chol<true>(dA, dL, dinfo, count, n, 0, nb, st)
                   : launch_chol<false>(dA, dL, dinfo, count, n, 0, nb, st)),
              "factorisation");
  return NPPB_OK;
}

int check_args(int64_t count, int32_t n) {
  if (count < 0 || n < 0) {
    set_error("negative count or order");
    return NPPB_E_ARG;
  }
  if (count > INT32_MAX) {
    set_error("batch count above 2^31-1");
    return NPPB_E_RANGE;
  }
  if (n > kStepMaxN) {
    set_error("order above 4096 is not served by the batched path");
    return NPPB_E_RANGE;
  }
  return NPPB_OK;
}

}  // namespace
}  // namespace nppb

using namespace nppb;

extern "C" {

int nppb_d_cholesky_batched(int64_t count, int32_t n, const double* dA, double* dL, int32_t* dinfo,
                            void* stream) {
  return guarded([&]() -> int {
    const int rc = check_args(count, n);
    if (rc != NPPB_OK) return rc;
    if (!count || !n) return NPPB_OK;
    if (!dA || !dL || !dinfo) {
      set_error("cholesky needs A, L and info");
      return NPPB_E_ARG;
    }
    if (!device()) return NPPB_E_NODEV;
    return cholesky_device(count, n, dA, dL, dinfo, static_cast<cudaStream_t>(stream));
  });
}

int nppb_cholesky_batched(int64_t count, int32_t n, const double* A, double* L, int32_t* info) {
  return guarded([&]() -> int {
    const int rc = check_args(count, n);
    if (rc != NPPB_OK) return rc;
    if (!count || !n) return NPPB_OK;
    if (!A || !L || !info) {
      set_error("cholesky needs A, L and info");
      return NPPB_E_ARG;
    }
    if (!device()) return NPPB_E_NODEV;
    cudaStream_t st = thread_stream();
    const size_t nn = (size_t)count * n * n;
    DevMem dA, dL, dI;
    NPPB_CUDA(dA.alloc(sizeof(double) * nn, st), "allocation");
    NPPB_CUDA(dL.alloc(sizeof(double) * nn, st), "allocation");
    NPPB_CUDA(dI.alloc(sizeof(int32_t) * count, st), "allocation");
    NPPB_CUDA(cudaMemcpyAsync(dA.as<double>(), A, sizeof(double) * nn, cudaMemcpyHostToDevice, st), "copy");
    const int r = cholesky_device(count, n, dA.as<double>(), dL.as<double>(), dI.as<int32_t>(), st);
    if (r != NPPB_OK) return r;
    NPPB_CUDA(cudaMemcpyAsync(L, dL.as<double>(), sizeof(double) * nn, cudaMemcpyDeviceToHost, st), "copy");
    NPPB_CUDA(cudaMemcpyAsync(info, dI.as<int32_t>(), sizeof(int32_t) * count, cudaMemcpyDeviceToHost, st), "copy");
    NPPB_CUDA(cudaStreamSynchronize(st), "synchronize");
    NPPB_CUDA(cudaGetLastError(), "kernel");
    return NPPB_OK;
  });
}

}  // extern "C"
