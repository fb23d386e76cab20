// Device pieces of the system-resident kernels (k_sys.cu, k_chol.cu): operand
// rings, block updates and triangular inverses on the FP64 tensor core.
#pragma once

#include <cooperative_groups.h>

#include "dmma.cuh"
#include "sys.hpp"

namespace nppb {
namespace {

constexpr int US = 40;   // row stride of the 32 x 32 operand tiles (16-byte reads: banks 4g + t)
constexpr int BS = 34;   // row stride of the tile read down its columns (banks 4t + g)
constexpr int TS = 34;   // row stride of the inversions' scratch tile
constexpr int PS = 34;   // row stride of the panel staging tiles (16-byte reads, one row per thread)
constexpr int kMaxWarps = kSysMaxN / 32;
namespace cg = cooperative_groups;
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The rows of a warp's operand tile: lane 4g + t serves rows g, g+8, g+16, g+24.
struct Rows {
  unsigned off[4];  // byte offset of the row in W
  int live;         // rows from row g of the tile on: row group i exists when 8i < live
};

// A warp's operand ring: stages of eight columns of its 32 rows, 2 KB each. A
// lane fetches exactly what it will feed to the tensor core itself (columns
// 2t, 2t+1 of rows 8i + g), so the ring is a lane-private prefetch buffer
// (conflict-free, no barrier) that costs no registers. Three stages are in
// flight: 24 tensor instructions, 1500 cycles, cover the latency of L2.
constexpr int kRing = 4;
constexpr int kRingDoubles = kRing * 256;  // of one warp

// One row group of a stage: columns col, col + 1 of row 8i + g. EDGE: the columns
// may end inside the block (zeros past them).
template <bool VEC, bool EDGE>
__device__ __forceinline__ void ring_load1(unsigned ring, int stage, int i, const double* W, const Rows& r, int col,
                                           int n) {
  const unsigned d = ring + (stage * 4 + i) * 512;
  int size = 8 * i < r.live ? 16 : 0;
  if (EDGE) {
    size = min(size, 8 * max(0, n - col));
    col = min(col, (n - 1) & ~1);  // the address stays inside the row
  }
  const char* p = reinterpret_cast<const char*>(W + col) + r.off[i];
  if constexpr (VEC) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(size));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(p), "r"(min(size, 8)));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8), "l"(size > 8 ? p + 8 : p),
                 "r"(max(size - 8, 0)));
  }
}

// The first three stages of block K.
template <bool VEC, bool EDGE>
__device__ __forceinline__ void ring_start(unsigned ring, const double* W, const Rows& r, int K, int n, bool live) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (live) ring_load1<VEC, EDGE>(ring, q, i, W, r, 32 * K + 8 * q + 2 * (threadIdx.x & 3), n);
    cp_commit();
  }
}

// Everything a block step shares. NI: 8-column groups of the strip.
template <int NI>
struct Acc {
  double v[2][NI][4];  // rows 16m + g, 16m + g + 8; columns 8i + 2t, + 1
};

// The two halves of a cluster barrier, by whole warps. A CTA's shared memory may be
// written by a peer only once the CTA is known to run: kernels that push before
// their first cluster barrier arrive on entry and wait ahead of that push, so
// that their own loads cover the wait.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ unsigned smem(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ double2 lds2(unsigned p) {  // stays where it is written
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(p));
  return v;
}

// acc -= (warp's rows of W, columns 32K..32K+31) * U, with u the lane's place in
// -U^T (column c of U at c * US; the lane reads column g + 8i, rows 2t, 2t + 1).
// The ring holds the first three stages; those of block Knext follow when `more`. A tensor instruction holds the pipe for 64 cycles, so every
// register is reloaded for the next stage right behind its last use and the
// prefetches are spread between the instructions.
template <int NI, bool VEC, bool EDGE>
__device__ __forceinline__ void update(Acc<NI>& acc, unsigned ring, const double* W, const Rows& r,
                                       unsigned u, int K, int Knext, bool more, int n) {
  const int t2 = 2 * (threadIdx.x & 3);
  double2 a[4], b[NI];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = lds2(ring + i * 512);
#pragma unroll
  for (int i = 0; i < NI; ++i) b[i] = lds2(u + i * (8 * US * 8));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int stage = (q + 3) % 4, col = q == 0 ? 32 * K + 24 + t2 : 32 * Knext + 8 * (q - 1) + t2;
    const bool live = q == 0 || more;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i < NI) dmma1688(acc.v[0][i], a[0], a[1], b[i]);
      if (live) ring_load1<VEC, EDGE>(ring, stage, i, W, r, col, n);
    }
    cp_commit();
    cp_wait<2>();  // the next stage has landed
    const unsigned next = ring + (q + 1) * 2048;
    if (q < 3) {
      a[0] = lds2(next);
      a[1] = lds2(next + 512);
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      dmma1688(acc.v[1][i], a[2], a[3], b[i]);
      if (q < 3) b[i] = lds2(u + i * (8 * US * 8) + 64 * (q + 1));
    }
    if (q < 3) {
      a[2] = lds2(next + 1024);
      a[3] = lds2(next + 1536);
    }
  }
}

// Inverse of a 32 x 32 triangle by one warp; put(row, column, value) gets all of
// it, zeros included, lane = column. D (stride PS, shared) holds it: kUnitLower
// takes what lies below the diagonal, kUpper and kLower that half with the
// diagonal; rows and columns from kb on become the identity's. The upper triangle
// is inverted as the lower triangle U^T. X is a scratch tile of stride TS.
//
// First the four 8 x 8 diagonal blocks, a lane per column; then, twice, the
// square below two neighbouring triangles T11, T22 of 8 and of 16 rows:
// X21 = -X22 (T21 X11). One warp alone issues an instruction every four or five
// cycles, so what counts is how few there are: whole tiles, no element tests.
//
// CHECK: a product with the inverse leaves a residual of the order of
// eps max|T| max|T^-1| relative to the result, where substitution leaves eps. Up to
// kTriProduct the two agree within a factor of two (6e-16 against 4e-16, the worst
// of 4000 triangles of all scalings; 6e-15 at 1000, 6e-12 at 1e7); above it, or
// with an infinity or a NaN, put gets T itself (its diagonal as reciprocals) and a
// mark where a zero is otherwise, and whoever uses the block substitutes. Blocks of
// n I + N(0,1) lie at 1, of N(0,1) at 2 to 20 but for the last.
constexpr double kTriProduct = 32.0;
enum TriKind { kUnitLower, kUpper, kLower };
template <TriKind KIND, bool CHECK, class Put>
__device__ __forceinline__ void tri_inverse(double* D, double* X, int kb, Put put) {
  constexpr bool UPPER = KIND == kUpper, DIAG = KIND != kUnitLower;
  static_assert(!CHECK || KIND != kLower);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (kb < 32) {
    for (int r = 0; r < 32; ++r)
      if (r >= kb || lane >= kb) D[r * PS + lane] = r == lane ? 1.0 : 0.0;
    __syncwarp();
  }
  // element (i, j) of the lower triangle that is inverted, and of its inverse
  auto T = [&](int i, int j) { return UPPER ? D[j * PS + i] : D[i * PS + j]; };
  auto at = [&](int i, int j) -> double& { return UPPER ? X[j * TS + i] : X[i * TS + j]; };
  {
    const int b = lane & ~7, c = lane & 7;
    const double rd = DIAG ? 1.0 / D[lane * PS + lane] : 1.0;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i == c ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if constexpr (DIAG) x[q] *= __shfl_sync(kAll, rd, b + q);
#pragma unroll
      for (int i = q + 1; i < 8; ++i) x[i] = fma(-T(b + i, b + q), x[q], x[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) at(b + i, b + c) = x[i];  // zeros above the diagonal among them
  }
  __syncwarp();
  {  // the 8 x 8 squares at (8, 0) and (24, 16)
    double s[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, x[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int k = 0; k < 8; k += 4)
#pragma unroll
      for (int h = 0; h < 2; ++h) dmma884(s[h], T(16 * h + 8 + g, 16 * h + k + t), at(16 * h + k + t, 16 * h + g));
#pragma unroll
    for (int h = 0; h < 2; ++h)  // the sum's place is the result's
#pragma unroll
      for (int e = 0; e < 2; ++e) at(16 * h + 8 + g, 16 * h + 2 * t + e) = s[h][e];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 8; k += 4)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        dmma884(x[h], at(16 * h + 8 + g, 16 * h + 8 + k + t), at(16 * h + 8 + k + t, 16 * h + g));
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        at(16 * h + 8 + g, 16 * h + 2 * t + e) = -x[h][e];
        at(16 * h + g, 16 * h + 8 + 2 * t + e) = 0.0;
      }
  }
  __syncwarp();
  {  // the 16 x 16 square at (16, 0)
    double s[2][2][2], x[2][2][2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int ni = 0; ni < 2; ++ni) s[m][ni][0] = s[m][ni][1] = x[m][ni][0] = x[m][ni][1] = 0.0;
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      const double b[2] = {at(k + t, g), at(k + t, 8 + g)};
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double a = T(16 + 8 * m + g, k + t);
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) dmma884(s[m][ni], a, b[ni]);
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) at(16 + 8 * m + g, 8 * ni + 2 * t + e) = s[m][ni][e];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      const double b[2] = {at(16 + k + t, g), at(16 + k + t, 8 + g)};
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double a = at(16 + 8 * m + g, 16 + k + t);
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) dmma884(x[m][ni], a, b[ni]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) at(16 + 8 * m + g, 8 * ni + 2 * t + e) = -x[m][ni][e];
  }
  __syncwarp();
  if constexpr (CHECK) {
    // high words of the magnitudes, of the kb x kb triangle proper
    unsigned big_t = DIAG ? 0u : 0x3ff00000u, big_x = 0u;
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
      const bool in = (UPPER ? r <= lane && lane < kb : r >= lane && r < kb);
      const unsigned ht = (unsigned)__double2hiint(D[r * PS + lane]) & 0x7fffffffu;
      const unsigned hx = (unsigned)__double2hiint(X[r * TS + lane]) & 0x7fffffffu;
      if (in && (DIAG || r != lane)) big_t = max(big_t, ht);
      if (in) big_x = max(big_x, hx);
    }
    big_t = __reduce_max_sync(kAll, big_t);
    big_x = __reduce_max_sync(kAll, big_x);
    const bool fine = big_t < 0x7ff00000u && big_x < 0x7ff00000u &&
                      __hiloint2double((int)big_t, 0) * __hiloint2double((int)big_x, 0) <= kTriProduct;
    if (!fine) {
      // the diagonal as two factors of its reciprocal, both within range: a power of two
      // in its place, the reciprocal of the rest in columns 0 and 1, zeros otherwise
      double scale = 1.0, rest = 1.0;
      if constexpr (UPPER) {
        const double d = D[lane * PS + lane];
        const unsigned h = (unsigned)__double2hiint(d) & 0x7fffffffu;
        scale = h < 0x07b00000u ? 0x1p128 : h >= 0x78300000u ? 0x1p-128 : 1.0;  // 2^-900, 2^900
        rest = 1.0 / (d * scale);
      }
#pragma unroll 1
      for (int r = 0; r < 32; ++r) {
        const double v = D[r * PS + lane], q = __shfl_sync(kAll, rest, r);
        if constexpr (UPPER)
          put(r, lane, r < lane ? v : r == lane ? scale : lane == 0 ? q : r == 31 && lane == 1 ? 1.0 : 0.0);
        else
          put(r, lane, r > lane ? v : r == lane || (r == 0 && lane == 31) ? 1.0 : 0.0);
      }
      if constexpr (UPPER) {
        __syncwarp();
        if (lane == 0) put(2, 1, rest);
      }
      __syncwarp();
      return;
    }
  }
#pragma unroll 4
  for (int r = 0; r < 32; ++r) {
    const bool zero = UPPER ? (lane < 16 && r >= 16) : (lane >= 16 && r < 16);
    put(r, lane, zero ? 0.0 : X[r * TS + lane]);
  }
  __syncwarp();  // the callers' scratch becomes an operand ring, whose copies overwrite what other lanes read here
}

constexpr int kPerWarp = 32 * PS;  // doubles of a warp's region: its ring, or its staging tile
static_assert(kPerWarp >= kRingDoubles);

}  // namespace
}  // namespace nppb
