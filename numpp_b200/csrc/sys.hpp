// System-resident LU and substitution (orders above 32): launch interface.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "nppb_internal.hpp"

namespace nppb {

constexpr int kSysMaxN = 512;  // one CTA per system: 16 warps of 32 rows
constexpr int kSysOuter = 4;   // blocks of an outer block (orders above 512)

// Leading dimension of a factor workspace: rows start on 32-byte sectors.
__host__ __device__ inline int sys_ld(int n) { return (n + 3) & ~3; }
__host__ __device__ inline int sys_blocks(int n) { return (n + 31) / 32; }
// Doubles of the diagonal blocks' inverses: per 32-column block L11^-1, then U11^-1.
__host__ __device__ inline int64_t sys_dinv(int n) { return (int64_t)sys_blocks(n) * 2048; }

// CTAs per work item (a strip, a Cholesky factor): what the order needs (16 blocks
// of 32 rows each), more while the items leave SMs idle (of 148) and every CTA keeps at
// least four blocks (a warp for each scheduler).
inline int sys_cluster(int n, int64_t items) {
  const int nb = sys_blocks(n);
  int cs = 1;
  while (nb > 16 * cs) cs *= 2;
  while (cs < 8 && items * cs * 2 <= 148 && nb >= 8 * cs) cs *= 2;
  return cs;
}

// CTAs per system of an outer block's panel over `rows` rows: 16 blocks each at
// most, more while the clusters leave SMs idle (columns are faster with fewer
// warps per CTA) and 28 of the 148 SMs to the update beside the panel: 31, 34 and 37 systems
// of order 1024 take 2534, 2655 and 2739 us so, 2727, 3056 and 3171 us with clusters
// up to all of them.
inline int sys_outer_cluster(int rows, int64_t systems) {
  int cs = 2;
  while (sys_blocks(rows) > 16 * cs) cs *= 2;
  while (cs < 8 && systems * cs * 2 <= 120 && sys_blocks(rows) >= 8 * cs) cs *= 2;
  return cs;
}

// A strip of at most 32 columns of one system's right-hand sides or inverse.
struct SysItem {
  int32_t sys;
  int16_t inverse;  // 1: columns of the inverse
  int16_t width;
  int32_t c0;
  int32_t pad_;
};

// Systems of one launch. With desc: system list[i] (or i) has its own order and
// offsets. Without: a uniform batch of order un.
struct SysArgs {
  const SysDesc* desc;
  const double* A;      // input matrices, row-major, leading dimension n
  double* W;            // factors: row r of A's row order, leading dimension ldw
  int32_t* perm;        // position -> row of A (and of W, unless w_by_position)
  double* dinv;         // inverses of the diagonal blocks
  const double* B;
  double* X;            // X and inv null: nothing is solved for
  double* inv;
  double* det;
  double* sign;
  double* logabs;
  int32_t* info;        // per-system output (may be null)
  int32_t* state;       // first zero pivot + 1 or 0, by slot (null: every system is solved)
  int un, unrhs, uinv;  // uniform batch
  int w_by_position;    // W holds rows in pivoted order with leading dimension n (kept factors)
};

// LU with partial pivoting of `nsys` systems with (maximum order) nmax <= 512, a
// CTA each.
cudaError_t launch_sys_lu(const SysArgs& sa, const int32_t* list, int nsys, int nmax, cudaStream_t st);
// Uniform batches above order 512, in outer blocks [jb, je) of 32-column blocks:
// W <- A; the block's panel (pin: permutation so far, pout: with its pivots;
// running: three doubles per system); U12 and the trailing update on columns
// [c0, c1) with pout.
cudaError_t launch_sys_copy(const SysArgs& sa, int nsys, cudaStream_t st);
cudaError_t launch_sys_outer(const SysArgs& sa, const int32_t* pin, int32_t* pout, double* running, int nsys, int jb,
                             int je, cudaStream_t st);
cudaError_t launch_sys_update(const SysArgs& sa, const int32_t* perm, int nsys, int jb, int je, int c0, int c1,
                              cudaStream_t st);
// All of it, the next panel beside the update: sa.perm gets the final permutation;
// other: a second one, running: the panels' state.
cudaError_t run_sys_outer(const SysArgs& sa, int32_t* other, double* running, int nsys, cudaStream_t st);
// Forward and back substitution: `nitems` strips of one width class (8, 16 or 32
// columns at most; `width` = the widest), or every strip of a uniform batch.
inline int sys_width_class(int width) { return width <= 8 ? 0 : width <= 16 ? 1 : 2; }
cudaError_t launch_sys_solve(const SysArgs& sa, const SysItem* items, int64_t nitems, int width, int nmax,
                             cudaStream_t st);
cudaError_t launch_sys_solve_uniform(const SysArgs& sa, int nsys, cudaStream_t st);
// Permutations and diagonal inverses of a uniform batch's kept factors (swap lists
// ipiv): fills sa.perm and sa.dinv.
cudaError_t launch_sys_prepare(const SysArgs& sa, const int32_t* ipiv, int nsys, cudaStream_t st);
cudaError_t sys_prepare_kernels();

}  // namespace nppb
