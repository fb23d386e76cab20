// System-resident LU and substitution: orders 33..512, one CTA per system.
//
// The reference factors one matrix by an unblocked right-looking elimination
// (src/linalg/linalg.cpp:48-71) and then substitutes (:73-90). Here one CTA keeps
// one system for the whole factorisation, left-looking by 32-column blocks:
// warp w owns the 32 rows at positions 32w..32w+31 of the pivoted order. For
// block column J it
//  1. reads its rows of the column block of A straight into the FP64 tensor
//     core's accumulator layout (every element of A is read once),
//  2. takes the earlier blocks K < J in turn: the rows at block K's positions
//     become U_KJ = L_KK^-1 A_KJ (shared memory, all warps), and every warp
//     below subtracts L_wK U_KJ, its own rows of L_wK coming from memory three
//     eight-column stages ahead of the tensor core,
//  3. factors what is left of the column block with one row per thread in
//     registers (panel()).
// Rows never move: a row stays where A has it, its position is a label, and the
// factors W hold row r of A in row r, so no exchange pass over the other columns
// exists. The factors are written once; the right-looking form this replaces
// read and wrote the whole trailing matrix once per 32 columns, in three
// launches per step.
//
// Substitution (k_sys_solve) is the same loop on a strip of at most 32
// right-hand sides or inverse columns: forward through the blocks with
// L_KK^-1, back with U_KK^-1, in one launch.
//
// What bounds it: FP64 tensor throughput in 2 (mma.m16n8k8, 64 FMA per cycle
// and SM), the dependent pivot steps in 3.
#include <climits>
#include <cmath>

#include "dmma.cuh"
#include "sys.hpp"

namespace nppb {
namespace {

constexpr int TS = 36;   // row stride of the 32 x 32 tiles read as mma operands (banks 4g + tq)
constexpr int US = 40;   // row stride of the transposed U tile (16-byte reads: banks 4g + tq)
constexpr int PS = 33;   // row stride of the panel staging tiles (one row per thread)
constexpr int kMaxWarps = kSysMaxN / 32;
constexpr unsigned kAll = 0xffffffffu;

// D(16x8) += A(16x8) B(8x8), FP64, one warp. Lane 4g + t holds A[g][t],
// A[g+8][t], A[g][t+4], A[g+8][t+4]; B[t][g], B[t+4][g]; D[g][2t], D[g][2t+1],
// D[g+8][2t], D[g+8][2t+1]. The k index may be permuted alike on both sides:
// the callers take k = 2t for slot t and 2t + 1 for slot t + 4, so that a lane's
// two values lie side by side.
__device__ __forceinline__ void dmma1688(double (&d)[4], double2 lo, double2 hi, double2 b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(lo.x), "d"(hi.x), "d"(lo.y), "d"(hi.y), "d"(b.x), "d"(b.y));
}

struct View {  // one system of the launch
  int n, nrhs, ldw, idx, slot;
  const double* A;
  double* W;
  int32_t* perm;
  double* dinv;
  int64_t b_off, inv_off;
};

__device__ __forceinline__ View view(const SysArgs& sa, int s) {
  View v;
  if (sa.desc) {
    const SysDesc d = sa.desc[s];
    v.n = d.n;
    v.nrhs = d.nrhs;
    v.idx = d.idx;
    v.slot = d.pad_;
    v.A = sa.A + d.a_off;
    v.W = sa.W + d.lu_off;
    v.perm = sa.perm + d.perm_off;
    v.dinv = sa.dinv + d.dinv_off;
    v.b_off = d.b_off;
    v.inv_off = d.inv_off;
  } else {
    const int64_t n = sa.un;
    v.n = sa.un;
    v.nrhs = sa.unrhs;
    v.idx = v.slot = s;
    v.A = sa.A + s * n * n;
    v.W = sa.W + s * n * (sa.w_by_position ? n : sys_ld(sa.un));
    v.perm = sa.perm + s * n;
    v.dinv = sa.dinv + s * sys_dinv(sa.un);
    v.b_off = s * n * sa.unrhs;
    v.inv_off = s * n * n;
  }
  v.ldw = sa.w_by_position ? v.n : sys_ld(v.n);
  return v;
}

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bar_active(int threads) {  // the warps of the panel
  asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory");
}

// A 32 x 32 inverse (row-major in global memory) into a tile of stride TS.
__device__ __forceinline__ void fetch_inverse(double* tile, const double* g) {
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const int r = i >> 4, c = (i & 15) * 2;
    cp16(tile + r * TS + c, g + r * 32 + c);
  }
  cp_commit();
}

// The rows of a warp's operand tile: lane 4g + t serves rows g, g+8, g+16, g+24.
struct Rows {
  int off[4];  // element offset of the row in W
  bool ok[4];
};

// A warp's operand ring: stages of eight columns of its 32 rows, 2 KB each. A
// lane fetches exactly what it will feed to the tensor core itself (columns
// 2t, 2t+1 of rows 8i + g), so the ring is a lane-private prefetch buffer
// (conflict-free, no barrier) that costs no registers. Three stages are in
// flight: 24 tensor instructions, 1500 cycles, cover the latency of L2.
constexpr int kRing = 4;
constexpr int kRingDoubles = kRing * 256;  // of one warp

// EDGE: the columns may end inside the block (zeros past them).
template <bool VEC, bool EDGE>
__device__ __forceinline__ void ring_load(double2* ring, int stage, const double* W, const Rows& r, int col, int n,
                                          bool live) {
  if (live) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int cols = !r.ok[i] ? 0 : EDGE ? max(0, min(2, n - col)) : 2;
      const double* p = W + (cols ? r.off[i] + col : 0);
      const unsigned d =
          static_cast<unsigned>(__cvta_generic_to_shared(ring + (stage * 4 + i) * 32 + (threadIdx.x & 31)));
      if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(p), "r"(8 * cols));
      } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(p), "r"(cols > 0 ? 8 : 0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8), "l"(cols > 1 ? p + 1 : p),
                     "r"(cols > 1 ? 8 : 0));
      }
    }
  }
  cp_commit();  // always: the waits count groups
}

// The first three stages of block K.
template <bool VEC, bool EDGE>
__device__ __forceinline__ void ring_start(double2* ring, const double* W, const Rows& r, int K, int n, bool live) {
#pragma unroll
  for (int q = 0; q < 3; ++q) ring_load<VEC, EDGE>(ring, q, W, r, 32 * K + 8 * q + 2 * (threadIdx.x & 3), n, live);
}

// Everything a block step shares. NI: 8-column groups of the strip.
template <int NI>
struct Acc {
  double v[2][NI][4];  // rows 16m + g, 16m + g + 8; columns 8i + 2t, + 1
};

// acc -= (warp's rows of W, columns 32K..32K+31) * U, with Ut holding -U^T
// (column c of U at Ut + c * US). The ring holds the first three stages; those
// of block Knext follow when `more`.
template <int NI, bool VEC, bool EDGE>
__device__ __forceinline__ void update(Acc<NI>& acc, double2* ring, const double* W, const Rows& r, const double* Ut,
                                       int K, int Knext, bool more, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q == 0) ring_load<VEC, EDGE>(ring, 3, W, r, 32 * K + 24 + 2 * t, n, true);
    else ring_load<VEC, EDGE>(ring, q - 1, W, r, 32 * Knext + 8 * (q - 1) + 2 * t, n, more);
    double2 b[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) b[i] = *reinterpret_cast<const double2*>(Ut + (8 * i + g) * US + 8 * q + 2 * t);
    cp_wait<3>();  // stage q has landed
    double2 a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = ring[(q * 4 + i) * 32 + lane];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int i = 0; i < NI; ++i) dmma1688(acc.v[m][i], a[2 * m], a[2 * m + 1], b[i]);
  }
}

// Tb <- the warp's accumulators (32 rows x 8 NI columns).
template <int NI>
__device__ __forceinline__ void store_tile(double* Tb, const Acc<NI>& acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      *reinterpret_cast<double2*>(Tb + (16 * m + g) * TS + 8 * i + 2 * t) = make_double2(acc.v[m][i][0], acc.v[m][i][1]);
      *reinterpret_cast<double2*>(Tb + (16 * m + g + 8) * TS + 8 * i + 2 * t) =
          make_double2(acc.v[m][i][2], acc.v[m][i][3]);
    }
}

// Ut <- -(Li Tb)^T over all warps, an 8 x 8 block of the product at a time;
// store(row, column, v0, v1) gets the product's column pairs. Li is lower
// (UPPER: upper) triangular.
template <int NI, bool UPPER, class Store>
__device__ __forceinline__ void tile_product(const double* Li, const double* Tb, double* Ut, Store store) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int u = warp; u < 4 * NI; u += nw) {
    const int mi = u / NI, ni = u - mi * NI;
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
    const int k0 = UPPER ? 8 * mi : 0, k1 = UPPER ? 32 : 8 * mi + 8;
    for (int k = k0; k < k1; k += 8) {
      dmma884(d0, Li[(8 * mi + g) * TS + k + t], Tb[(k + t) * TS + 8 * ni + g]);
      dmma884(d1, Li[(8 * mi + g) * TS + k + 4 + t], Tb[(k + 4 + t) * TS + 8 * ni + g]);
    }
    const double v0 = d0[0] + d1[0], v1 = d0[1] + d1[1];
    const int row = 8 * mi + g, col = 8 * ni + 2 * t;
    Ut[col * US + row] = -v0;
    Ut[(col + 1) * US + row] = -v1;
    store(row, col, v0, v1);
  }
}

// Inverse of a 32 x 32 triangle by one warp, out (row-major, global memory) in
// full with its zeros. D (stride PS, shared) holds L below the unit diagonal and
// U on and above it, kb live rows and columns (identity past them); X is a
// scratch tile of stride TS. The upper triangle is inverted as the lower
// triangle U^T. First the four 8 x 8 diagonal blocks, a lane per column, then
// the blocks below them: X_ij = -X_ii (T_ij X_jj + ... + T_i,i-1 X_i-1,j).
template <bool UPPER>
__device__ __forceinline__ void tri_inverse(const double* D, double* X, double* __restrict__ out, int kb) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto T = [&](int i, int k) {
    const bool in = i < kb && k < kb;
    return in ? (UPPER ? D[k * PS + i] : D[i * PS + k]) : (i == k ? 1.0 : 0.0);
  };
  {
    const int b = lane & ~7, c = lane & 7;
    const double rd = UPPER ? 1.0 / T(b + c, b + c) : 1.0;
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double s = i == c ? 1.0 : 0.0;
#pragma unroll
      for (int q = 0; q < i; ++q) s = fma(-T(b + i, b + q), x[q], s);
      if constexpr (UPPER) s *= __shfl_sync(kAll, rd, b + i);
      x[i] = i >= c ? s : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) X[(b + i) * TS + b + c] = x[i];
  }
  __syncwarp();
  for (int i = 1; i < 4; ++i)
    for (int j = 0; j < i; ++j) {
      double s[2] = {0.0, 0.0}, x[2] = {0.0, 0.0};
      for (int k = 8 * j; k < 8 * i; k += 4) dmma884(s, T(8 * i + g, k + t), X[(k + t) * TS + 8 * j + g]);
      // the sum's place is X_ij's until the product with X_ii replaces it
      X[(8 * i + g) * TS + 8 * j + 2 * t] = s[0];
      X[(8 * i + g) * TS + 8 * j + 2 * t + 1] = s[1];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; k += 4)
        dmma884(x, X[(8 * i + g) * TS + 8 * i + k + t], X[(8 * i + k + t) * TS + 8 * j + g]);
      __syncwarp();
      X[(8 * i + g) * TS + 8 * j + 2 * t] = -x[0];
      X[(8 * i + g) * TS + 8 * j + 2 * t + 1] = -x[1];
      __syncwarp();
    }
#pragma unroll 8
  for (int r = 0; r < 32; ++r) {
    const int i = UPPER ? lane : r, j = UPPER ? r : lane;
    out[r * 32 + lane] = j > i ? 0.0 : X[i * TS + j];
  }
}

// ---------------------------------------------------------------------------
// Panel: the pivot of each column is the first largest |a| in position order
// (the reference's rule, linalg.cpp:55-57). One row per thread. Columns go in
// groups of eight held in a[0..7]: inside a group each pivot step touches the
// group's columns only (one barrier per column, the warps' candidates through
// shared memory), then the group's pivot rows are solved for the columns right
// of it and the eight steps are applied to those at once. The group loop is
// rolled (the registers rotate by eight), so the code stays in the instruction
// cache: the form unrolled over 32 columns took 2500 cycles a column, mostly
// issue of 240 instructions per warp.
struct __align__(16) Cand {
  unsigned hi, lo;  // |a| as two words; 0, 0: no candidate
  int pos, pad;
};

struct __align__(16) PanelShared {
  Cand cand[2][kMaxWarps];
  double row[2][kMaxWarps][8];
  double raw[8][24];  // pivot rows of a group, right of it, before the solve
  double u[8][24];    // and after
  double l8[8][8];
  int info;
};

// Whether this lane holds the largest (hi, lo), ties to the smallest pos; `any`:
// some lane has a candidate. Nearly always one lane has the largest high word.
__device__ __forceinline__ bool warp_winner(unsigned hi, unsigned lo, int pos, bool& any) {
  const unsigned mh = __reduce_max_sync(kAll, hi);
  bool me = hi == mh;
  const unsigned top = __ballot_sync(kAll, me);
  any = true;
  if ((top & (top - 1)) != 0 || mh == 0) {
    const unsigned ml = __reduce_max_sync(kAll, me ? lo : 0u);
    any = (mh | ml) != 0;
    me = me && lo == ml;
    const int p = __reduce_min_sync(kAll, me ? pos : INT_MAX);
    me = me && pos == p && any;
  }
  return me;
}

// 1 / x by Newton's iteration on the mantissa from a single-precision start
// (error 2^-23, 2^-46, then rounding), without a branch, so that it runs beside
// the search for the winner. Exponent field of x in 1..2044.
__device__ __forceinline__ double newton_reciprocal(double x) {
  const int hi = __double2hiint(x);
  const double m = __hiloint2double((hi & 0x800fffff) | 0x3ff00000, __double2loint(x));
  double y = (double)__fdividef(1.0f, (float)m);
  y = fma(y, fma(-m, y, 1.0), y);
  y = fma(y, fma(-m, y, 1.0), y);
  return __hiloint2double(__double2hiint(y) - (((hi >> 20) & 0x7ff) - 1023) * (1 << 20), __double2loint(y));
}

// a: the thread's row of the column block; pos: its position in the panel (0 =
// the first row), updated; row: where the finished columns go (32 doubles of
// the thread's own). Returns 0 or the column of the first zero pivot + 1.
__device__ __forceinline__ int panel(PanelShared& sh, double (&a)[32], int& pos, bool valid, int kb, int aw, int na,
                                     double* row, int& nswap) {
  const int lane = threadIdx.x & 31, nthr = na * 32;
  bool alive = valid;  // not a pivot row yet
#pragma unroll 1
  for (int sp = 0; sp < 4; ++sp) {
    const int j0 = 8 * sp;
    if (j0 < kb) {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int j = j0 + s;
        if (j < kb) {  // uniform
          constexpr unsigned kInf = 0x7ff00000u;
          const int par = s & 1;
          unsigned hi = (unsigned)__double2hiint(a[s]) & 0x7fffffffu, lo = (unsigned)__double2loint(a[s]);
          if (!alive || hi > kInf || (hi == kInf && lo)) hi = lo = 0;  // a NaN is no candidate
          bool any;
          if (warp_winner(hi, lo, pos, any)) {
            sh.cand[par][aw] = Cand{hi, lo, pos, 0};
#pragma unroll
            for (int c = s & ~1; c < 8; c += 2)
              *reinterpret_cast<double2*>(&sh.row[par][aw][c]) = make_double2(a[c], a[c + 1]);
          }
          if (!any && lane == 0) sh.cand[par][aw] = Cand{0u, 0u, INT_MAX, 0};
          bar_active(nthr);
          const Cand cd = lane < na ? sh.cand[par][lane] : Cand{0u, 0u, INT_MAX, 0};
          double rp = newton_reciprocal(lane < na ? sh.row[par][lane][s] : 1.0);
          const bool best = warp_winner(cd.hi, cd.lo, cd.pos, any);
          if (!any) return j + 1;  // the same in every warp of the panel
          const int gw = 31 - __clz(__ballot_sync(kAll, best));
          const int gk = __shfl_sync(kAll, cd.pos, gw);
          rp = __shfl_sync(kAll, rp, gw);
          const double* prow = sh.row[par][gw];
          const unsigned ghi = __shfl_sync(kAll, cd.hi, gw);
          if (ghi < 0x00100000u || ghi >= 0x7fd00000u) rp = 1.0 / prow[s];  // outside newton_reciprocal's range
          const bool chosen = pos == gk;
          if (pos == j) pos = gk;
          if (chosen) {
            pos = j;
            alive = false;
          }
          nswap += gk != j;
          const double f = alive ? a[s] * rp : 0.0;
          if (alive) a[s] = f;
#pragma unroll
          for (int c = s + 1; c < 8; ++c) a[c] = fma(-f, prow[c], a[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) row[j0 + c] = a[c];
    if (j0 + 8 < kb) {
      const int mine = pos - j0;  // this row's place among the group's pivots
      if (valid && mine >= 0 && mine < 8) {
#pragma unroll
        for (int c = 0; c < 24; c += 2) *reinterpret_cast<double2*>(&sh.raw[mine][c]) = make_double2(a[8 + c], a[9 + c]);
#pragma unroll
        for (int c = 0; c < 8; c += 2) *reinterpret_cast<double2*>(&sh.l8[mine][c]) = make_double2(a[c], a[c + 1]);
      }
      bar_active(nthr);
      if (aw == 0 && lane < 24) {
        double x[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) x[s] = sh.raw[s][lane];
#pragma unroll
        for (int q = 0; q < 7; ++q)
#pragma unroll
          for (int s = q + 1; s < 8; ++s) x[s] = fma(-sh.l8[s][q], x[q], x[s]);
#pragma unroll
        for (int s = 0; s < 8; ++s) sh.u[s][lane] = x[s];
      }
      const int lim = valid ? min(max(mine, 0), 8) : 0;  // steps this row took part in
#pragma unroll
      for (int s = 0; s < 8; ++s) a[s] = s < lim ? a[s] : 0.0;
      bar_active(nthr);
#pragma unroll
      for (int grp = 0; grp < 3; ++grp) {
        if (j0 + 8 * (grp + 1) < kb) {
#pragma unroll
          for (int s = 0; s < 8; ++s) {
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
              const double2 u = *reinterpret_cast<const double2*>(&sh.u[s][8 * grp + c]);
              a[8 + 8 * grp + c] = fma(-a[s], u.x, a[8 + 8 * grp + c]);
              a[9 + 8 * grp + c] = fma(-a[s], u.y, a[9 + 8 * grp + c]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 24; ++c) a[c] = a[c + 8];
  }
  return 0;
}

// Shared memory of k_sys_lu, in doubles. The panel's staging tiles take the
// place of the rings (idle by then); the diagonal block that the inversions
// read takes U's.
struct LuLayout {
  int stage, tb, li, ut, d11, x2, total;
};
__host__ __device__ inline LuLayout lu_layout(int warps) {
  LuLayout l{};
  l.stage = 0;
  l.tb = warps * 32 * PS;  // >= the rings' warps * kRingDoubles
  l.li = l.tb + 32 * TS;
  l.ut = l.li + 32 * TS;
  l.d11 = l.ut;
  l.x2 = l.ut + 32 * US;
  l.total = l.x2 + 32 * TS;
  return l;
}
static_assert(32 * PS >= kRingDoubles);

__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_lu(SysArgs sa, const int32_t* __restrict__ list) {
  extern __shared__ __align__(16) double sm[];
  __shared__ PanelShared ps;
  __shared__ int s_perm[kSysMaxN];
  __shared__ double s_det[3];  // det, log|det|, sign
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const LuLayout lay = lu_layout(nw);
  double* Tb = sm + lay.tb;
  double* Li = sm + lay.li;
  double* Ut = sm + lay.ut;
  double* D11 = sm + lay.d11;
  double* X2 = sm + lay.x2;
  double* stage = sm + lay.stage + warp * 32 * PS;
  double2* ring = reinterpret_cast<double2*>(sm + warp * kRingDoubles);
  const View v = view(sa, list ? list[blockIdx.x] : blockIdx.x);
  const int n = v.n, ldw = v.ldw, nb = sys_blocks(n);
  for (int i = tid; i < n; i += blockDim.x) s_perm[i] = i;
  if (tid == 0) {
    ps.info = 0;
    s_det[0] = s_det[2] = 1.0;
    s_det[1] = 0.0;
  }
  const bool want_det = sa.det || sa.sign || sa.logabs;
  const bool avec = n % 2 == 0 && (reinterpret_cast<uintptr_t>(v.A) & 15) == 0;
  __syncthreads();

  for (int J = 0; J < nb; ++J) {
    const int kb = min(32, n - 32 * J);
    // 1. the warp's rows of the column block
    Acc<4> acc;
    Rows r;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = 32 * warp + 8 * i + g;
      r.ok[i] = p < n;
      const int row = r.ok[i] ? s_perm[p] : 0;
      r.off[i] = row * ldw;
      const double* src = v.A + (int64_t)row * n;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int col = 32 * J + 8 * ni + 2 * t;
        double x = 0.0, y = 0.0;
        if (r.ok[i] && col < n) {
          if (avec) {  // n is even: the pair ends inside the row
            const double2 z = __ldcs(reinterpret_cast<const double2*>(src + col));
            x = z.x;
            y = z.y;
          } else {
            x = __ldcs(src + col);
            if (col + 1 < n) y = __ldcs(src + col + 1);
          }
        }
        acc.v[i >> 1][ni][2 * (i & 1)] = x;
        acc.v[i >> 1][ni][2 * (i & 1) + 1] = y;
      }
    }
    // 2. the earlier blocks
    if (J > 0) {
      const bool below = warp > 0 && warp < nb;
      if (J == 1) __syncthreads();  // the first block's inverse has been written
      fetch_inverse(Li, v.dinv);
      ring_start<true, false>(ring, v.W, r, 0, n, below);
      for (int K = 0; K < J; ++K) {
        if (warp == K) store_tile<4>(Tb, acc);
        cp_wait<3>();  // the inverse; at most three operand stages stay in flight
        __syncthreads();
        tile_product<4, false>(Li, Tb, Ut, [&](int row, int col, double v0, double v1) {
          double* o = v.W + s_perm[32 * K + row] * ldw + 32 * J + col;
          if (32 * J + col < ldw) *reinterpret_cast<double2*>(o) = make_double2(v0, v1);
        });
        __syncthreads();
        if (K + 1 < J) fetch_inverse(Li, v.dinv + (K + 1) * 2048);
        else cp_commit();
        if (warp > K && warp < nb) {
          update<4, true, false>(acc, ring, v.W, r, Ut, K, K + 1, K + 1 < J && warp > K + 1, n);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) cp_commit();  // the waits count groups
        }
      }
      cp_wait<0>();
      __syncthreads();  // the rings become the staging tiles, Ut the diagonal block
    }
    // 3. the panel: warps J..nb-1, a row per thread
    if (warp >= J && warp < nb) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            stage[(16 * m + g + 8 * (e >> 1)) * PS + 8 * ni + 2 * t + (e & 1)] = acc.v[m][ni][e];
      __syncwarp();
      double a[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) a[c] = stage[lane * PS + c];
      const int p = 32 * warp + lane;
      const bool valid = p < n;
      const int phys = valid ? s_perm[p] : 0;
      int pos = p - 32 * J, nswap = 0;
      if (valid && J + 1 < nb) {  // the row's next column block on its way into L2
        const double* nx = v.A + (int64_t)phys * n + 32 * (J + 1);
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(16, n - 32 * (J + 1) - 1)));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(31, n - 32 * (J + 1) - 1)));
      }
      const int info = panel(ps, a, pos, valid, kb, warp - J, nb - J, stage + lane * PS, nswap);
      if (info) {
        if (tid == 32 * J) ps.info = 32 * J + info;
      } else {
        if (valid) s_perm[32 * J + pos] = phys;
        __syncwarp();
        const int off = phys * ldw, at = valid ? pos : n;
#pragma unroll 8
        for (int rr = 0; rr < 32; ++rr) {
          const int o = __shfl_sync(kAll, off, rr), p2 = __shfl_sync(kAll, at, rr);
          const double x = stage[rr * PS + lane];
          if (p2 < n && lane < kb) v.W[o + 32 * J + lane] = x;
          if (p2 < kb) D11[p2 * PS + lane] = x;
        }
        if (tid == 32 * J && (nswap & 1)) {
          s_det[0] = -s_det[0];
          s_det[2] = -s_det[2];
        }
      }
    }
    __syncthreads();
    if (ps.info) {
      if (tid == 0) {
        if (sa.state) sa.state[v.slot] = ps.info;
        if (sa.det) sa.det[v.idx] = 0.0;
        if (sa.sign) sa.sign[v.idx] = 0.0;
        if (sa.logabs) sa.logabs[v.idx] = -INFINITY;
        if (sa.info) sa.info[v.idx] = ps.info;
      }
      return;
    }
    // the diagonal block's inverses and the pivots' part of det / slogdet, each by
    // one warp, beside the other warps' loads of the next column block
    double* di = v.dinv + (int64_t)J * 2048;
    if (warp == 0) tri_inverse<false>(D11, Tb, di, kb);
    if (warp == 1 % nw) tri_inverse<true>(D11, X2, di + 1024, kb);
    if (warp == 2 % nw && want_det) {
      // folded in the reference's order (linalg.cpp:400-403, 425-431)
      const double pv = lane < kb ? D11[lane * PS + lane] : 1.0;
      const double lg = log(fabs(pv)), sgn = pv / fabs(pv);
      double det = s_det[0], la = s_det[1], sg = s_det[2];
      for (int j = 0; j < kb; ++j) {
        det *= __shfl_sync(kAll, pv, j);
        la += __shfl_sync(kAll, lg, j);
        sg *= __shfl_sync(kAll, sgn, j);
      }
      __syncwarp();
      if (lane == 0) {
        s_det[0] = det;
        s_det[1] = la;
        s_det[2] = sg;
        if (J + 1 == nb) {
          if (sa.det) sa.det[v.idx] = det;
          if (sa.sign) sa.sign[v.idx] = sg;
          if (sa.logabs) sa.logabs[v.idx] = la;
        }
      }
    }
  }
  for (int i = tid; i < n; i += blockDim.x) v.perm[i] = s_perm[i];
  if (tid == 0) {
    if (sa.state) sa.state[v.slot] = 0;
    if (sa.info) sa.info[v.idx] = 0;
  }
}

// ---------------------------------------------------------------------------
// Substitution of one strip: C = P B (or P times columns of the identity), then
// Y_K = L_KK^-1 C_K and C_w -= L_wK Y_K downwards, X_K = U_KK^-1 Y_K and
// Y_w -= U_wK X_K upwards.
constexpr int solve_smem(int warps) { return (warps * kRingDoubles + 64 * TS + 32 * US) * 8; }

template <int NI, bool VEC>
__device__ __forceinline__ void solve_strip(const SysArgs& sa, const View& v, bool inverse, int c0, int width,
                                            double* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* ring = reinterpret_cast<double2*>(sm + warp * kRingDoubles);
  double* Tb = sm + (blockDim.x >> 5) * kRingDoubles;
  double* Li = Tb + 32 * TS;
  double* Ut = Li + 32 * TS;
  const int g = lane >> 2, t = lane & 3;
  const int n = v.n, nb = sys_blocks(n);
  const int ldx = inverse ? n : v.nrhs;
  double* X = inverse ? sa.inv + v.inv_off : sa.X + v.b_off;
  const double* B = sa.B + v.b_off;
  Acc<NI> acc;
  Rows r;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = 32 * warp + 8 * i + g;
    r.ok[i] = p < n;
    const int row = r.ok[i] ? v.perm[p] : 0;
    r.off[i] = (sa.w_by_position ? (r.ok[i] ? p : 0) : row) * v.ldw;
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = 8 * ni + 2 * t + e;
        double x = 0.0;
        if (r.ok[i] && col < width) x = inverse ? (row == c0 + col ? 1.0 : 0.0) : B[(int64_t)row * ldx + c0 + col];
        acc.v[i >> 1][ni][2 * (i & 1) + e] = x;
      }
  }
  auto no_store = [](int, int, double, double) {};
  fetch_inverse(Li, v.dinv);
  ring_start<VEC, false>(ring, v.W, r, 0, n, warp > 0 && warp < nb);
  for (int K = 0; K < nb; ++K) {
    if (warp == K) store_tile<NI>(Tb, acc);
    cp_wait<3>();  // the inverse; at most three operand stages stay in flight
    __syncthreads();
    tile_product<NI, false>(Li, Tb, Ut, no_store);
    __syncthreads();
    // the next block's L_KK^-1, after the last one the first U_KK^-1 (same block)
    fetch_inverse(Li, v.dinv + (K + 1 < nb ? (K + 1) * 2048 : K * 2048 + 1024));
    if (warp > K && warp < nb) {
      update<NI, VEC, false>(acc, ring, v.W, r, Ut, K, K + 1, warp > K + 1, n);
    } else {
      if (warp == K) {  // Y_K back into its owner's registers for the way up
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              acc.v[m][ni][e] = -Ut[(8 * ni + 2 * t + (e & 1)) * US + 16 * m + g + 8 * (e >> 1)];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) cp_commit();  // the waits count groups
    }
  }
  ring_start<VEC, true>(ring, v.W, r, nb - 1, n, warp < nb - 1);
  for (int K = nb - 1; K >= 0; --K) {
    if (warp == K) store_tile<NI>(Tb, acc);
    cp_wait<3>();
    __syncthreads();
    tile_product<NI, true>(Li, Tb, Ut, [&](int row, int col, double v0, double v1) {
      if (32 * K + row < n) {
        double* o = X + (int64_t)(32 * K + row) * ldx + c0 + col;
        if (col < width) o[0] = v0;
        if (col + 1 < width) o[1] = v1;
      }
    });
    __syncthreads();
    if (K > 0) fetch_inverse(Li, v.dinv + (K - 1) * 2048 + 1024);
    else cp_commit();
    if (warp < K) {
      update<NI, VEC, true>(acc, ring, v.W, r, Ut, K, K - 1, warp < K - 1, n);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) cp_commit();
    }
  }
}

__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_solve(SysArgs sa, const SysItem* __restrict__ items) {
  extern __shared__ __align__(16) double sm[];
  SysItem it;
  if (items) {
    it = items[blockIdx.x];
  } else {
    const int nr = (sa.unrhs + 31) / 32, ni = sa.uinv ? (sa.un + 31) / 32 : 0;
    it.sys = blockIdx.x / (nr + ni);
    const int k = blockIdx.x - it.sys * (nr + ni);
    it.inverse = k >= nr;
    it.c0 = 32 * (k >= nr ? k - nr : k);
    it.width = (int16_t)min(32, (it.inverse ? sa.un : sa.unrhs) - it.c0);
  }
  const View v = view(sa, it.sys);
  if (sa.state && sa.state[v.slot]) return;  // singular: nothing to solve with
  const bool vec = v.ldw % 2 == 0 && (reinterpret_cast<uintptr_t>(v.W) & 15) == 0;
  if (it.width <= 8) {
    if (vec) solve_strip<1, true>(sa, v, it.inverse, it.c0, it.width, sm);
    else solve_strip<1, false>(sa, v, it.inverse, it.c0, it.width, sm);
  } else if (it.width <= 16) {
    if (vec) solve_strip<2, true>(sa, v, it.inverse, it.c0, it.width, sm);
    else solve_strip<2, false>(sa, v, it.inverse, it.c0, it.width, sm);
  } else {
    if (vec) solve_strip<4, true>(sa, v, it.inverse, it.c0, it.width, sm);
    else solve_strip<4, false>(sa, v, it.inverse, it.c0, it.width, sm);
  }
}

// ---------------------------------------------------------------------------
// Kept factors: the permutation of the swap list (every thread follows its own
// rows through the swaps; the list is read by broadcast) in CTA (s, 0), the
// diagonal blocks' inverses in the CTAs (s, b).
__global__ void __launch_bounds__(64)
k_sys_prepare(SysArgs sa, const int32_t* __restrict__ ipiv, const int32_t* __restrict__ list) {
  __shared__ double D[32 * PS];
  __shared__ __align__(16) double X[2][32 * TS];
  const int s = list ? list[blockIdx.x] : blockIdx.x;
  const View v = view(sa, s);
  const int n = v.n, b = (int)blockIdx.y - 1;
  if (b >= sys_blocks(n)) return;
  if (b < 0) {
    extern __shared__ int piv[];
    const int32_t* src = ipiv + (sa.desc ? sa.desc[s].piv_off : (int64_t)s * n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int p = src[i];
      piv[i] = p < i || p >= n ? i : p;  // a swap list only names rows >= its own
    }
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x) {
      int at[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) at[e] = i0 + e * (int)blockDim.x;
      for (int k = 0; k < n; ++k) {
        const int p = piv[k];
#pragma unroll
        for (int e = 0; e < 8; ++e) at[e] = at[e] == k ? p : at[e] == p ? k : at[e];
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (i0 + e * (int)blockDim.x < n) v.perm[at[e]] = i0 + e * blockDim.x;
    }
    return;
  }
  const int kb = min(32, n - 32 * b);
  const double* M = v.W + (int64_t)32 * b * v.ldw + 32 * b;
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) {
    const int r = i >> 5, c = i & 31;
    if (r < kb && c < kb) D[r * PS + c] = M[(int64_t)r * v.ldw + c];
  }
  __syncthreads();
  double* di = v.dinv + (int64_t)b * 2048;
  if (threadIdx.x < 32) tri_inverse<false>(D, X[0], di, kb);
  else tri_inverse<true>(D, X[1], di + 1024, kb);
}

}  // namespace

cudaError_t launch_sys_lu(const SysArgs& sa, const int32_t* list, int nsys, int nmax, cudaStream_t st) {
  if (nsys <= 0) return cudaSuccess;
  if (nmax > kSysMaxN) return cudaErrorInvalidValue;
  const int nw = sys_blocks(nmax);
  k_sys_lu<<<nsys, 32 * nw, sizeof(double) * lu_layout(nw).total, st>>>(sa, list);
  return cudaGetLastError();
}

cudaError_t launch_sys_solve(const SysArgs& sa, const SysItem* items, int64_t nitems, int nsys, int nmax,
                             cudaStream_t st) {
  if (!items) nitems = (int64_t)nsys * ((sa.unrhs + 31) / 32 + (sa.uinv ? (sa.un + 31) / 32 : 0));
  if (nitems <= 0) return cudaSuccess;
  if (nmax > kSysMaxN || nitems > INT_MAX) return cudaErrorInvalidValue;
  const int nw = sys_blocks(nmax);
  k_sys_solve<<<(unsigned)nitems, 32 * nw, solve_smem(nw), st>>>(sa, items);
  return cudaGetLastError();
}

cudaError_t launch_sys_prepare(const SysArgs& sa, const int32_t* ipiv, const int32_t* list, int nsys, int nmax,
                               cudaStream_t st) {
  if (nsys <= 0) return cudaSuccess;
  const dim3 grid((unsigned)nsys, (unsigned)sys_blocks(nmax) + 1);
  k_sys_prepare<<<grid, 64, sizeof(int) * (size_t)nmax, st>>>(sa, ipiv, list);
  return cudaGetLastError();
}

cudaError_t sys_prepare_kernels() {
  cudaError_t e = cudaFuncSetAttribute(k_sys_lu, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(double) * lu_layout(kMaxWarps).total);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sys_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, solve_smem(kMaxWarps));
  return e;
}

}  // namespace nppb
