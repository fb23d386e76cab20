// System-resident LU and substitution: orders 33..512 on one CTA per system, larger
// ones by outer blocks of 128 columns (k_sys_outer, k_sys_rows, k_sys_gemm).
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
// L_KK^-1, back with U_KK^-1 (with U_KK itself where that is ill-conditioned, so
// that the solution keeps the backward error of a substitution), in one launch.
//
// What bounds it: FP64 tensor throughput in 2 (mma.m16n8k8, 64 FMA per cycle
// and SM), the dependent pivot steps in 3.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "sys_device.cuh"

namespace nppb {
namespace {

constexpr int GS = 10;  // row stride of the transposed 8-row U tile of a panel group

// tri_inverse's output into a row-major 32 x 32 array.
__device__ __forceinline__ auto into(double* out) {
  return [out](int r, int c, double v) { out[r * 32 + c] = v; };
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

__device__ __forceinline__ void bar_active(int threads) {  // the warps of the panel
  asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory");
}

// A 32 x 32 inverse (row-major in global memory) into a tile of stride TS, by
// threads first .. first + nthr - 1.
__device__ __forceinline__ void fetch_inverse(double* tile, const double* g, int nthr, int first = 0) {
  for (int i = (int)threadIdx.x - first; i < 512; i += nthr) {
    const int r = i >> 4, c = (i & 15) * 2;
    cp16(tile + r * US + c, g + r * 32 + c);
  }
  cp_commit();
}

// Tb <- the warp's accumulators (32 rows x 8 NI columns).
template <int NI>
__device__ __forceinline__ void store_tile(double* Tb, const Acc<NI>& acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      double* o = Tb + (16 * m + g) * BS + 8 * i + 2 * t;
      *reinterpret_cast<double2*>(o) = make_double2(acc.v[m][i][0], acc.v[m][i][1]);
      *reinterpret_cast<double2*>(o + 8 * BS) = make_double2(acc.v[m][i][2], acc.v[m][i][3]);
    }
}

// Ut <- -(Li Tb)^T: the product of a diagonal block's inverse (lower, UPPER: upper
// triangular: half of the steps for half of its rows) with the block's rows.
// Warps 0..3, one on each scheduler, take eight columns each (with one group of
// eight: eight rows each); the others go on to the next barrier.
// CS > 1: into every CTA of the cluster.
template <int NI, bool UPPER, int CS>
__device__ __forceinline__ void tile_product(const double* Li, const double* Tb, double* Ut) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warp = threadIdx.x >> 5;
  if (warp >= 4) return;
  const int step = min(4, (int)(blockDim.x >> 5));
  auto put = [&](int col, int row, double v) {
    if constexpr (CS == 1) {
      Ut[col * US + row] = v;
    } else {
#pragma unroll
      for (int c = 0; c < CS; ++c) cg::this_cluster().map_shared_rank(Ut, c)[col * US + row] = v;
    }
  };
  auto left = [&](int row, int q) { return *reinterpret_cast<const double2*>(Li + row * US + 8 * q + 2 * t); };
  auto right = [&](int col, int q) {
    const double* b = Tb + (8 * q + 2 * t) * BS + col;
    return make_double2(b[0], b[BS]);
  };
  if constexpr (NI > 1) {
    for (int ni = warp; ni < NI; ni += step) {
      double d[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) d[m][e] = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 b = right(8 * ni + g, q);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          if (UPPER ? (q < 2 && m == 1) : (q >= 2 && m == 0)) continue;  // zeros of the triangle
          dmma1688(d[m], left(16 * m + g, q), left(16 * m + 8 + g, q), b);
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          put(8 * ni + 2 * t + (e & 1), 16 * m + g + 8 * (e >> 1), -d[m][e]);
    }
  } else {
    for (int mi = warp; mi < 4; mi += step) {
      double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 x = left(8 * mi + g, q), y = right(g, q);
        dmma884(d[0], x.x, y.x);
        dmma884(d[1], x.y, y.y);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) put(2 * t + e, 8 * mi + g, -(d[0][e] + d[1][e]));
    }
  }
}

// A block that is marked as too ill-conditioned for that: T holds the triangle itself
// as tri_inverse leaves it, and the rows are substituted in their tile, by one warp
// with a lane per column, eight rows in registers at a time (no division here: with
// one, strips of 32 columns spill around it and every solve loses 1%). The loads are
// written where they are to happen, for the registers.
template <bool UPPER>
__device__ __forceinline__ bool tri_marked(const double* T) { return T[UPPER ? 31 * US + 1 : 31] != 0.0; }

__device__ __forceinline__ double lds1(unsigned p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(p) : "memory");
  return v;
}
__device__ __forceinline__ void sts1(unsigned p, double v) {
  asm volatile("st.shared.f64 [%0], %1;\n" ::"r"(p), "d"(v) : "memory");
}

template <int NI, bool UPPER>
__device__ __forceinline__ void tile_substitute(const double* T, double* Tb) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32 || lane >= 8 * NI) return;
  const unsigned c = smem(Tb + lane), tri = smem(T);
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    const int i0 = UPPER ? 24 - 8 * s : 8 * s;
    const unsigned ci = c + i0 * (8 * BS), ti = tri + i0 * (8 * US);  // row i0 of the strip and of T
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = lds1(ci + i * (8 * BS));
#pragma unroll 1
    for (int p = 0; p < 8 * s; ++p) {  // the rows solved before
      const int q = UPPER ? 31 - p : p;
      const double y = lds1(c + q * (8 * BS));
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = fma(-lds1(ti + i * (8 * US) + 8 * q), y, x[i]);
    }
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int j = UPPER ? 7 - p : p;
      double col[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (UPPER ? i < j : i > j) col[i] = lds1(ti + i * (8 * US) + 8 * (i0 + j));
      if constexpr (UPPER) {
        const unsigned row = ti + j * (8 * US);
        x[j] = x[j] * lds1(row + 8 * (i0 + j)) * lds1(i0 + j ? row : tri + 8 * (2 * US + 1));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (UPPER ? i < j : i > j) x[i] = fma(-col[i], x[j], x[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sts1(ci + i * (8 * BS), x[i]);
  }
}

// Ut <- -Tb^T, as tile_product leaves it.
template <int NI, int CS>
__device__ __forceinline__ void tile_negate(const double* Tb, double* Ut) {
  for (int i = threadIdx.x; i < 256 * NI; i += blockDim.x) {
    const int row = i & 31, col = i >> 5;
    const double v = -Tb[row * BS + col];
    if constexpr (CS == 1) {
      Ut[col * US + row] = v;
    } else {
#pragma unroll
      for (int c = 0; c < CS; ++c) cg::this_cluster().map_shared_rank(Ut, c)[col * US + row] = v;
    }
  }
}

// The marks of a system's blocks, at most 16: L's in the lower half, U's in the upper. Read once
// on entry, behind the strip's own loads, instead of from the tile after each block's barrier:
// 229 re-solves of 201 x 64 160 us (166), 400 inverses of order 201 914 us (922). On clusters the
// tile's form stays: 48 re-solves of 777 x 16 take 208 us with it, 223 us with this one.
__device__ __forceinline__ unsigned tri_marks(const double* dinv, int nb) {
  const int lane = threadIdx.x & 31, b = lane & 15;
  return __ballot_sync(kAll, b < nb && dinv[b * 2048 + (lane < 16 ? 31 : 1024 + 31 * 32 + 1)] != 0.0);
}

// The product's rows to memory, by warps first .. first + count - 1 (those that
// have nothing to update): row(r) is where row r goes, or null; PAIRS: 16 bytes
// at once, else up to `cols` columns.
template <int NI, bool PAIRS, class Row>
__device__ __forceinline__ void product_out(const double* Ut, int cols, int first, int count, Row row) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int mi = (int)(threadIdx.x >> 5) - first; mi < 4; mi += count) {
    double* o = row(8 * mi + g);
    if (!o) continue;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int col = 8 * i + 2 * t;
      const double v0 = -Ut[col * US + 8 * mi + g], v1 = -Ut[(col + 1) * US + 8 * mi + g];
      if constexpr (PAIRS) {
        if (col < cols) *reinterpret_cast<double2*>(o + col) = make_double2(v0, v1);
      } else {
        if (col < cols) o[col] = v0;
        if (col + 1 < cols) o[col + 1] = v1;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Panel: the pivot of each column is the first largest |a| in position order
// (the reference's rule, linalg.cpp:55-57). The warps keep their 32 x 32 tiles of
// the column block in the tensor core's accumulators and take the columns in
// four groups of eight. A group's columns go through the staging tile to one
// row per thread; each pivot step then touches the group's columns only (one
// barrier per column, the warps' candidates through shared memory). After the
// group its pivot rows are solved for the columns right of it, and the eight
// steps are applied to those at once by the tensor core.
//
// Latency bounds it: a column is two warp reductions, a division and a barrier
// deep, so everything that can be is started on the likely outcome (the
// candidate with the largest high word, which is nearly always unique) and
// repeated exactly otherwise. The group loop is rolled (the accumulators rotate),
// which keeps the code in the instruction cache.
// Cycles per column with 1 / 16 warps: 535 / 1120 (the step-wise panel: 2500).
struct __align__(16) Cand {
  unsigned hi, lo;  // |a| as two words; 0, 0: no candidate
  int pos, pad;
};

struct __align__(16) PanelShared {
  Cand cand[2][kMaxWarps];
  double row[2][kMaxWarps][8];
  double rp[2][kMaxWarps];
  double raw[8][24];    // pivot rows of a group, right of it, before the solve
  double l8[8][8];
  double u[24 * GS];    // minus the solved rows, transposed
  int info;
};

// Whether this lane holds the largest (hi, lo), ties to the smallest pos; `any`:
// some lane has a candidate.
__device__ __forceinline__ bool exact_winner(unsigned hi, unsigned lo, int pos, bool& any) {
  const unsigned mh = __reduce_max_sync(kAll, hi);
  bool me = hi == mh;
  const unsigned ml = __reduce_max_sync(kAll, me ? lo : 0u);
  any = (mh | ml) != 0;
  me = any && me && lo == ml;
  const int first = __reduce_min_sync(kAll, me ? pos : INT_MAX);  // by every lane
  return me && pos == first;
}

constexpr unsigned kInf = 0x7ff00000u;  // high word of infinity

// The rare level-one cases: lanes that share the high word, NaN (no candidate),
// infinities, or no candidate at all.
template <class Publish>
__device__ __forceinline__ void exact_publish(PanelShared& sh, double x, bool live, int par, int aw, int pos,
                                           Publish publish) {
  unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu, lo = (unsigned)__double2loint(x);
  if (!live || hi > kInf || (hi == kInf && lo)) hi = lo = 0;
  bool any;
  const bool me = exact_winner(hi, lo, pos, any);
  __syncwarp();
  if (me) publish(hi, lo, 1.0 / x);
  else if (!any && (threadIdx.x & 31) == 0) sh.cand[par][aw] = Cand{0u, 0u, INT_MAX, 0};
}

// acc: the warp's tile of the column block (clobbered); pos: the position in the
// panel of the thread's row (row `lane` of the tile; 0 = the panel's first row),
// updated; tile: the warp's staging tile, which ends with the finished columns.
// Returns 0 or the column of the first zero pivot + 1.
__device__ __forceinline__ int panel(PanelShared& sh, Acc<4>& acc, int& pos, bool valid, int kb, int aw, int na,
                                     double* tile, int& nswap) {
  const int lane = threadIdx.x & 31, nthr = na * 32, g = lane >> 2, t = lane & 3;
  unsigned live = valid ? 0x7fffffffu : 0u;  // mask of the magnitude's high word; 0: a pivot row already
#pragma unroll 1
  for (int j0 = 0; j0 < kb; j0 += 8) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      *reinterpret_cast<double2*>(tile + (16 * m + g) * PS + j0 + 2 * t) = make_double2(acc.v[m][0][0], acc.v[m][0][1]);
      *reinterpret_cast<double2*>(tile + (16 * m + g + 8) * PS + j0 + 2 * t) =
          make_double2(acc.v[m][0][2], acc.v[m][0][3]);
    }
    __syncwarp();
    double a[8];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 x = *reinterpret_cast<const double2*>(tile + lane * PS + j0 + c);
      a[c] = x.x;
      a[c + 1] = x.y;
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int j = j0 + s;
      if (j < kb) {  // uniform
        const int par = s & 1;
        const unsigned hi = (unsigned)__double2hiint(a[s]) & live;
        const unsigned mh = __reduce_max_sync(kAll, hi);
        const double rp = 1.0 / (hi ? a[s] : 1.0);  // every candidate's, beside the reduction
        const bool me = hi == mh;
        const unsigned top = __ballot_sync(kAll, me);
        auto publish = [&](unsigned h, unsigned l, double r) {
          sh.cand[par][aw] = Cand{h, l, pos, 0};
          sh.rp[par][aw] = r;
#pragma unroll
          for (int c = s & ~1; c < 8; c += 2)
            *reinterpret_cast<double2*>(&sh.row[par][aw][c]) = make_double2(a[c], a[c + 1]);
        };
        if (me) publish(hi, (unsigned)__double2loint(a[s]), rp);
        if ((top & (top - 1)) != 0 || mh >= kInf) exact_publish(sh, a[s], live != 0, par, aw, pos, publish);
        bar_active(nthr);
        const Cand cd = lane < na ? sh.cand[par][lane] : Cand{0u, 0u, INT_MAX, 0};
        const unsigned key = lane < na ? (cd.hi & ~15u) | (15u - lane) : 0u;
        const unsigned mk = __reduce_max_sync(kAll, key);
        const unsigned amb = __ballot_sync(kAll, lane < na && (key ^ mk) < 16u);
        int gw = 15 - (int)(mk & 15u);
        double r = sh.rp[par][gw];
        int gk = sh.cand[par][gw].pos;
        if ((amb & (amb - 1)) != 0 || mk < 16u) {
          bool any;
          const bool best = exact_winner(cd.hi, cd.lo, cd.pos, any);
          if (!any) return j + 1;  // the same in every warp of the panel
          gw = 31 - __clz(__ballot_sync(kAll, best));
          r = sh.rp[par][gw];
          gk = sh.cand[par][gw].pos;
        }
        const double* prow = sh.row[par][gw];
        const bool chosen = pos == gk;
        if (pos == j) pos = gk;
        if (chosen) {
          pos = j;
          live = 0;
        }
        nswap += gk != j;
        const double f = live ? a[s] * r : 0.0;
        if (live) a[s] = f;
#pragma unroll
        for (int c = s + 1; c < 8; ++c) a[c] = fma(-f, prow[c], a[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; c += 2) *reinterpret_cast<double2*>(tile + lane * PS + j0 + c) = make_double2(a[c], a[c + 1]);
    if (j0 + 8 >= kb) break;
    // the row's step in the group; 8: still below, -1: done before
    const bool in_group = valid && pos >= j0 && pos < j0 + 8;
    const int mine = live ? 8 : in_group ? pos - j0 : -1;
    if (in_group) {
#pragma unroll
      for (int c = 0; c < 8; c += 2) *reinterpret_cast<double2*>(&sh.l8[pos - j0][c]) = make_double2(a[c], a[c + 1]);
    }
    __syncwarp();
    int lim[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      lim[i] = __shfl_sync(kAll, mine, 8 * i + g);
      if (lim[i] >= 0 && lim[i] < 8) {
#pragma unroll
        for (int ni = 1; ni < 4; ++ni)
          *reinterpret_cast<double2*>(&sh.raw[lim[i]][8 * (ni - 1) + 2 * t]) =
              make_double2(acc.v[i >> 1][ni][2 * (i & 1)], acc.v[i >> 1][ni][2 * (i & 1) + 1]);
      }
    }
    // the multipliers as tensor-core operand; a row takes part in the steps before its own
    double2 l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      l[i] = *reinterpret_cast<const double2*>(tile + (8 * i + g) * PS + j0 + 2 * t);
      if (2 * t >= lim[i]) l[i].x = 0.0;
      if (2 * t + 1 >= lim[i]) l[i].y = 0.0;
    }
    bar_active(nthr);
    if (aw == 0) {
      const int c = min(lane, 23);
      double x[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) x[s] = sh.raw[s][c];
#pragma unroll
      for (int q = 0; q < 7; ++q) {
#pragma unroll
        for (int s = q + 1; s < 8; ++s) x[s] = fma(-sh.l8[s][q], x[q], x[s]);
      }
      if (lane < 24) {
#pragma unroll
        for (int s = 0; s < 8; s += 2)
          *reinterpret_cast<double2*>(&sh.u[lane * GS + s]) = make_double2(-x[s], -x[s + 1]);
      }
    }
    bar_active(nthr);
#pragma unroll
    for (int ni = 1; ni < 4; ++ni) {
      const double2 b = *reinterpret_cast<const double2*>(&sh.u[(8 * (ni - 1) + g) * GS + 2 * t]);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        dmma1688(acc.v[m][ni], l[2 * m], l[2 * m + 1], b);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc.v[m][ni - 1][e] = acc.v[m][ni][e];
      }
    }
  }
  return 0;
}

// Shared memory, in doubles: the tiles, then a region per warp that is its operand
// ring, in the panel its staging tile and in an inversion its scratch tile. The
// diagonal block that the inversions read takes U's place.
constexpr int kTb = 0, kLi = 32 * US, kUt = 64 * US, kWarp = 96 * US;
static_assert(PS <= US && 32 * TS <= kPerWarp);
constexpr int sys_smem(int warps) { return 8 * (kWarp + warps * kPerWarp); }
// of a cluster's CTA: U twice, behind the per-warp regions
constexpr int sys_cluster_smem(int warps) { return sys_smem(warps) + 8 * 32 * US; }

__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_lu(SysArgs sa, const int32_t* __restrict__ list) {
  extern __shared__ __align__(16) double sm[];
  __shared__ PanelShared ps;
  __shared__ int s_perm[kSysMaxN];
  __shared__ double s_det[3];  // det, log|det|, sign
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  double* Tb = sm + kTb;
  double* Li = sm + kLi;
  double* Ut = sm + kUt;
  double* D11 = Ut;
  double* stage = sm + kWarp + warp * kPerWarp;
  const unsigned ring = smem(stage) + 16 * lane;
  const unsigned ulane = smem(Ut + g * US + 2 * t);
  // what the inner loops do not need stays out of the registers
  __shared__ View s_v;
  if (tid == 0) s_v = view(sa, list ? list[blockIdx.x] : blockIdx.x);
  __syncthreads();
  double* const W = s_v.W;
  const int n = s_v.n, nb = sys_blocks(n);
  for (int i = tid; i < n; i += blockDim.x) s_perm[i] = i;
  if (tid == 0) {
    ps.info = 0;
    s_det[0] = s_det[2] = 1.0;
    s_det[1] = 0.0;
  }
  __syncthreads();

  for (int J = 0; J < nb; ++J) {
    const int kb = min(32, n - 32 * J);
    // 1. the warp's rows of the column block
    Acc<4> acc;
    Rows r;
    const double* A = s_v.A;
    const bool avec = n % 2 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    r.live = n - 32 * warp - g;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int p = 32 * warp + 8 * i + g;
      const bool ok = p < n;
      const int row = ok ? s_perm[p] : 0;
      r.off[i] = (unsigned)row * s_v.ldw * 8;
      const double* src = A + (int64_t)row * n;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int col = 32 * J + 8 * ni + 2 * t;
        double x = 0.0, y = 0.0;
        if (ok && col < n) {
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
      fetch_inverse(Li, s_v.dinv, blockDim.x);
      ring_start<true, false>(ring, W, r, 0, n, below);
      for (int K = 0; K < J; ++K) {
        if (warp == K) store_tile<4>(Tb, acc);
        cp_wait<2>();  // the inverse; at most two operand stages stay in flight
        __syncthreads();
        tile_product<4, false, 1>(Li, Tb, Ut);
        __syncthreads();
        if (warp > K && warp < nb) {
          update<4, true, false>(acc, ring, W, r, ulane, K, K + 1, K + 1 < J && warp > K + 1, n);
        } else {
          if (warp <= K) {  // the warps that are done: U out, the next inverse in
            if (K + 1 < J) fetch_inverse(Li, s_v.dinv + (K + 1) * 2048, 32 * (K + 1));
            product_out<4, true>(Ut, s_v.ldw - 32 * J, 0, K + 1,
                                 [&](int row) { return W + s_perm[32 * K + row] * s_v.ldw + 32 * J; });
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) cp_commit();  // the waits count groups
        }
      }
      cp_wait<0>();
      __syncthreads();  // the rings become the staging tiles, Ut the diagonal block
    }
    // 3. the panel: warps J..nb-1
    if (warp >= J && warp < nb) {
      const int p = 32 * warp + lane;
      const bool valid = p < n;
      const int phys = valid ? s_perm[p] : 0;
      int pos = p - 32 * J, nswap = 0;
      if (valid && J + 1 < nb) {  // the row's next column block on its way into L2
        const double* nx = s_v.A + (int64_t)phys * n + 32 * (J + 1);
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(16, n - 32 * (J + 1) - 1)));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + min(31, n - 32 * (J + 1) - 1)));
      }
      const int info = panel(ps, acc, pos, valid, kb, warp - J, nb - J, stage, nswap);
      if (info) {
        if (tid == 32 * J) ps.info = 32 * J + info;
      } else {
        if (valid) s_perm[32 * J + pos] = phys;
        __syncwarp();
        const int off = phys * s_v.ldw, at = valid ? pos : n;
#pragma unroll 8
        for (int rr = 0; rr < 32; ++rr) {
          const int o = __shfl_sync(kAll, off, rr), p2 = __shfl_sync(kAll, at, rr);
          const double x = stage[rr * PS + lane];
          if (p2 < n && lane < kb) W[o + 32 * J + lane] = x;
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
        if (sa.state) sa.state[s_v.slot] = ps.info;
        if (sa.det) sa.det[s_v.idx] = 0.0;
        if (sa.sign) sa.sign[s_v.idx] = 0.0;
        if (sa.logabs) sa.logabs[s_v.idx] = -INFINITY;
        if (sa.info) sa.info[s_v.idx] = ps.info;
      }
      return;
    }
    // the diagonal block's inverses (U's for the substitution only) and the pivots' part of det / slogdet, each by
    // one warp, beside the other warps' loads of the next column block
    double* di = s_v.dinv + (int64_t)J * 2048;
    if (warp == 0) tri_inverse<kUnitLower, false>(D11, stage, kb, into(di));
    if ((sa.X || sa.inv) && warp == 1 % nw) tri_inverse<kUpper, true>(D11, stage, kb, into(di + 1024));
    if (warp == 2 % nw && (sa.det || sa.sign || sa.logabs)) {
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
          if (sa.det) sa.det[s_v.idx] = det;
          if (sa.sign) sa.sign[s_v.idx] = sg;
          if (sa.logabs) sa.logabs[s_v.idx] = la;
        }
      }
    }
  }
  for (int i = tid; i < n; i += blockDim.x) s_v.perm[i] = s_perm[i];
  if (tid == 0) {
    if (sa.state) sa.state[s_v.slot] = 0;
    if (sa.info) sa.info[s_v.idx] = 0;
  }
}

// ---------------------------------------------------------------------------
// Orders above 512: outer blocks of 128 columns. Rows keep their place in W, a copy
// of A; what moves is the permutation.
//  k_sys_outer   a cluster of CS CTAs per system factors the outer block's columns
//                over all rows that are left, left-looking inside the block like
//                k_sys_lu;
//  k_sys_rows    U12 = L11^-1 A12, a CTA per 32-column strip right of the block;
//  k_sys_gemm    A22 -= L21 U12, K = 128, 128 x 64 tiles, rows through the
//                permutation.
// The next outer block's columns are updated first and its panel then runs beside
// the rest of the update (run_sys_outer). The step-wise kernels this replaces
// updated the trailing matrix with K = 32 and so at the speed of memory, moved rows
// and took 2.4 us per column of a 1024-row panel.
//
// In the cluster block b of 32 positions (counted from the outer block's first)
// belongs to warp b / CS of CTA b % CS, so that every CTA keeps its share of the
// rows that are left. Per column the candidates (with their rows) go straight
// into every CTA's table, one cluster barrier, and every warp finds the winner in
// its own CTA's copy; the solved rows of a block step are pushed the same way (as
// in the substitution), the pivot rows of a panel group, the new positions and the
// diagonal block too. All warps take part in all cluster barriers.
struct __align__(16) Record {  // a warp's candidate
  Cand c;
  double rp, pad;
  double row[8];
};

struct __align__(16) ClusterShared {
  Record own[kMaxWarps];
  Record none;  // no candidate
  double raw[8][24];
  double l8[8][8];
  double u[24 * GS];
  double pv[32];  // the panel's pivots
};

// Whether the warps' candidates go into every CTA's table directly (a pair of
// CTAs), or the CTAs' best ones do: with more CTAs the fewer remote stores outweigh
// the extra stage. First outer block, us: 64 x 1024 on pairs 262 directly, 269 by
// CTA; 16 x 1024 on four 230 / 220; 8 x 4096 on eight 410 / 303.
__host__ __device__ constexpr bool outer_direct(int cs) { return cs == 2; }
constexpr int outer_smem(int warps, int cs) {
  return sys_cluster_smem(warps) + 2 * (outer_direct(cs) ? warps * cs : cs) * (int)sizeof(Record);
}

// The best candidate of a warp's lanes (a lane without one has in = false): its
// lane, or -1 if there is none. Decided on the high words without their last
// seven bits, which hold the lane, and exactly where that leaves a choice.
template <class Load>
__device__ __forceinline__ int best_lane(bool in, Load load) {
  constexpr unsigned kIdx = 127u;
  const int lane = threadIdx.x & 31;
  const unsigned key = in ? (load().hi & ~kIdx) | (kIdx - lane) : 0u;
  const unsigned mk = __reduce_max_sync(kAll, key);
  const unsigned amb = __ballot_sync(kAll, in && (key ^ mk) <= kIdx);
  if ((amb & (amb - 1)) == 0 && mk > kIdx) return (int)(kIdx - (mk & kIdx));
  Cand c{0u, 0u, INT_MAX, 0};
  if (in) c = load();
  bool any;
  const bool best = exact_winner(c.hi, c.lo, c.pos, any);
  const unsigned who = __ballot_sync(kAll, best);
  return any ? 31 - __clz(who) : -1;
}

// As panel(), over the cluster. Every warp's candidate (direct), or the best of the
// CTA's, which its first warp finds, is pushed into every CTA's table; one cluster
// barrier, and every warp finds the winner in its own CTA's copy. slot: the warp's
// block relative to the panel's first, na: their number; [w0, w1): the CTA's
// active warps.
template <int CS>
__device__ __forceinline__ int cluster_panel(ClusterShared& sh, Record* table, Acc<4>& acc, int& pos, bool valid,
                                             bool active, int kb, int slot, int na, int w0, int w1, double* tile,
                                             int& nswap) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  cg::cluster_group cl = cg::this_cluster();
  Record* own = &sh.own[warp];
  constexpr bool kDirect = outer_direct(CS);
  const int rank = (int)cl.block_rank(), threads = blockDim.x, entries = kDirect ? na : CS;
  const int mine_at = kDirect ? slot : rank;  // this record's place in the tables
  // 16-byte piece lane % 6 of the record to CTA lane / 6, and to CTA lane / 6 + 5
  const int to = lane / 6, piece = lane - 6 * to;
  double2* dst0 = nullptr;
  double2* dst1 = nullptr;
  if (kDirect ? active : warp == 0) {
    if (lane < 30 && to < CS) dst0 = reinterpret_cast<double2*>(cl.map_shared_rank(table + mine_at, to)) + piece;
    if (lane < 30 && to + 5 < CS)
      dst1 = reinterpret_cast<double2*>(cl.map_shared_rank(table + mine_at, to + 5)) + piece;
  }
  if (!kDirect && warp == 0) {
    if (lane == 0) sh.none.c = Cand{0u, 0u, INT_MAX, 0};
    __syncwarp();
  }
  unsigned live = valid ? 0x7fffffffu : 0u;
#pragma unroll 1
  for (int j0 = 0; j0 < kb; j0 += 8) {
    double a[8];
    if (active) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        double* o = tile + (16 * m + g) * PS + j0 + 2 * t;
        *reinterpret_cast<double2*>(o) = make_double2(acc.v[m][0][0], acc.v[m][0][1]);
        *reinterpret_cast<double2*>(o + 8 * PS) = make_double2(acc.v[m][0][2], acc.v[m][0][3]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 x = active ? *reinterpret_cast<const double2*>(tile + lane * PS + j0 + c) : make_double2(0.0, 0.0);
      a[c] = x.x;
      a[c + 1] = x.y;
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int j = j0 + s;
      if (j < kb) {  // uniform
        Record* tab = table + (s & 1) * entries;
        const int at = (s & 1) * entries * (int)(sizeof(Record) / 16);
        if (active) {  // uniform in the warp
          const unsigned hi = (unsigned)__double2hiint(a[s]) & live;
          const unsigned mh = __reduce_max_sync(kAll, hi);
          const double rp = kDirect ? 1.0 / (hi ? a[s] : 1.0) : 0.0;  // every candidate's, beside the reduction
          const bool me = hi == mh;
          const unsigned top = __ballot_sync(kAll, me);
          auto publish = [&](unsigned h, unsigned l, double r) {
            own->c = Cand{h, l, pos, 0};
            if (kDirect) own->rp = r;
#pragma unroll
            for (int c = s & ~1; c < 8; c += 2)
              *reinterpret_cast<double2*>(&own->row[c]) = make_double2(a[c], a[c + 1]);
          };
          if (me) publish(hi, (unsigned)__double2loint(a[s]), rp);
          if ((top & (top - 1)) != 0 || mh >= kInf) {
            unsigned h = (unsigned)__double2hiint(a[s]) & 0x7fffffffu, l = (unsigned)__double2loint(a[s]);
            if (!live || h > kInf || (h == kInf && l)) h = l = 0;
            bool any;
            const bool win = exact_winner(h, l, pos, any);
            __syncwarp();
            if (win) publish(h, l, kDirect ? 1.0 / a[s] : 0.0);
            else if (!any && lane == 0) own->c = Cand{0u, 0u, INT_MAX, 0};
          }
          if (kDirect) {
            __syncwarp();
            if (dst0) dst0[at] = reinterpret_cast<const double2*>(own)[piece];
          }
        }
        if constexpr (!kDirect) {  // the CTA's best candidate: its first warp waits for the others
          if (warp == 0) {
            asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory");
            const int w = best_lane(lane < w1 - w0, [&] { return sh.own[w0 + lane].c; });
            const Record* best = w < 0 ? &sh.none : &sh.own[w0 + w];
            double2 x = reinterpret_cast<const double2*>(best)[piece];
            if (piece == 1) x.x = 1.0 / best->row[s];  // one reciprocal a CTA, not one a warp
            if (dst0) dst0[at] = x;
            if (dst1) dst1[at] = x;
            __syncwarp();
          } else {
            __syncwarp();
            asm volatile("bar.arrive 1, %0;\n" ::"r"(threads) : "memory");
          }
        }
        cl.sync();
        const int gw = best_lane(lane < entries, [&] { return tab[lane].c; });
        if (gw < 0) return j + 1;  // the same in every warp of the cluster
        const double r = tab[gw].rp;
        const int gk = tab[gw].c.pos;
        const double* prow = tab[gw].row;
        if (threadIdx.x == 0) sh.pv[j] = prow[s];
        const bool chosen = valid && pos == gk;
        if (pos == j) pos = gk;
        if (chosen) {
          pos = j;
          live = 0;
        }
        nswap += gk != j;
        const double f = live ? a[s] * r : 0.0;
        if (live) a[s] = f;
#pragma unroll
        for (int c = s + 1; c < 8; ++c) a[c] = fma(-f, prow[c], a[c]);
      }
    }
    if (active) {
#pragma unroll
      for (int c = 0; c < 8; c += 2)
        *reinterpret_cast<double2*>(tile + lane * PS + j0 + c) = make_double2(a[c], a[c + 1]);
    }
    if (j0 + 8 >= kb) break;
    // the row's step in the group; 8: still below, -1: done before (or no row)
    const bool in_group = valid && !live && pos >= j0 && pos < j0 + 8;
    const int mine = live ? 8 : in_group ? pos - j0 : -1;
    double2 l[4];
    if (active) {
      if (in_group) {
        for (int to = 0; to < CS; ++to) {
          double2* o = reinterpret_cast<double2*>(cl.map_shared_rank(&sh.l8[pos - j0][0], to));
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c] = make_double2(a[2 * c], a[2 * c + 1]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int lim = __shfl_sync(kAll, mine, 8 * i + g);
        if (lim >= 0 && lim < 8) {
          for (int to = 0; to < CS; ++to) {
            double* o = cl.map_shared_rank(&sh.raw[lim][2 * t], to);
#pragma unroll
            for (int ni = 1; ni < 4; ++ni)
              *reinterpret_cast<double2*>(o + 8 * (ni - 1)) =
                  make_double2(acc.v[i >> 1][ni][2 * (i & 1)], acc.v[i >> 1][ni][2 * (i & 1) + 1]);
          }
        }
        l[i] = *reinterpret_cast<const double2*>(tile + (8 * i + g) * PS + j0 + 2 * t);
        if (2 * t >= lim) l[i].x = 0.0;
        if (2 * t + 1 >= lim) l[i].y = 0.0;
      }
    }
    cl.sync();
    if (warp == 0) {
      const int c = min(lane, 23);
      double x[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) x[s] = sh.raw[s][c];
#pragma unroll
      for (int q = 0; q < 7; ++q)
#pragma unroll
        for (int s = q + 1; s < 8; ++s) x[s] = fma(-sh.l8[s][q], x[q], x[s]);
      if (lane < 24) {
#pragma unroll
        for (int s = 0; s < 8; s += 2)
          *reinterpret_cast<double2*>(&sh.u[lane * GS + s]) = make_double2(-x[s], -x[s + 1]);
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int ni = 1; ni < 4; ++ni) {
        const double2 b = *reinterpret_cast<const double2*>(&sh.u[(8 * (ni - 1) + g) * GS + 2 * t]);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          dmma1688(acc.v[m][ni], l[2 * m], l[2 * m + 1], b);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc.v[m][ni - 1][e] = acc.v[m][ni][e];
        }
      }
    }
  }
  return 0;
}

// The outer block of blocks [jb, je). perm_in: the positions so far, perm_out: with
// this block's pivots (the update beside it reads the former). running: det,
// log|det| and sign by slot.
template <int CS>
__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_outer(SysArgs sa, const int32_t* __restrict__ perm_in, int32_t* __restrict__ perm_out,
            double* __restrict__ running, int jb, int je) {
  extern __shared__ __align__(16) double sm[];
  __shared__ ClusterShared sh;
  __shared__ int s_perm[kSysMaxN];  // the rows at this CTA's positions
  __shared__ double s_det[3];       // det, log|det|, sign (CTA 0)
  __shared__ View s_v;
  __shared__ int s_skip;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rank = (int)blockIdx.x % CS;
  double* Tb = sm + kTb;
  double* Li = sm + kLi;
  double* U0 = sm + kUt;
  double* U1 = sm + kWarp + nw * kPerWarp;
  Record* table = reinterpret_cast<Record*>(U1 + 32 * US);
  double* D11 = Tb;
  double* stage = sm + kWarp + warp * kPerWarp;
  const unsigned ring = smem(stage) + 16 * lane;
  const int sys = (int)blockIdx.x / CS;
  if (tid == 0) {
    s_v = view(sa, sys);
    s_skip = jb > 0 && sa.state[s_v.slot];
    const double* run = running + 3 * (int64_t)s_v.slot;
    s_det[0] = jb ? run[0] : 1.0;
    s_det[1] = jb ? run[1] : 0.0;
    s_det[2] = jb ? run[2] : 1.0;
  }
  __syncthreads();
  if (s_skip) return;  // the same for every CTA of the cluster
  double* const W = s_v.W;
  const int n = s_v.n, nb = sys_blocks(n), ldw = s_v.ldw;
  const int blk = jb + warp * CS + rank;  // the warp's block
  const int32_t* pin = perm_in + (int64_t)sys * n;
  int32_t* pout = perm_out + (int64_t)sys * n;
  for (int i = tid; i < 32 * nw; i += blockDim.x) {
    const int p = 32 * (jb + (i >> 5) * CS + rank) + (i & 31);
    s_perm[i] = p >= n ? 0 : jb ? pin[p] : p;
  }
  for (int p = rank * blockDim.x + tid; p < 32 * jb; p += CS * blockDim.x) pout[p] = pin[p];
  cl.sync();

  for (int J = jb; J < je; ++J) {
    const int kb = min(32, n - 32 * J);
    // the warp's rows of the column block
    Acc<4> acc;
    Rows r;
    r.live = n - 32 * blk - g;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool ok = 8 * i < r.live;
      const int row = ok ? s_perm[32 * warp + 8 * i + g] : 0;
      r.off[i] = (unsigned)row * ldw * 8;
      const double* src = W + (int64_t)row * ldw;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int col = 32 * J + 8 * ni + 2 * t;
        double2 x = make_double2(0.0, 0.0);
        if (ok && col < n) {
          x = __ldcg(reinterpret_cast<const double2*>(src + col));  // the pair ends inside the row's padding
          if (col + 1 >= n) x.y = 0.0;
        }
        acc.v[i >> 1][ni][2 * (i & 1)] = x.x;
        acc.v[i >> 1][ni][2 * (i & 1) + 1] = x.y;
      }
    }
    // the block's earlier columns
    if (J > jb) {
      const int first = jb + rank;                   // this CTA's first block
      if (J - 1 == first) __syncthreads();           // its inverse has just been written
      if (first < J) fetch_inverse(Li, s_v.dinv + (int64_t)first * 2048, blockDim.x);
      else cp_commit();
      ring_start<true, false>(ring, W, r, jb, n, blk > jb && blk < nb);
      for (int K = jb; K < J; ++K) {
        double* Ut = K & 1 ? U1 : U0;
        const bool mine = (K - jb) % CS == rank;
        if (mine) {
          if (K == first) __syncthreads();  // the inversions are done with the diagonal block in Tb
          if (blk == K) store_tile<4>(Tb, acc);
          cp_wait<2>();  // the inverse; at most two operand stages stay in flight
          __syncthreads();
          tile_product<4, false, CS>(Li, Tb, Ut);
        }
        cl.sync();
        if (blk > K && blk < nb) {
          update<4, true, false>(acc, ring, W, r, smem(Ut + g * US + 2 * t), K, K + 1, K + 1 < J && blk > K + 1, n);
        } else {
          if (mine && blk <= K) {  // the owner's warps that are done: U out, its next inverse in
            const int free = (K - jb) / CS + 1;
            if (K + CS < J) fetch_inverse(Li, s_v.dinv + (int64_t)(K + CS) * 2048, 32 * free);
            product_out<4, true>(Ut, ldw - 32 * J, 0, free,
                                 [&](int row) { return W + (int64_t)s_perm[(K - jb) / CS * 32 + row] * ldw + 32 * J; });
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) cp_commit();  // the waits count groups
        }
      }
      cp_wait<0>();
      __syncwarp();  // the ring becomes the staging tile
    }
    // the panel
    const bool active = blk >= J && blk < nb, valid = active && lane < n - 32 * blk;
    const int phys = valid ? s_perm[32 * warp + lane] : 0;
    int pos = 32 * (blk - J) + lane, nswap = 0;
    // the CTA's warps whose blocks lie in [J, nb)
    const int w0 = max(0, (J - jb - rank + CS - 1) / CS), w1 = min(nw, max(w0, (nb - jb - rank + CS - 1) / CS));
    const int info = cluster_panel<CS>(sh, table, acc, pos, valid, active, kb, blk - J, nb - J, w0, w1, stage, nswap);
    if (info) {  // the same in every thread of the cluster; nothing is on its way to another CTA
      if (tid == 0 && rank == 0) {
        sa.state[s_v.slot] = 32 * J + info;
        if (sa.det) sa.det[s_v.idx] = 0.0;
        if (sa.sign) sa.sign[s_v.idx] = 0.0;
        if (sa.logabs) sa.logabs[s_v.idx] = -INFINITY;
        if (sa.info) sa.info[s_v.idx] = 32 * J + info;
      }
      return;
    }
    if (active) {
      if (valid) {
        const int b = J - jb + (pos >> 5);
        cl.map_shared_rank(s_perm, b % CS)[b / CS * 32 + (pos & 31)] = phys;
      }
      __syncwarp();
      double* d11 = cl.map_shared_rank(D11, (J - jb) % CS);
      const int off = phys * ldw, at = valid ? pos : n;
#pragma unroll 8
      for (int rr = 0; rr < 32; ++rr) {
        const int o = __shfl_sync(kAll, off, rr), p2 = __shfl_sync(kAll, at, rr);
        const double x = stage[rr * PS + lane];
        if (p2 < n && lane < kb) W[o + 32 * J + lane] = x;
        if (p2 < kb) d11[p2 * PS + lane] = x;
      }
    }
    cl.sync();  // rows, positions and the diagonal block are everywhere
    double* di = s_v.dinv + (int64_t)J * 2048;
    if ((J - jb) % CS == rank) {
      if (warp == 0) tri_inverse<kUnitLower, false>(D11, stage, kb, into(di));
      if ((sa.X || sa.inv) && warp == 1 % nw) tri_inverse<kUpper, true>(D11, stage, kb, into(di + 1024));
    }
    if (rank == 0 && warp == 2 % nw) {
      // folded in the reference's order (linalg.cpp:400-403, 425-431)
      const double pv = lane < kb ? sh.pv[lane] : 1.0;
      const double lg = log(fabs(pv)), sgn = pv / fabs(pv);
      double det = s_det[0], la = s_det[1], sg = s_det[2];
      if (nswap & 1) {
        det = -det;
        sg = -sg;
      }
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
        if (J + 1 == je) {
          double* run = running + 3 * (int64_t)s_v.slot;
          run[0] = det;
          run[1] = la;
          run[2] = sg;
        }
        if (J + 1 == nb) {
          if (sa.det) sa.det[s_v.idx] = det;
          if (sa.sign) sa.sign[s_v.idx] = sg;
          if (sa.logabs) sa.logabs[s_v.idx] = la;
        }
      }
    }
  }
  for (int i = tid; i < 32 * nw; i += blockDim.x) {
    const int p = 32 * (jb + (i >> 5) * CS + rank) + (i & 31);
    if (p < n) pout[p] = s_perm[i];
  }
  if (tid == 0 && rank == 0) {
    sa.state[s_v.slot] = 0;
    if (sa.info && je == nb) sa.info[s_v.idx] = 0;
  }
}

// U12 on columns [c0 + 32 blockIdx.x, +32) of system blockIdx.y: the outer block's
// rows (four blocks, a warp each), forward substitution as in solve_strip.
__global__ void __launch_bounds__(128, 4)
k_sys_rows(SysArgs sa, const int32_t* __restrict__ perm, int jb, int je, int c0, int c1) {
  extern __shared__ __align__(16) double sm[];
  __shared__ View s_v;
  __shared__ int s_perm[128], s_skip;
  double* Tb = sm + kTb;
  double* Li = sm + kLi;
  double* Ut = sm + kUt;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const unsigned ring = smem(sm + kWarp + warp * kPerWarp) + 16 * lane;
  if (threadIdx.x == 0) {
    s_v = view(sa, blockIdx.y);
    s_skip = sa.state[s_v.slot];
  }
  __syncthreads();
  if (s_skip) return;
  const int n = s_v.n, ldw = s_v.ldw, cols = je - jb;
  double* const W = s_v.W;
  // an outer block that something lies right of is full
  s_perm[threadIdx.x] = (int)threadIdx.x < 32 * cols ? perm[(int64_t)blockIdx.y * n + 32 * jb + threadIdx.x] : 0;
  __syncthreads();
  const int col0 = c0 + 32 * (int)blockIdx.x;
  Acc<4> acc;
  Rows r;
  r.live = 32;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = s_perm[32 * warp + 8 * i + g];
    r.off[i] = (unsigned)row * ldw * 8;
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
      const int col = col0 + 8 * ni + 2 * t;
      double2 x = make_double2(0.0, 0.0);
      if (col < c1) x = *reinterpret_cast<const double2*>(W + (int64_t)row * ldw + col);
      acc.v[i >> 1][ni][2 * (i & 1)] = x.x;
      acc.v[i >> 1][ni][2 * (i & 1) + 1] = x.y;
    }
  }
  fetch_inverse(Li, s_v.dinv + (int64_t)jb * 2048, blockDim.x);
  ring_start<true, false>(ring, W, r, jb, n, warp > 0 && warp < cols);
  for (int K = 0; K < cols; ++K) {
    if (warp == K) store_tile<4>(Tb, acc);
    cp_wait<2>();
    __syncthreads();
    tile_product<4, false, 1>(Li, Tb, Ut);
    __syncthreads();
    if (warp > K && warp < cols) {
      update<4, true, false>(acc, ring, W, r, smem(Ut + g * US + 2 * t), jb + K, jb + K + 1, warp > K + 1, n);
    } else {
      if (warp <= K) {
        if (K + 1 < cols) fetch_inverse(Li, s_v.dinv + (int64_t)(jb + K + 1) * 2048, 32 * (K + 1));
        product_out<4, true>(Ut, c1 - col0, 0, K + 1,
                             [&](int row) { return W + (int64_t)s_perm[32 * K + row] * ldw + col0; });
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) cp_commit();
    }
  }
}

// A22 -= L21 U12 on columns [c0, c1): one CTA per 128 x 64 tile (grid.z = system).
// Positions p0 + 128 y .. of the permutation give the rows; K = the outer block's
// 128 columns in eight slabs of 16 through a ring of three (cp.async, 16 bytes).
// Eight warps of 32 x 32 accumulators; the C tile is read while the first slabs
// arrive. Bounds: FP64 tensor throughput (a tile is 8.4 us of an SM's pipe against
// 128 KB of C read and written), two CTAs per SM to cover the ends of a tile.
constexpr int GM = 128, GN = 64, GK = 16, GSTAGES = 3;
constexpr int GBS = GN + 2;  // row stride of a U slab (8-byte reads down a column: banks 4t + g)
constexpr int kGemmSlab = GM * GK + GK * GBS;
constexpr int kGemmSmem = 8 * GSTAGES * kGemmSlab;

__global__ void __launch_bounds__(256, 2)
k_sys_gemm(SysArgs sa, const int32_t* __restrict__ perm, int jb, int je, int c0, int c1) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_up[128], s_row[GM], s_skip;
  __shared__ View s_v;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    s_v = view(sa, blockIdx.z);
    s_skip = sa.state[s_v.slot];
  }
  __syncthreads();
  if (s_skip) return;
  const int n = s_v.n, ldw = s_v.ldw;
  double* const W = s_v.W;
  const int p0 = 32 * je + GM * (int)blockIdx.y, col0 = c0 + GN * (int)blockIdx.x;
  const int32_t* pm = perm + (int64_t)blockIdx.z * n;
  if (tid < 128) s_row[tid] = p0 + tid < n ? pm[p0 + tid] : -1;
  else s_up[tid - 128] = pm[32 * jb + tid - 128];
  __syncthreads();
  // rows of a slab: 16-byte piece c of row r at piece c ^ 4 (r & 1): two neighbouring
  // rows fall into the two halves of the banks
  auto load = [&](int slab) {
    double* a = sm + slab % GSTAGES * kGemmSlab;
    double* b = a + GM * GK;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + 256 * i, r = idx >> 3, c = idx & 7, row = s_row[r];
      const double* src = W + (int64_t)max(row, 0) * ldw + 32 * jb + GK * slab + 2 * c;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem(a + r * GK + 2 * (c ^ 4 * (r & 1)))),
                   "l"(src), "r"(row >= 0 ? 16 : 0));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = tid + 256 * i, r = idx >> 5, c = (idx & 31) * 2;
      const int col = min(col0 + c, ldw - 2);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem(b + r * GBS + c)),
                   "l"(W + (int64_t)s_up[GK * slab + r] * ldw + col));
    }
    cp_commit();
  };
  constexpr int kSlabs = 128 / GK;
  load(0);
  load(1);
  const int wm = 32 * (warp >> 1), wn = 32 * (warp & 1);
  double acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = s_row[wm + 16 * m + 8 * h + g];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int col = col0 + wn + 8 * ni + 2 * t;
        double2 x = make_double2(0.0, 0.0);
        if (row >= 0 && col < c1) x = *reinterpret_cast<const double2*>(W + (int64_t)row * ldw + col);
        acc[m][ni][2 * h] = -x.x;  // the tile accumulates L U - A and is negated on the way out
        acc[m][ni][2 * h + 1] = -x.y;
      }
    }
  for (int k = 0; k < kSlabs; ++k) {
    cp_wait<1>();
    __syncthreads();  // slab k is here, and slab k - 1 has been read
    if (k + 2 < kSlabs) load(k + 2);
    else cp_commit();
    const double* a = sm + k % GSTAGES * kGemmSlab;
    const double* b = a + GM * GK;
#pragma unroll
    for (int q = 0; q < GK / 8; ++q) {
      double2 av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = wm + 8 * i + g;
        av[i] = *reinterpret_cast<const double2*>(a + r * GK + 2 * ((4 * q + t) ^ 4 * (r & 1)));
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const double* p = b + (8 * q + 2 * t) * GBS + wn + 8 * ni + g;
        bv[ni] = make_double2(p[0], p[GBS]);
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
      const int row = s_row[wm + 16 * m + 8 * h + g];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int col = col0 + wn + 8 * ni + 2 * t;
        if (row >= 0 && col < c1)
          *reinterpret_cast<double2*>(W + (int64_t)row * ldw + col) =
              make_double2(-acc[m][ni][2 * h], -acc[m][ni][2 * h + 1]);
      }
    }
}

// W <- A, rows padded to the workspace's leading dimension (zeros).
__global__ void __launch_bounds__(256)
k_sys_copy(const double* __restrict__ A, double* __restrict__ W, int64_t rows, int n, int ldw) {
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 8)
    for (int c = threadIdx.x & 31; c < ldw; c += 32) W[r * ldw + c] = c < n ? __ldcs(A + r * n + c) : 0.0;
}

// ---------------------------------------------------------------------------
// Substitution of one strip: C = P B (or P times columns of the identity), then
// Y_K = L_KK^-1 C_K and C_w -= L_wK Y_K downwards, X_K = U_KK^-1 Y_K and
// Y_w -= U_wK X_K upwards.

struct Strip {  // what the inner loops do not need, in shared memory
  View v;
  const double* B;
  double* X;  // column c0 of row 0
  int ldx, c0, width, inverse;
};

// In a cluster of CS CTAs (orders above 512, or few strips) block b belongs to warp
// b / CS of CTA b % CS. The owner of block K pushes the solved rows into every
// CTA; U alternates between two tiles, so that one cluster barrier per block
// suffices: a tile is rewritten two blocks later, after the barrier in between
// that every CTA passes with its update done.
template <int NI, bool VEC, int CS>
__device__ __forceinline__ void solve_strip(const SysArgs& sa, const Strip& s, double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int rank = CS > 1 ? (int)blockIdx.x % CS : 0;
  const int blk = warp * CS + rank;  // the warp's block
  double* Tb = sm + kTb;
  double* Li = sm + kLi;
  double* U0 = sm + kUt;
  double* U1 = CS > 1 ? sm + kWarp + nw * kPerWarp : U0;
  const int g = lane >> 2, t = lane & 3;
  const unsigned ring = smem(sm + kWarp + warp * kPerWarp) + 16 * lane;
  const double* const W = s.v.W;
  const int n = s.v.n, nb = sys_blocks(n);
  if constexpr (CS > 1) cluster_arrive();
  const unsigned marks = CS == 1 ? tri_marks(s.v.dinv, nb) : 0u;
  Acc<NI> acc;
  Rows r;
  r.live = n - 32 * blk - g;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = 32 * blk + 8 * i + g;
    const bool ok = p < n;
    const int row = ok ? s.v.perm[p] : 0;
    r.off[i] = (unsigned)(sa.w_by_position ? (ok ? p : 0) : row) * s.v.ldw * 8;
#pragma unroll
    for (int ni = 0; ni < NI; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = 8 * ni + 2 * t + e;
        double x = 0.0;
        if (ok && col < s.width)
          x = s.inverse ? (row == s.c0 + col ? 1.0 : 0.0) : s.B[(int64_t)row * s.ldx + col];
        acc.v[i >> 1][ni][2 * (i & 1) + e] = x;
      }
  }
  // One block: the owner's rows times the inverse, to every CTA of the cluster.
  auto solve_block = [&](int K, double* Ut, auto upper) {
    if (CS == 1 || K % CS == rank) {
      if (blk == K) store_tile<NI>(Tb, acc);
      cp_wait<2>();  // the inverse; at most two operand stages stay in flight
      __syncthreads();
      constexpr bool kUp = decltype(upper)::value;
      const bool marked = CS == 1 ? marks >> (kUp ? K + 16 : K) & 1 : tri_marked<kUp>(Li);  // uniform
      if (!marked) {
        tile_product<NI, kUp, CS>(Li, Tb, Ut);
      } else {
        tile_substitute<NI, kUp>(Li, Tb);
        __syncthreads();
        tile_negate<NI, CS>(Tb, Ut);
      }
    }
    if constexpr (CS > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  // A CTA fetches the inverse of its own next block, by the warps that have
  // nothing to update.
  if (rank < nb) fetch_inverse(Li, s.v.dinv + rank * 2048, blockDim.x);
  else cp_commit();
  ring_start<VEC, false>(ring, W, r, 0, n, blk > 0 && blk < nb);
  if constexpr (CS > 1) cluster_wait();  // every CTA runs: block 0's rows may be pushed
  for (int K = 0; K < nb; ++K) {
    double* Ut = K & 1 ? U1 : U0;
    solve_block(K, Ut, std::false_type{});
    if (blk > K && blk < nb) {
      update<NI, VEC, false>(acc, ring, W, r, smem(Ut + g * US + 2 * t), K, K + 1, blk > K + 1, n);
    } else {
      if (K % CS == rank && blk <= K) {
        // the next L_KK^-1; after the CTA's last one its first U_KK^-1 (same block)
        const int free = K / CS + 1;
        fetch_inverse(Li, s.v.dinv + (K + CS < nb ? (K + CS) * 2048 : K * 2048 + 1024), 32 * free);
      }
      if (blk == K) {  // Y_K back into its owner's registers for the way up
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
  ring_start<VEC, true>(ring, W, r, nb - 1, n, blk < nb - 1);
  for (int K = nb - 1; K >= 0; --K) {
    // the tiles go on alternating: the last block of the way down used tile (nb - 1) & 1
    double* Ut = (nb - 1 - K) & 1 ? (nb & 1 ? U0 : U1) : (nb & 1 ? U1 : U0);
    solve_block(K, Ut, std::true_type{});
    if (blk < K) {
      update<NI, VEC, true>(acc, ring, W, r, smem(Ut + g * US + 2 * t), K, K - 1, blk < K - 1, n);
    } else {
      if (K % CS == rank) {
        const int first = K / CS, free = nw - first;
        if (K >= CS) fetch_inverse(Li, s.v.dinv + (K - CS) * 2048 + 1024, 32 * free, 32 * first);
        product_out<NI, false>(Ut, s.width, first, free, [&](int row) {
          return 32 * K + row < n ? s.X + (int64_t)(32 * K + row) * s.ldx : nullptr;
        });
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) cp_commit();
    }
  }
  if constexpr (CS > 1) cg::this_cluster().sync();  // no CTA leaves while another may still write to it
}

// A kernel per strip width: narrow strips need fewer registers, so more of their
// CTAs share an SM. items == nullptr: strips `first` .. `first` + `per` - 1 of the
// right-hand sides (inverse: of the inverse) of every system of a uniform batch.
template <int NI, bool VEC, int CS>
__global__ void __launch_bounds__(kSysMaxN, 1)
k_sys_solve(SysArgs sa, const SysItem* __restrict__ items, int inverse, int first, int per) {
  extern __shared__ __align__(16) double sm[];
  __shared__ Strip s_s;
  __shared__ int s_skip;
  if (threadIdx.x == 0) {
    const int b = (int)blockIdx.x / CS;
    SysItem it;
    if (items) {
      it = items[b];
    } else {
      it.sys = b / per;
      it.inverse = (int16_t)inverse;
      it.c0 = 32 * (first + b - it.sys * per);
      it.width = (int16_t)min(32, (inverse ? sa.un : sa.unrhs) - it.c0);
    }
    const View v = view(sa, it.sys);
    s_s.v = v;
    s_s.inverse = it.inverse;
    s_s.c0 = it.c0;
    s_s.width = it.width;
    s_s.ldx = it.inverse ? v.n : v.nrhs;
    s_s.B = sa.B + v.b_off + it.c0;
    s_s.X = (it.inverse ? sa.inv + v.inv_off : sa.X + v.b_off) + it.c0;
    s_skip = sa.state && sa.state[v.slot];  // singular: nothing to solve with
  }
  __syncthreads();
  if (!s_skip) solve_strip<NI, VEC, CS>(sa, s_s, sm);  // the same for every CTA of a cluster
}

// ---------------------------------------------------------------------------
// Kept factors: the permutation of the swap list (every thread follows its own
// rows through the swaps; the list is read by broadcast) in CTA (s, 0), the
// diagonal blocks' inverses in the CTAs (s, b + 1).
__global__ void __launch_bounds__(64)
k_sys_prepare(SysArgs sa, const int32_t* __restrict__ ipiv) {
  __shared__ double D[32 * PS];
  __shared__ double X[2][32 * TS];
  const View v = view(sa, blockIdx.x);
  const int n = v.n, b = (int)blockIdx.y - 1;
  if (b < 0) {
    extern __shared__ int piv[];
    const int32_t* src = ipiv + (int64_t)blockIdx.x * n;
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
  if (threadIdx.x >= 32) tri_inverse<kUpper, true>(D, X[1], kb, into(di + 1024));
  else tri_inverse<kUnitLower, true>(D, X[0], kb, into(di));
}

}  // namespace

cudaError_t launch_sys_lu(const SysArgs& sa, const int32_t* list, int nsys, int nmax, cudaStream_t st) {
  if (nsys <= 0) return cudaSuccess;
  if (nmax > kSysMaxN) return cudaErrorInvalidValue;
  const int nw = sys_blocks(nmax);
  k_sys_lu<<<nsys, 32 * nw, sys_smem(nw), st>>>(sa, list);
  return cudaGetLastError();
}

namespace {

template <int CS>
cudaError_t launch_outer1(const SysArgs& sa, const int32_t* pin, int32_t* pout, double* running, int nsys, int jb,
                          int je, cudaStream_t st) {
  const int blocks = sys_blocks(sa.un) - jb, nw = std::max(1, (blocks + CS - 1) / CS);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)nsys * CS);
  cfg.blockDim = dim3(32 * nw);
  cfg.dynamicSmemBytes = outer_smem(nw, CS);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sys_outer<CS>, sa, pin, pout, running, jb, je);
}

template <int CS>
cudaError_t prepare_outer() {
  return cudaFuncSetAttribute(k_sys_outer<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              outer_smem(kMaxWarps, CS));
}

}  // namespace

cudaError_t launch_sys_outer(const SysArgs& sa, const int32_t* pin, int32_t* pout, double* running, int nsys, int jb,
                             int je, cudaStream_t st) {
  const int cs = sys_outer_cluster(32 * (sys_blocks(sa.un) - jb), nsys);
  switch (cs) {
    case 2: return launch_outer1<2>(sa, pin, pout, running, nsys, jb, je, st);
    case 4: return launch_outer1<4>(sa, pin, pout, running, nsys, jb, je, st);
    case 8: return launch_outer1<8>(sa, pin, pout, running, nsys, jb, je, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_sys_update(const SysArgs& sa, const int32_t* perm, int nsys, int jb, int je, int c0, int c1,
                              cudaStream_t st) {
  if (c0 >= c1) return cudaSuccess;
  if (nsys > 65535) return cudaErrorInvalidValue;
  k_sys_rows<<<dim3((unsigned)(c1 - c0 + 31) / 32, (unsigned)nsys), 128, sys_smem(4), st>>>(sa, perm, jb, je, c0, c1);
  const int rows = sa.un - 32 * je;
  if (rows > 0)
    k_sys_gemm<<<dim3((unsigned)(c1 - c0 + GN - 1) / GN, (unsigned)(rows + GM - 1) / GM, (unsigned)nsys), 256,
                 kGemmSmem, st>>>(sa, perm, jb, je, c0, c1);
  return cudaGetLastError();
}

cudaError_t launch_sys_copy(const SysArgs& sa, int nsys, cudaStream_t st) {
  if (sa.A == sa.W) return cudaSuccess;  // in place
  const int64_t rows = (int64_t)nsys * sa.un;
  k_sys_copy<<<(unsigned)std::min<int64_t>((rows + 7) / 8, 148 * 16), 256, 0, st>>>(sa.A, sa.W, rows, sa.un,
                                                                                    sys_ld(sa.un));
  return cudaGetLastError();
}

namespace {

template <int NI, bool VEC, int CS>
cudaError_t launch_strips3(const SysArgs& sa, const SysItem* items, int64_t nitems, int nmax, int inverse, int first,
                           int per, cudaStream_t st) {
  const int nw = (sys_blocks(nmax) + CS - 1) / CS;
  if constexpr (CS == 1) {
    k_sys_solve<NI, VEC, 1><<<(unsigned)nitems, 32 * nw, sys_smem(nw), st>>>(sa, items, inverse, first, per);
    return cudaGetLastError();
  } else {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nitems * CS);
    cfg.blockDim = dim3(32 * nw);
    cfg.dynamicSmemBytes = sys_cluster_smem(nw);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_sys_solve<NI, VEC, CS>, sa, items, inverse, first, per);
  }
}

template <int NI>
cudaError_t launch_strips(const SysArgs& sa, const SysItem* items, int64_t nitems, int nmax, int inverse, int first,
                          int per, cudaStream_t st) {
  if (nitems <= 0) return cudaSuccess;
  const int cs = sys_cluster(nmax, nitems);
  if (cs > 8 || nitems * cs > INT_MAX) return cudaErrorInvalidValue;
  // 16-byte operand loads: workspaces always, kept factors (uniform batches) of even order
  const bool vec = !sa.w_by_position || (sa.un % 2 == 0 && (reinterpret_cast<uintptr_t>(sa.W) & 15) == 0);
#define NPPB_STRIPS(CS)                                                                              \
  return vec ? launch_strips3<NI, true, CS>(sa, items, nitems, nmax, inverse, first, per, st)        \
             : launch_strips3<NI, false, CS>(sa, items, nitems, nmax, inverse, first, per, st)
  switch (cs) {
    case 1: NPPB_STRIPS(1);
    case 2: NPPB_STRIPS(2);
    case 4: NPPB_STRIPS(4);
    default: NPPB_STRIPS(8);
  }
#undef NPPB_STRIPS
}

cudaError_t launch_strips(const SysArgs& sa, const SysItem* items, int64_t nitems, int nmax, int width, int inverse,
                          int first, int per, cudaStream_t st) {
  switch (sys_width_class(width)) {
    case 0: return launch_strips<1>(sa, items, nitems, nmax, inverse, first, per, st);
    case 1: return launch_strips<2>(sa, items, nitems, nmax, inverse, first, per, st);
    default: return launch_strips<4>(sa, items, nitems, nmax, inverse, first, per, st);
  }
}

template <int NI, int CS>
cudaError_t prepare_strips1() {
  const int smem = CS == 1 ? sys_smem(kMaxWarps) : sys_cluster_smem(kMaxWarps);
  cudaError_t e = cudaFuncSetAttribute(k_sys_solve<NI, true, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sys_solve<NI, false, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  return e;
}

template <int NI>
cudaError_t prepare_strips() {
  cudaError_t e = prepare_strips1<NI, 1>();
  if (e == cudaSuccess) e = prepare_strips1<NI, 2>();
  if (e == cudaSuccess) e = prepare_strips1<NI, 4>();
  if (e == cudaSuccess) e = prepare_strips1<NI, 8>();
  return e;
}

}  // namespace

cudaError_t launch_sys_solve(const SysArgs& sa, const SysItem* items, int64_t nitems, int width, int nmax,
                             cudaStream_t st) {
  return launch_strips(sa, items, nitems, nmax, width, 0, 0, 1, st);
}

cudaError_t launch_sys_solve_uniform(const SysArgs& sa, int nsys, cudaStream_t st) {
  const int full = sa.unrhs / 32, rest = sa.unrhs % 32, ni = sa.uinv ? sys_blocks(sa.un) : 0;
  cudaError_t e = launch_strips(sa, nullptr, (int64_t)nsys * full, sa.un, 32, 0, 0, full, st);
  if (e == cudaSuccess && rest) e = launch_strips(sa, nullptr, nsys, sa.un, rest, 0, full, 1, st);
  if (e == cudaSuccess && ni) e = launch_strips(sa, nullptr, (int64_t)nsys * ni, sa.un, 32, 1, 0, ni, st);
  return e;
}

cudaError_t launch_sys_prepare(const SysArgs& sa, const int32_t* ipiv, int nsys, cudaStream_t st) {
  const dim3 grid((unsigned)nsys, (unsigned)sys_blocks(sa.un) + 1);
  k_sys_prepare<<<grid, 64, sizeof(int) * (size_t)sa.un, st>>>(sa, ipiv);
  return cudaGetLastError();
}

cudaError_t sys_prepare_kernels() {
  cudaError_t e = cudaFuncSetAttribute(k_sys_lu, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       sys_smem(kMaxWarps));
  if (e == cudaSuccess) e = prepare_outer<2>();
  if (e == cudaSuccess) e = prepare_outer<4>();
  if (e == cudaSuccess) e = prepare_outer<8>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sys_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, sys_smem(4));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_sys_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
  if (e == cudaSuccess) e = prepare_strips<1>();
  if (e == cudaSuccess) e = prepare_strips<2>();
  if (e == cudaSuccess) e = prepare_strips<4>();
  return e;
}

}  // namespace nppb
