// Batched least squares and singular values through one-sided Jacobi. C++20.
//
// The reference solves lstsq through its economy SVD, a cyclic one-sided
// Jacobi on the tall orientation (A, or A^T when m < n), and returns the
// solution, the residuals (overdetermined and full rank only), the rank at
// tol = (rcond < 0 ? eps * max(m, n) : rcond) * s_max and the singular values
// (src/linalg/linalg.cpp:620-712, 755-784). Here one CTA takes one problem of
// the batch, its matrices in shared memory (column-major):
//  1. tall problems are first reduced to their N x N triangle by Householder
//     reflections, a warp per trailing column, the right-hand sides carried
//     along as further columns (one barrier per reflection);
//  2. one-sided Jacobi on the triangle's columns (or on the matrix itself:
//     lsq_plan says when),
//     the pairs of a sweep in round-robin order: the N / 2 disjoint pairs of a
//     round run at once, eight lanes per pair, one barrier per round; up to 60
//     sweeps until the largest relative dot product is below 1e-15;
//  3. the column norms (the singular values, sorted descending), the rank,
//     x = V diag(1/s or 0) U^T b, or by substitution with a triangle of full
//     rank, and the residuals.
// Latency bounds it: N - 1 dependent rounds per sweep, each two dot-product
// reductions deep plus a division, a square root and a reciprocal square root.
// 1024 problems of 200 x 32 with one right-hand side, one B200: 0.68 ms, against
// 18.2 ms with the whole CTA on one pair after the other on all 200 rows (1.2 ms
// on the triangle with V accumulated and the angles in FP64).
// Sums run in a different order than the reference's, so the results agree
// within rounding, not bit for bit.
#include <cuda_runtime.h>

#include <cmath>
#include <new>

#include "../../include/numpp_b200.h"
#include "nppb_internal.hpp"
#include "runtime.hpp"

using namespace nppb;

namespace {

constexpr int LT = 256;               // threads per problem
constexpr int kLsqMaxN = 64;          // columns of the tall orientation
constexpr int kLsqMaxK = 64;          // right-hand sides
constexpr int32_t kLsqLeft = -1;      // rank of a problem that the first launch has left to the second
constexpr double kLsqMostA = 0x1p480, kLsqMostB = 0x1p900;  // largest magnitudes that are reduced to the triangle
constexpr size_t kLsqMaxSmem = 220 * 1024;  // dynamic shared memory of one problem
constexpr size_t kLsqHalfSmem = 112 * 1024;  // of two that share an SM

#define NPPB_CUDA(call, what)                            \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return cuda_status(e_, what); \
  } while (0)

// What one problem needs with its matrix, V and U^T b alone; larger problems
// are declined.
size_t lsq_base(int M, int N, int k) {
  return sizeof(double) * ((size_t)M * N + (size_t)N * N + (size_t)N * (k > 0 ? k : 1) + N + 3 * (LT / 32)) +
         sizeof(int) * (size_t)N;
}

// Shared memory of one problem (offsets in doubles).
struct LsqLayout {
  int ws, js, vs;     // column strides: the tall matrix, the Jacobi columns, V
  int qr;             // reduced to the triangle first
  int nbuf;           // right-hand sides carried through the reflections at once
  int buf, j, v, r;   // first double of the right-hand-side columns, Jacobi columns, V and the triangle
  int tau, head, diag, t1, sig, ord, doubles;
};

// Column stride = 8 modulo 16 doubles: the four lane groups of a warp work on
// neighbouring columns, which then fall into the two halves of the banks.
int lsq_stride8(int n) { return (n + 7) / 16 * 16 + 8; }

// nbuf: right-hand sides carried at once (at least 1 of k > 0); negative: no reduction.
LsqLayout lsq_layout(int m, int n, int k, int nbuf) {
  const int wide = m < n, M = wide ? n : m, N = wide ? m : n;
  LsqLayout l{};
  l.ws = M | 1;
  l.qr = nbuf >= 0 ? 1 : 0;
  int at = l.ws * N;
  if (l.qr) {
    l.js = l.vs = lsq_stride8(N);
    l.nbuf = nbuf;
    l.buf = at;
    at += l.nbuf * l.ws;
    // once every right-hand side has been carried along, nothing reads the
    // reflections any more, and what follows takes their place
    const bool over = !wide && k <= l.nbuf && 3 * l.js <= l.ws;
    int o = over ? 0 : at;
    l.j = o;
    l.v = o + l.js * N;
    l.r = o + 2 * l.js * N;
    o += 3 * l.js * N;
    if (!over) at = o;
  } else {
    l.js = l.ws;
    l.vs = lsq_stride8(N);
    if (lsq_base(M, N, k) + sizeof(double) * (size_t)(l.vs - N) * N > kLsqMaxSmem) l.vs = N;
    l.j = 0;
    l.v = at;
    at += l.vs * N;
  }
  l.tau = at;
  l.head = at + N;
  l.diag = at + 2 * N;
  if (l.qr) at += 3 * N;
  l.t1 = at;
  at += N * (k > 0 ? k : 1);
  l.sig = at;
  at += 2 * N;
  l.ord = at;
  at += (N + 1) / 2;
  l.doubles = at;
  return l;
}

// A round of at most four pairs of long columns: a warp a pair leaves most of the CTA
// idle, so the whole CTA takes one pair after the other (300 x 3 with rcond = 0: 32 us so, one
// problem; 6000 x 3: 79 us, 238 us with a warp a pair).
__host__ __device__ bool wide_pairs(int N, int rows) {
  const int E = N + (N & 1);
  return E <= 8 && rows > 100 * E;
}

// Reducing to the triangle pays for M >= 2 N (a sweep then runs on N instead
// of M rows) and N >= 3 (one or two columns have no sweeps to speak of: 64 x 1 takes 6
// us directly, 11 us with the reduction and its second launch). Right-hand sides in
// groups of fewer than four leave the CTA idle: 5000 x 4 with 20 takes 1045 us one by one,
// 429 us directly; so do long solutions of wide problems behind the first group (2048
// of 5 x 2000 with 20: 2110 us, 1441 us directly). Its rounding is at the level of the default tolerance's factor
// eps * max(m, n); a smaller rcond keeps the sweeps on the matrix itself, so
// that exactly dependent columns still give exact zeros there, and so do
// small problems, whose default tolerance is a few eps.
LsqLayout lsq_plan(int m, int n, int k, double rcond) {
  const int wide = m < n, M = wide ? n : m, N = wide ? m : n;
  const bool robust = rcond < 0 || rcond >= 2.220446049250313e-16 * M;
  if (M >= 2 * N && M >= 64 && N >= 3 && robust && !(wide && k > LT / 32 && wide_pairs(N, M))) {
    // the largest group of at least four that leaves room for two CTAs an SM, else that fits at all
    const int most = k < LT / 32 ? k : LT / 32, least = k < 4 ? k : 4;
    for (const size_t limit : {kLsqHalfSmem, kLsqMaxSmem})
      for (int nbuf = most; nbuf >= least; --nbuf) {
        const LsqLayout l = lsq_layout(m, n, k, nbuf);
        if (sizeof(double) * (size_t)l.doubles <= limit) return l;
      }
  }
  return lsq_layout(m, n, k, -1);
}

template <int W>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = W / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// x <- (I - tau v v^T) x on rows [q, M) by one warp; v = (head, w[q+1 .. M)).
__device__ __forceinline__ void reflect(const double* w, double head, double tau, double* x, int q, int M) {
  const int lane = threadIdx.x & 31;
  double d = 0.0;
  for (int r = q + lane; r < M; r += 32) d = fma(r == q ? head : w[r], x[r], d);
  d = lane_sum<32>(d) * tau;
  for (int r = q + lane; r < M; r += 32) x[r] = fma(-d, r == q ? head : w[r], x[r]);
}

// 2^e for |e| <= 1022, and the exponent of a non-negative number (-1023 for zero and denormals).
__device__ __forceinline__ double power2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ int exponent(double x) { return (__double2hiint(x) >> 20) - 1023; }

// The FP64 pipe (a warp instruction every two cycles) is what the rounds share:
// the angle, of which only c^2 + s^2 = 1 has to hold to the last bit, and the
// relative dot product, which is only compared with the threshold, are
// therefore taken in FP32 on values scaled into its range by powers of two. A
// rotation then leaves 1e-7 of the dot product instead of 1e-16, and the sweeps
// end on the same measured 1e-15.
// aa, bb: the columns' squared norms, cc their dot product. x_i <- cs x_i - sj x_j,
// x_j <- sn x_i + cj x_j; false: nothing to turn.
__device__ __forceinline__ bool jacobi_angle(double aa, double bb, double cc, float& worst, double& cs, double& sn,
                                             double& sj, double& cj) {
  if (!(aa > 0.0) || !(bb > 0.0) || !(fabs(cc) > 0.0)) return false;  // nothing to turn (or a NaN)
  if (isinf(aa) || isinf(bb) || isinf(cc)) return false;
  // |cc| / sqrt(aa bb): aa and bb scaled to [1, 4) by even powers of two
  const int ea = max(min(exponent(aa), 1022), -1022) & ~1, eb = max(min(exponent(bb), 1022), -1022) & ~1;
  const float fa = (float)(aa * power2(-ea)), fb = (float)(bb * power2(-eb));
  const float fc = (float)(fabs(cc) * power2(-((ea + eb) / 2)));
  worst = fmaxf(worst, fc * rsqrtf(fa * fb));
  // tan of the rotation angle, the smaller root of t^2 + 2 zeta t - 1 = 0 with
  // zeta = (bb - aa) / (2 |cc|); both legs halved and scaled by one power of two. An
  // angle near or below FP32's range (columns of very different lengths) would
  // never turn the pair: there the root is 1 / (2 zeta) to the last bit.
  const double p = fabs(0.5 * bb - 0.5 * aa), s1 = fabs(cc);
  const double down = power2(-max(min(max(exponent(p), exponent(s1)), 1022), -1022));
  const float fp = (float)(p * down), fs = (float)(s1 * down);
  double td = fs / (fp + sqrtf(fmaf(fp, fp, fs * fs)));
  if (fs < 0x1p-60f * fp) td = 0.5 * (s1 / p);
  if (bb < aa) td = -td;
  cs = rsqrt(fma(td, td, 1.0));
  sn = cs * td;
  sj = cc < 0.0 ? -sn : sn;
  cj = cc < 0.0 ? -cs : cs;
  return true;
}

// One-sided Jacobi on N columns of `rows` rows at J (stride js), the rotations
// accumulated in V (stride vs) with VECS. In round t of the round-robin over an
// even number E of players, E - 1 meets t and the others meet the one with
// t + p = t - p (mod E - 1): E / 2 disjoint pairs, LP lanes each (R8: with LP = 8 only).
template <bool VECS, int R8, int LP>
__device__ __forceinline__ void jacobi_round(double* J, int js, double* V, int vs, int N, int rows, int t,
                                             float& worst) {
  const int E = N + (N & 1), pair = threadIdx.x / LP, l8 = threadIdx.x % LP;
  int i = pair == 0 ? E - 1 : t + pair < E - 1 ? t + pair : t + pair - (E - 1);
  int j = pair == 0 ? t : t >= pair ? t - pair : t - pair + E - 1;
  if (i > j) {
    const int h = i;
    i = j;
    j = h;
  }
  const bool on = pair < E / 2 && j < N;
  if (!__any_sync(0xffffffffu, on)) return;
  double* wi = J + (on ? i : 0) * js;
  double* wj = J + (on ? j : 0) * js;
  double aa = 0.0, bb = 0.0, cc = 0.0;
  double xi[R8 > 0 ? R8 : 1], xj[R8 > 0 ? R8 : 1];  // R8 > 0: at most 8 R8 rows, kept in registers
  if constexpr (R8 > 0) {
#pragma unroll
    for (int q = 0; q < R8; ++q) {
      const int r = l8 + 8 * q;
      xi[q] = r < rows ? wi[r] : 0.0;
      xj[q] = r < rows ? wj[r] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < R8; ++q) {
      aa = fma(xi[q], xi[q], aa);
      bb = fma(xj[q], xj[q], bb);
      cc = fma(xi[q], xj[q], cc);
    }
  } else {
    for (int r = l8; r < rows; r += LP) {
      const double x = wi[r], y = wj[r];
      aa = fma(x, x, aa);
      bb = fma(y, y, bb);
      cc = fma(x, y, cc);
    }
  }
  aa = lane_sum<LP>(aa);
  bb = lane_sum<LP>(bb);
  cc = lane_sum<LP>(cc);
  double cs, sn, sj, cj;
  if (!on || !jacobi_angle(aa, bb, cc, worst, cs, sn, sj, cj)) return;
  if constexpr (R8 > 0) {
#pragma unroll
    for (int q = 0; q < R8; ++q) {
      const int r = l8 + 8 * q;
      if (r < rows) {
        wi[r] = cs * xi[q] - sj * xj[q];
        wj[r] = sn * xi[q] + cj * xj[q];
      }
    }
  } else {
    for (int r = l8; r < rows; r += LP) {
      const double x = wi[r], y = wj[r];
      wi[r] = cs * x - sj * y;
      wj[r] = sn * x + cj * y;
    }
  }
  if constexpr (VECS) {
    double* vi = V + i * vs;
    double* vj = V + j * vs;
    for (int r = l8; r < N; r += LP) {
      const double x = vi[r], y = vj[r];
      vi[r] = cs * x - sj * y;
      vj[r] = sn * x + cj * y;
    }
  }
}

// One pair by the whole CTA: few and very long columns.
template <bool VECS>
__device__ __forceinline__ void jacobi_wide(double* wi, double* wj, double* vi, double* vj, int N, int rows,
                                            double (*red)[LT / 32], float& worst) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double aa = 0.0, bb = 0.0, cc = 0.0;
  for (int r = threadIdx.x; r < rows; r += LT) {
    const double x = wi[r], y = wj[r];
    aa = fma(x, x, aa);
    bb = fma(y, y, bb);
    cc = fma(x, y, cc);
  }
  aa = lane_sum<32>(aa);
  bb = lane_sum<32>(bb);
  cc = lane_sum<32>(cc);
  if (lane == 0) {
    red[0][warp] = aa;
    red[1][warp] = bb;
    red[2][warp] = cc;
  }
  __syncthreads();
  aa = bb = cc = 0.0;
#pragma unroll
  for (int w = 0; w < LT / 32; ++w) {
    aa += red[0][w];
    bb += red[1][w];
    cc += red[2][w];
  }
  double cs, sn, sj, cj;
  if (jacobi_angle(aa, bb, cc, worst, cs, sn, sj, cj)) {  // the same in every thread
    for (int r = threadIdx.x; r < rows; r += LT) {
      const double x = wi[r], y = wj[r];
      wi[r] = cs * x - sj * y;
      wj[r] = sn * x + cj * y;
    }
    if (VECS && (int)threadIdx.x < N) {
      const double x = vi[threadIdx.x], y = vj[threadIdx.x];
      vi[threadIdx.x] = cs * x - sj * y;
      vj[threadIdx.x] = sn * x + cj * y;
    }
  }
  __syncthreads();  // the columns are final, and red has been read
}

template <bool VECS>
__device__ __forceinline__ void jacobi_sweeps(double* J, int js, double* V, int vs, int N, int rows, float* s_off,
                                              double (*red)[LT / 32]) {
  const int E = N + (N & 1), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int sweep = 0; sweep < 60 && N > 1; ++sweep) {
    float worst = 0.f;
    const bool by_cta = VECS && wide_pairs(N, rows);
    if (by_cta) {
      for (int i = 0; i < N; ++i)
        for (int j = i + 1; j < N; ++j)
          jacobi_wide<VECS>(J + i * js, J + j * js, V + i * vs, V + j * vs, N, rows, red, worst);
    }
    for (int t = 0; t < E - 1 && !by_cta; ++t) {
      if (rows <= 32) jacobi_round<VECS, 4, 8>(J, js, V, vs, N, rows, t, worst);
      else if (E / 2 > LT / 32) jacobi_round<VECS, 0, 8>(J, js, V, vs, N, rows, t, worst);
      else jacobi_round<VECS, 0, 32>(J, js, V, vs, N, rows, t, worst);  // a warp for each of few pairs
      __syncthreads();  // the next round pairs these columns differently
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if (lane == 0) s_off[warp] = worst;
    __syncthreads();
    float all = 0.f;
#pragma unroll
    for (int w = 0; w < LT / 32; ++w) all = fmaxf(all, s_off[w]);
    if (all < 1e-15f) break;  // the same value in every thread
    __syncthreads();          // s_off is rewritten after the next sweep
  }
}

// One problem per CTA. A (m x n), B (m x k) row-major in global memory; X
// (n x k), S (min(m, n)), rank, resid (k) and has_resid out. k = 0: singular
// values (and rank) only. QR: by way of the triangle. Each way has its own kernel: in one
// for both the direct way ran 2 to 14% longer (2000 of 5 x 2000 with 64 and rcond = 0 2587 us,
// 2123 now; 300 of 64 x 2 11.4, 10.4).
template <bool QR>
__global__ void __launch_bounds__(LT, 4)
k_lstsq(int m, int n, int k, const double* __restrict__ A, const double* __restrict__ B, double rcond, LsqLayout l,
        int left_only, double* __restrict__ X, double* __restrict__ S, int32_t* __restrict__ rank,
        double* __restrict__ resid, int32_t* __restrict__ has_resid) {
  extern __shared__ __align__(16) double lsq[];
  const bool wide = m < n;
  const int M = wide ? n : m, N = wide ? m : n;
  double* W = lsq;                 // the tall matrix, then (qr) the reflections below its diagonal
  double* buf = lsq + l.buf;       // (qr) right-hand sides, M rows each
  double* J = lsq + l.j;           // the columns the sweeps work on
  double* V = lsq + l.v;
  double* R = lsq + l.r;           // (qr) the triangle
  double* tau = lsq + l.tau;
  double* head = lsq + l.head;
  double* diag = lsq + l.diag;
  double* T1 = lsq + l.t1;         // N x k (row c at T1 + c * k)
  double* sig = lsq + l.sig;       // singular values, then the sorted reciprocals behind them
  double* sinv = sig + N;
  int* ord = reinterpret_cast<int*>(lsq + l.ord);
  __shared__ float s_off[LT / 32];
  __shared__ double red[3][LT / 32];
  __shared__ int s_rank, s_leave;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = LT / 32;
  const int64_t z = blockIdx.x;
  const double* Az = A + z * (int64_t)m * n;
  const double* Bz = B + z * (int64_t)m * k;
  if (left_only && rank[z] != kLsqLeft) return;
  int odd = 0;
  for (int idx = tid; idx < m * n; idx += LT) {  // coalesced reads of the row-major matrix
    const int r = idx / n, c = idx - r * n;
    const double x = Az[idx];
    W[wide ? r * l.ws + c : c * l.ws + r] = x;
    odd |= !(fabs(x) <= kLsqMostA);
  }
  // a NaN or an infinity must stay in its own column, where a reflection would
  // spread it, and a reflection's sums must stay within range: such a problem is
  // left to the launch that sweeps the matrix itself (here, at a reflection of tiny
  // length below, and at the right-hand sides)
  if (QR && tid == 0) s_leave = 0;
  if (QR && __syncthreads_or(odd)) {
    if (tid == 0) rank[z] = kLsqLeft;
    return;
  }
  const int js = l.js;
  const int Mj = QR ? N : M;  // rows of the Jacobi columns
  if constexpr (QR) {
    const int carried = wide ? 0 : l.nbuf;  // right-hand sides reflected along
    for (int idx = tid; idx < carried * M; idx += LT) {
      const int r = idx / carried, c = idx - r * carried;
      const double x = Bz[(int64_t)r * k + c];
      buf[c * l.ws + r] = x;
      odd |= !(fabs(x) <= kLsqMostB);
    }
    if (__syncthreads_or(odd)) {
      if (tid == 0) rank[z] = kLsqLeft;
      return;
    }
    // Warp 0 takes column q + 1 first and derives reflection q + 1 from it
    // while the other columns are still being updated: one barrier per column.
    for (int q = -1; q < N; ++q) {
      const double* w = W + (size_t)max(q, 0) * l.ws;
      const double h = q < 0 ? 0.0 : head[q], t = q < 0 ? 0.0 : tau[q];
      for (int c = q + 1 + warp; c < (q < 0 ? 1 : N + carried); c += NWARP) {
        double* x = c < N ? W + (size_t)c * l.ws : buf + (size_t)(c - N) * l.ws;
        if (q >= 0) reflect(w, h, t, x, q, M);
        if (c == q + 1 && c < N) {
          __syncwarp();
          double s2 = 0.0;
          for (int r = c + 1 + lane; r < M; r += 32) s2 = fma(x[r], x[r], s2);
          s2 = lane_sum<32>(s2);
          const double x0 = x[c];
          double beta = x0, tc = 0.0, hc = 1.0;
          const double n2 = fma(x0, x0, s2);
          if (n2 < 0x1p-960) {  // squares near or past the end of the range, or a column of zeros
            bool some = false;
            for (int r = c + lane; r < M; r += 32) some |= x[r] != 0.0;
            if (__any_sync(0xffffffffu, some)) s_leave = 1;
          } else if (s2 != 0.0) {  // else nothing is left to annihilate
            beta = -copysign(sqrt(n2), x0);
            hc = x0 - beta;
            // v near length 1 (an exact scaling): v^T x then stays within range with x
            const int e = exponent(n2) >> 1;
            if (e < -15 || e > 15) {
              const double sc = power2(-e);
              for (int r = c + 1 + lane; r < M; r += 32) x[r] *= sc;
              hc *= sc;
              s2 *= sc * sc;
            }
            tc = 2.0 / fma(hc, hc, s2);
          }
          if (lane == 0) {
            tau[c] = tc;
            head[c] = hc;
            diag[c] = beta;
          }
        }
      }
      __syncthreads();
    }
    if (s_leave) {
      if (tid == 0) rank[z] = kLsqLeft;
      return;
    }
    // the triangle out of W: through registers, J's place may be W's
    double tri[kLsqMaxN * kLsqMaxN / LT];
#pragma unroll
    for (int i = 0; i < kLsqMaxN * kLsqMaxN / LT; ++i) {
      const int idx = tid + i * LT, c = idx / N, r = idx - c * N;
      tri[i] = idx >= N * N || r > c ? 0.0 : (r == c ? diag[c] : W[c * l.ws + r]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kLsqMaxN * kLsqMaxN / LT; ++i) {
      const int idx = tid + i * LT, c = idx / N, r = idx - c * N;
      if (idx < N * N) J[c * js + r] = R[c * js + r] = tri[i];
    }
  }
  for (int idx = tid; idx < N * N; idx += LT) {
    const int c = idx / N, r = idx - c * N;
    V[c * l.vs + r] = c == r ? 1.0 : 0.0;
  }
  __syncthreads();

  // A triangle of full rank gives x by substitution: V is only accumulated (in
  // sweeps of their own) for the rank-deficient ones.
  bool vecs = !QR;
  jacobi_sweeps<!QR>(J, js, V, l.vs, N, Mj, s_off, red);
again:
  // singular values: the column norms; the columns normalised in place
  for (int c = warp; c < N; c += NWARP) {
    double s2 = 0.0;
    for (int r = lane; r < Mj; r += 32) s2 = fma(J[c * js + r], J[c * js + r], s2);
    const double s = sqrt(lane_sum<32>(s2));
    if (lane == 0) sig[c] = s;
    for (int r = lane; r < Mj; r += 32) J[c * js + r] = s > 0.0 ? J[c * js + r] / s : 0.0;
  }
  if (tid < N) ord[tid] = tid;
  if (tid == 0) s_rank = 0;
  __syncthreads();
  const double own = tid < N ? sig[tid] : 0.0;
  const double top = rcond < 0 ? 2.220446049250313e-16 * (m > n ? m : n) : rcond;  // times s_max: the tolerance
  if (!__syncthreads_or(isnan(own))) {
    // descending order, equal values by column: a value's place is the number of values ahead of it
    if (tid < N) {
      int place = 0;
      double smax = 0.0;
      for (int c = 0; c < N; ++c) {
        const double o = sig[c];
        place += o > own || (o == own && c < tid);
        smax = fmax(smax, o);
      }
      ord[place] = tid;
      S[z * N + place] = own;
      sinv[place] = own > top * smax ? 1.0 / own : 0.0;
      if (own > top * smax) atomicAdd(&s_rank, 1);
    }
  } else if (tid == 0) {  // no order with a NaN: the stable insertion sort's result, as the reference has it
    for (int a = 1; a < N; ++a) {
      const int o = ord[a];
      int b = a - 1;
      while (b >= 0 && sig[ord[b]] < sig[o]) {
        ord[b + 1] = ord[b];
        --b;
      }
      ord[b + 1] = o;
    }
    const double tol = top * sig[ord[0]];
    for (int c = 0; c < N; ++c) {
      const double v = sig[ord[c]];
      S[z * N + c] = v;
      sinv[c] = v > tol ? 1.0 / v : 0.0;
      s_rank += v > tol;
    }
  }
  __syncthreads();
  if (tid == 0) rank[z] = s_rank;
  if (k == 0) return;
  const bool full = QR && !vecs && s_rank == N;
  if (QR && !vecs && !full) {
    __syncthreads();  // every thread has read s_rank
    for (int idx = tid; idx < N * N; idx += LT) {
      const int c = idx / N, r = idx - c * N;
      J[c * js + r] = R[c * js + r];
    }
    __syncthreads();
    jacobi_sweeps<true>(J, js, V, l.vs, N, Mj, s_off, red);
    vecs = true;
    goto again;
  }

  // T1 = diag(1/s) (left vectors)^T b. Tall: the columns of J against b, or
  // (qr) against the first N rows of Q^T b; wide: the columns of V against b.
  double* Xz = X + z * (int64_t)n * k;
  const bool form = m > n && s_rank == n;
  if (tid == 0) has_resid[z] = form ? 1 : 0;
  const int step = QR ? l.nbuf : k;  // right-hand sides at a time
  for (int j0 = 0; j0 < k; j0 += step) {
    const int jn = min(step, k - j0);
    if (QR && !wide && j0 > 0) {  // the first group went through the reflections with the matrix
      if (warp < jn) {
        double* x = buf + (size_t)warp * l.ws;
        for (int r = lane; r < M; r += 32) {
          x[r] = Bz[(int64_t)r * k + j0 + warp];
          odd |= !(fabs(x[r]) <= kLsqMostB);
        }
        __syncwarp();
        for (int q = 0; q < N; ++q) {
          reflect(W + (size_t)q * l.ws, head[q], tau[q], x, q, M);
          __syncwarp();
        }
      }
      if (__syncthreads_or(odd)) {
        if (tid == 0) rank[z] = kLsqLeft;
        return;
      }
    }
    if (full) {
      // R x = (Q^T b)'s first N rows (tall) or R^T y = b, x = Q y (wide): a warp
      // per right-hand side, lane r holds rows r and r + 32
      for (int j = warp; j < jn; j += NWARP) {
        const int ra = lane, rb = lane + 32;
        double* xb = buf + (size_t)j * l.ws;
        double va = ra < N ? (wide ? Bz[(int64_t)ra * k + j0 + j] : xb[ra]) : 0.0;
        double vb = rb < N ? (wide ? Bz[(int64_t)rb * k + j0 + j] : xb[rb]) : 0.0;
        const double da = ra < N ? 1.0 / R[ra * js + ra] : 0.0, db = rb < N ? 1.0 / R[rb * js + rb] : 0.0;
        for (int s = 0; s < N; ++s) {
          const int q = wide ? s : N - 1 - s;
          const double mine = q < 32 ? va * da : vb * db;
          const double xq = __shfl_sync(0xffffffffu, mine, q & 31);
          const double ca = wide ? R[min(ra, N - 1) * js + q] : R[q * js + min(ra, N - 1)];
          const double cb = wide ? R[min(rb, N - 1) * js + q] : R[q * js + min(rb, N - 1)];
          if (ra == q) va = xq;
          else if (wide ? ra > q : ra < q) va = fma(-ca, xq, va);
          if (rb == q) vb = xq;
          else if (wide ? rb > q : rb < q) vb = fma(-cb, xq, vb);
        }
        if (wide) {
          if (ra < N) xb[ra] = va;
          if (rb < N) xb[rb] = vb;
        } else {
          if (ra < N) Xz[(int64_t)ra * k + j0 + j] = va;
          if (rb < N) Xz[(int64_t)rb * k + j0 + j] = vb;
        }
      }
    }
    for (int q = warp; !full && q < N * jn; q += NWARP) {
      const int c = q / jn, j = q - c * jn;
      const double* uc = wide ? V + (size_t)ord[c] * l.vs : J + (size_t)ord[c] * js;
      const bool own = QR && !wide;
      const int rows = QR || wide ? N : M;
      double t = 0.0;
      for (int p = lane; p < rows; p += 32)
        t = fma(uc[p], own ? buf[(size_t)j * l.ws + p] : Bz[(int64_t)p * k + j0 + j], t);
      t = lane_sum<32>(t);
      if (lane == 0) T1[(size_t)c * k + j0 + j] = sinv[c] * t;
    }
    __syncthreads();
    // x = (right vectors) T1: V's columns (tall), J's (wide), or (wide, qr)
    // Q applied to J's
    const int xr = QR && wide ? N : n, stride = wide ? js : l.vs;
    for (int q = tid; !full && q < xr * jn; q += LT) {
      const int i = q / jn, j = q - i * jn;
      const double* v = (wide ? J : V) + i;
      const double* tc = T1 + j0 + j;
      double t = 0.0;
#pragma unroll 4
      for (int c = 0; c < N; ++c) t = fma(v[ord[c] * stride], tc[c * k], t);
      if (QR && wide) buf[(size_t)j * l.ws + i] = t;
      else Xz[(int64_t)i * k + j0 + j] = t;
    }
    if (QR && wide) {
      __syncthreads();
      if (warp < jn) {
        double* x = buf + (size_t)warp * l.ws;
        for (int r = N + lane; r < M; r += 32) x[r] = 0.0;
        __syncwarp();
        for (int q = N - 1; q >= 0; --q) {
          reflect(W + (size_t)q * l.ws, head[q], tau[q], x, q, M);
          __syncwarp();
        }
        for (int r = lane; r < M; r += 32) Xz[(int64_t)r * k + j0 + warp] = x[r];
      }
    }
    __syncthreads();  // buf is refilled by the next group; x is complete for the residuals
    if (form) {
      // residuals: (qr) the part of Q^T b that the columns of A cannot reach, else the
      // rows of b - A x; one warp per column, or the whole CTA where few columns are long
      const bool all = m >= 256 && (jn < NWARP || !QR);
      for (int j = all ? 0 : warp; j < jn; j += all ? 1 : NWARP) {
        double acc = 0.0;
        for (int i = (QR ? n : 0) + (all ? tid : lane); i < m; i += all ? LT : 32) {
          double d;
          if constexpr (QR) {
            d = buf[(size_t)j * l.ws + i];
          } else {
            double ax = 0.0;
            for (int p = 0; p < n; ++p) ax = fma(Az[(int64_t)i * n + p], Xz[(int64_t)p * k + j0 + j], ax);
            d = Bz[(int64_t)i * k + j0 + j] - ax;
          }
          acc = fma(d, d, acc);
        }
        acc = lane_sum<32>(acc);
        if (!all) {
          if (lane == 0) resid[z * k + j0 + j] = acc;
          continue;
        }
        if (lane == 0) red[j & 1][warp] = acc;
        __syncthreads();
        if (tid == 0) {
          double sum = 0.0;
#pragma unroll
          for (int w = 0; w < NWARP; ++w) sum += red[j & 1][w];
          resid[z * k + j0 + j] = sum;
        }
      }
      __syncthreads();
    }
  }
}

int check(int64_t count, int32_t m, int32_t n, int32_t k) {
  if (count < 0 || m < 0 || n < 0 || k < 0) {
    set_error("negative count, shape or nrhs");
    return NPPB_E_ARG;
  }
  if (count > INT32_MAX) {
    set_error("batch count above 2^31-1");
    return NPPB_E_RANGE;
  }
  const int M = m > n ? m : n, N = m < n ? m : n;
  if (N > kLsqMaxN || k > kLsqMaxK || (int64_t)M * N > (int64_t)kLsqMaxSmem / 8 || lsq_base(M, N, k) > kLsqMaxSmem) {
    set_error("least squares on the device: min(m, n) <= 64, nrhs <= 64 and the tall matrix, V and U^T b "
              "within 220 KiB of shared memory (about m * n + min(m, n)^2 <= 26000)");
    return NPPB_DECLINED;
  }
  return NPPB_OK;
}

int lstsq_device(int64_t count, int32_t m, int32_t n, int32_t k, const double* dA, const double* dB, double rcond,
                 double* dX, double* dS, int32_t* drank, double* dres, int32_t* dhas, cudaStream_t st) {
  const LsqLayout l = lsq_plan(m, n, k, rcond);
  const size_t smem = sizeof(double) * (size_t)l.doubles;
  // one value for every shape: threads with different shapes do not disturb one another
  NPPB_CUDA(cudaFuncSetAttribute(k_lstsq<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLsqMaxSmem + 4096),
            "attribute");
  if (l.qr)
    NPPB_CUDA(cudaFuncSetAttribute(k_lstsq<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLsqMaxSmem + 4096),
              "attribute");
  const auto kernel = l.qr ? k_lstsq<true> : k_lstsq<false>;
  kernel<<<(unsigned)count, LT, smem, st>>>(m, n, k, dA, dB, rcond, l, 0, dX, dS, drank, dres, dhas);
  NPPB_CUDA(cudaGetLastError(), "least squares");
  if (l.qr) {  // problems with a NaN or an infinity; the others' CTAs return at once
    const LsqLayout d = lsq_layout(m, n, k, -1);
    k_lstsq<false><<<(unsigned)count, LT, sizeof(double) * (size_t)d.doubles, st>>>(m, n, k, dA, dB, rcond, d, 1, dX, dS,
                                                                            drank, dres, dhas);
    NPPB_CUDA(cudaGetLastError(), "least squares");
  }
  return NPPB_OK;
}

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

}  // namespace

extern "C" {

int nppb_d_lstsq_batched(int64_t count, int32_t m, int32_t n, int32_t k, const double* dA, const double* dB,
                         double rcond, double* dX, double* dS, int32_t* drank, double* dres, int32_t* dhas,
                         void* stream) {
  return guarded([&]() -> int {
    const int rc = check(count, m, n, k);
    if (rc != NPPB_OK) return rc;
    if (!count || !m || !n) return NPPB_OK;
    if (!dA || !dS || !drank || (k && (!dB || !dX || !dres || !dhas))) {
      set_error("lstsq needs A, S, rank and, with right-hand sides, B, X, residuals and their flags");
      return NPPB_E_ARG;
    }
    if (!device()) return NPPB_E_NODEV;
    return lstsq_device(count, m, n, k, dA, dB, rcond, dX, dS, drank, dres, dhas, static_cast<cudaStream_t>(stream));
  });
}

int nppb_lstsq_batched(int64_t count, int32_t m, int32_t n, int32_t k, const double* A, const double* B,
                       double rcond, double* X, double* S, int32_t* rank, double* resid, int32_t* has_resid) {
  return guarded([&]() -> int {
    const int rc = check(count, m, n, k);
    if (rc != NPPB_OK) return rc;
    if (!count || !m || !n) return NPPB_OK;
    if (!A || !S || !rank || (k && (!B || !X || !resid || !has_resid))) {
      set_error("lstsq needs A, S, rank and, with right-hand sides, B, X, residuals and their flags");
      return NPPB_E_ARG;
    }
    if (!device()) return NPPB_E_NODEV;
    cudaStream_t st = thread_stream();
    const size_t c = (size_t)count, kk = (size_t)(m < n ? m : n);
    DevMem dA, dB, dX, dS, dR, dres, dh;
    NPPB_CUDA(dA.alloc(sizeof(double) * c * m * n, st), "allocation");
    NPPB_CUDA(dS.alloc(sizeof(double) * c * kk, st), "allocation");
    NPPB_CUDA(dR.alloc(sizeof(int32_t) * c, st), "allocation");
    NPPB_CUDA(cudaMemcpyAsync(dA.as<double>(), A, sizeof(double) * c * m * n, cudaMemcpyHostToDevice, st), "copy");
    if (k) {
      NPPB_CUDA(dB.alloc(sizeof(double) * c * m * k, st), "allocation");
      NPPB_CUDA(dX.alloc(sizeof(double) * c * n * k, st), "allocation");
      NPPB_CUDA(dres.alloc(sizeof(double) * c * k, st), "allocation");
      NPPB_CUDA(dh.alloc(sizeof(int32_t) * c, st), "allocation");
      NPPB_CUDA(cudaMemcpyAsync(dB.as<double>(), B, sizeof(double) * c * m * k, cudaMemcpyHostToDevice, st), "copy");
    }
    const int r = lstsq_device(count, m, n, k, dA.as<double>(), k ? dB.as<double>() : nullptr, rcond,
                               k ? dX.as<double>() : nullptr, dS.as<double>(), dR.as<int32_t>(),
                               k ? dres.as<double>() : nullptr, k ? dh.as<int32_t>() : nullptr, st);
    if (r != NPPB_OK) return r;
    NPPB_CUDA(cudaMemcpyAsync(S, dS.as<double>(), sizeof(double) * c * kk, cudaMemcpyDeviceToHost, st), "copy");
    NPPB_CUDA(cudaMemcpyAsync(rank, dR.as<int32_t>(), sizeof(int32_t) * c, cudaMemcpyDeviceToHost, st), "copy");
    if (k) {
      NPPB_CUDA(cudaMemcpyAsync(X, dX.as<double>(), sizeof(double) * c * n * k, cudaMemcpyDeviceToHost, st), "copy");
      NPPB_CUDA(cudaMemcpyAsync(resid, dres.as<double>(), sizeof(double) * c * k, cudaMemcpyDeviceToHost, st),
                "copy");
      NPPB_CUDA(cudaMemcpyAsync(has_resid, dh.as<int32_t>(), sizeof(int32_t) * c, cudaMemcpyDeviceToHost, st),
                "copy");
    }
    NPPB_CUDA(cudaStreamSynchronize(st), "synchronize");
    NPPB_CUDA(cudaGetLastError(), "kernel");
    return NPPB_OK;
  });
}

}  // extern "C"
