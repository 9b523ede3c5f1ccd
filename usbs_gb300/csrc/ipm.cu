// k x k bundle subproblems and small dense steps of the USBS iteration, FP64,
// one CTA per instance.
//
//  * ipm_kernel  mode 0: solve_quad_subprob_ipm  (solver/usbs.py:25-192)
//                mode 1: compute_lb_spec_est_ipm (solver/usbs.py:195-356)
//    Primal-dual interior point on (S, eta, T, zeta, omega) in svec
//    coordinates: Newton system (s x s) assembled from the symmetric Kronecker
//    product T (x) S^-1 and solved by LU; line search over the step grid
//    0.9^j, j < ipm_max_iters, keeping the largest step at which S + a dS and
//    T + a dT stay positive definite (32 LDL^T tests at a time), exactly the reference's "smallest eigenvalue > 0" rule.
//  * eigS_kernel  eigh(S) of the bundle matrix and everything the outer
//    iteration derives from it (solver/usbs.py:409-412, 568-585, 627-644).
//  * cholqr_kernel  R^-1 of one (shifted) Cholesky-QR pass for the new bundle
//    basis (replaces the Householder QR of solver/usbs.py:641-642).
#include "common.cuh"
#include "recip.cuh"
#include "dense.cuh"
#include "internal.h"
#include "solver.h"

namespace usbs {

constexpr double RSQ2 = 0.70710678118654752440;

__device__ __forceinline__ double nanmin2(double a, double b) {
  if (isnan(a) || isnan(b)) return __longlong_as_double(0x7ff8000000000000ll);
  return a < b ? a : b;
}

struct IpmShared {
  int bi[IPM_MAXS], ci[IPM_MAXS];
  double q12[IPM_MAXS], h1[IPM_MAXS], sI[IPM_MAXS], sS[IPM_MAXS], sT[IPM_MAXS];
  double F1[IPM_MAXS], ord[IPM_MAXS], dsT[IPM_MAXS], sSi[IPM_MAXS];
  double S[IPM_MAXK * IPM_MAXK], T[IPM_MAXK * IPM_MAXK], Si[IPM_MAXK * IPM_MAXK];
  double dS[IPM_MAXK * IPM_MAXK], dT[IPM_MAXK * IPM_MAXK];
  double dinv[IPM_MAXS];
  double u2[IPM_MAXS], w2[IPM_MAXS];   // per-column terms of the rank-2 correction
  int cord[IPM_MAXS];                  // svec indices, off-diagonal ones first
  double part3[3 * IPM_MAXS];          // partial sums of cta_matvec3
};

// sum_a x[a] y[a], computed redundantly by every warp (identical in all threads)
__device__ __forceinline__ double dot_s(const double* x, const double* y, int s) {
  double v = 0.0;
  for (int a = threadIdx.x & 31; a < s; a += 32) v += x[a] * y[a];
  return warp_sum(v);
}

__device__ __forceinline__ double svec_of(const double* M, int k, int b, int c) {
  return (b == c) ? M[b * k + b] : (RSQ2 * M[c * k + b] + RSQ2 * M[b * k + c]);
}

__device__ __forceinline__ void svec_inv_to(const double* v, int k, int s, const int* bi,
                                            const int* ci, double* M) {
  for (int a = threadIdx.x; a < s; a += blockDim.x) {
    const int b = bi[a], c = ci[a];
    if (b == c) M[b * k + b] = v[a];
    else { M[b * k + c] = RSQ2 * v[a]; M[c * k + b] = RSQ2 * v[a]; }
  }
}

// 0.5 * [U (T (x) X + X (x) T) U^T]_{a, a2}, U the svec isometry.
// The same entry with each distinct product summed once: of the 2 na nb
// products of the definition every one appears twice (T_ii2 X_jj2 for the
// ordering (i, j) equals X_jj2 T_ii2 for (j, i)), and 0.5 * 2 is exact, so
//   entry = w * sum over the orderings (i2, j2) of a2 of T_b,i2 X_c,j2 + X_b,i2 T_c,j2
// (one ordering when a is diagonal), w = 1/2 when a and a2 are both diagonal or
// both off-diagonal, 1/sqrt(2) otherwise.
__device__ __forceinline__ double symkron_sum(const double* T, const double* X, int k, int b,
                                              int c, int b2, int c2) {
  double S = T[b * k + b2] * X[c * k + c2];
  S = fma(X[b * k + b2], T[c * k + c2], S);
  if (b2 != c2 && b != c) {
    S = fma(T[b * k + c2], X[c * k + b2], S);
    S = fma(X[b * k + c2], T[c * k + b2], S);
  }
  return (((b == c) == (b2 == c2)) ? 0.5 : RSQ2) * S;
}

// 32 positive-definiteness tests of M + step dM (k x k, lower triangle) by LDL^T
// without pivoting, whole CTA, eight lanes each: test t < 16 is of (S, dS), the
// others of (T, dT).  PD iff every pivot is positive (equivalent to Cholesky
// succeeding, i.e. to the smallest eigenvalue being > 0, up to round-off at the
// boundary).  One reciprocal per column (on the integer pipes), no square roots.
// Right-looking, the trailing triangle's entries dealt to the eight lanes: an
// entry sees a_ij + s da_ij, then - l_ip u_jp for p = 0, 1, ..., u_jp = l_jp d_p,
// one FMA each.  The FP64 unit takes a warp instruction every 19 cycles SM-wide
// but one warp only every 60: with one lane per test on one warp a round of 32
// tests took 26k cycles (k = 11).
// ws: 32 (s + IPM_MAXK) doubles.  Returns the mask of the tests that passed.
__device__ unsigned pd_tests(const double* S, const double* dS, const double* T, const double* dT,
                             int k, int s, const int* bi, const int* ci, bool active, double step,
                             double* ws, unsigned* mask) {
  constexpr int G = 8, EU = (IPM_MAXS + G - 1) / G;
  const int tid = threadIdx.x, lane = tid & 31, g = lane & (G - 1);
  const int test = tid / G;
  double* M = ws + test * (s + IPM_MAXK);
  double* L = M + s;
  const double* A = (test < 16) ? S : T;
  const double* dA = (test < 16) ? dS : dT;
  if (tid == 0) *mask = 0u;
  int bc[EU];                          // packed coordinates of this lane's triangle entries
#pragma unroll
  for (int u = 0; u < EU; ++u) {
    const int t = g + G * u;
    bc[u] = (t < s) ? (bi[t] << 8) | ci[t] : 0;
  }
  bool pd = active;
  if (active) {
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int t = g + G * u;
      if (t < s) {
        const int e = (bc[u] >> 8) * k + (bc[u] & 255);
        M[t] = A[e] + step * dA[e];
      }
    }
  }
  __syncthreads();
  for (int p = 0; p < k; ++p) {
    const double d = pd ? M[p * (p + 1) / 2 + p] : 1.0;
    if (!(d > 0.0)) pd = false;
    if (__any_sync(0xffffffffu, pd)) {
      const double inv = recip_exact(d);
      for (int i = p + 1 + g; i < k; i += G)
        if (pd) L[i] = M[i * (i + 1) / 2 + p] * inv;
      __syncwarp();
      const int m = (k - 1 - p) * (k - p) / 2;
#pragma unroll
      for (int u = 0; u < EU; ++u) {
        if (G * u < m) {
          const int t = g + G * u;
          if (t < m && pd) {
            const int i = p + 1 + (bc[u] >> 8), j = p + 1 + (bc[u] & 255);
            double* v = M + i * (i + 1) / 2 + j;
            *v -= L[i] * M[j * (j + 1) / 2 + p];
          }
        }
      }
    }
    __syncwarp();
  }
  if (pd && g == 0) atomicOr(mask, 1u << test);
  __syncthreads();
  return *mask;
}

struct IpmScal {
  double eta, zeta, omega, mu, step, trS, k1, k2, den, ze, F2, d_eta, d_omega, d_zeta, st, cS,
      cT, q22, h2, t1, t2, t3, t4, rden, mow, moe, lbc;
  int cont, it;
};

// sum_a x[a] y[a] by one warp (lane 0 holds the result)
__device__ __forceinline__ double wdot(const double* x, const double* y, int s) {
  double v = 0.0;
  for (int a = threadIdx.x & 31; a < s; a += 32) v += x[a] * y[a];
  return warp_sum(v);
}

// |x| of a double as an integer key: for finite values the ordering of the keys
// is the ordering of |x|, so pivot comparisons stay off the FP64 pipe.
__device__ __forceinline__ unsigned long long abs_key(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// Inverse of an n x n matrix (n <= IPM_MAXK, row-major, lda = n) by Gauss-Jordan
// elimination with partial pivoting on [A | I], whole CTA.  ws holds two n x 2n
// augmented matrices: a pivot step reads one and writes the other, so it takes
// one barrier, and each thread forms one entry of the new matrix, the pivot row's
// scaled entry included.  Every warp picks the pivot itself (largest |a| by
// integer keys, ties to the smaller row) and forms its reciprocal on the integer
// pipes.  Per element the arithmetic is that of the row-by-row algorithm (rows
// j and piv exchanged, pivot row scaled by 1/a_jj, a_ic - a_ij * row_c).  Returns
// false if a pivot is zero or infinite.  (With the exchange, the column copy, the scaling
// and the update as four steps between barriers it took 28k cycles at n = 11.)
__device__ bool cta_inverse(const double* A, int n, double* Ainv, double* ws) {
  const int tid = threadIdx.x, lane = tid & 31, ld = 2 * n;
  double* cur = ws;
  double* nxt = ws + n * ld;
  for (int e = tid; e < n * ld; e += IPM_BLOCK) {
    const int i = e / ld, c = e - i * ld;
    cur[e] = (c < n) ? A[i * n + c] : ((c - n == i) ? 1.0 : 0.0);
  }
  bool ok = true;
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const bool valid = lane >= j && lane < n;
    const double a = valid ? cur[lane * ld + j] : 0.0;
    const unsigned long long key = abs_key(a);
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, valid ? hi : 0u);
    const bool th = valid && hi == mhi;
    const unsigned mlo = __reduce_max_sync(0xffffffffu, th ? lo : 0u);
    const int piv = (int)__reduce_min_sync(0xffffffffu, (th && lo == mlo) ? (unsigned)lane : (unsigned)j + 32u) & 31;
    const double pv = __shfl_sync(0xffffffffu, a, piv);
    const bool zero = abs_key(pv) == 0ull;
    const double inv = zero ? 0.0 : recip_exact(pv);
    if (abs_key(inv) == 0ull) ok = false;        // a zero or an infinite pivot
    for (int e = tid; e < n * ld; e += IPM_BLOCK) {
      const int i = e / ld, c = e - i * ld;
      const int src = (i == j) ? piv : (i == piv) ? j : i;
      const double rowc = cur[piv * ld + c] * inv;
      nxt[e] = (i == j) ? rowc : cur[src * ld + c] - cur[src * ld + j] * rowc;
    }
    __syncthreads();
    double* t = cur; cur = nxt; nxt = t;
  }
  for (int e = tid; e < n * n; e += IPM_BLOCK) Ainv[e] = cur[(e / n) * ld + n + e % n];
  __syncthreads();
  return ok;
}

// y[a] = sum_b M[a, b] x[b] (s x s, row-major) as three partial chains per row,
// combined in a fixed order (a 66-long dependent FP64 chain costs ~4k cycles)
__device__ void cta_matvec3(const double* M, const double* x, int s, double* part, double* y) {
  const int tid = threadIdx.x;
  if (tid < 3 * s) {
    const int a = tid / 3, q = tid - 3 * (tid / 3);
    const int b0 = (q * s) / 3, b1 = ((q + 1) * s) / 3;
    double v = 0.0;
    for (int b = b0; b < b1; ++b) v += M[a * s + b] * x[b];
    part[tid] = v;
  }
  __syncthreads();
  for (int a = tid; a < s; a += blockDim.x) y[a] = (part[3 * a] + part[3 * a + 1]) + part[3 * a + 2];
  __syncthreads();
}

// LU with partial pivoting and solve, whole CTA (G&VL Alg. 3.4.1, right-looking
// with a one-column look-ahead).  A is stored column-major (A[c * lda + i] is
// row i, column c).  Every element sees the arithmetic of the textbook algorithm
// (a_ic - l_i a_jc, l_i = a_ij * (1/a_jj)).  Partial pivoting is needed: in
// the bundle subproblems' Newton systems about two thirds of the
// factorisations exchange rows somewhere.
// On GB300 the SM's FP64 unit takes one warp instruction every 19 cycles, a single
// warp one every 60, and the trailing update is bound by it while more than about
// 40 positions are left; below, a column's pivot chain (one FMA, the argmax, the
// reciprocal, the multipliers) is a sequence of latencies that bounds the
// factorisation.  So while the other warps eliminate b and
// apply the rank-1 update of column j to columns j+2.., warp 0 alone takes
// column j+1 through registers: lane l keeps positions n-1-l, n-33-l, n-65-l (a
// position's row, its value in the current column and its multiplier), and only
// the register blocks that still hold positions take part.  Rows are not moved:
// the exchange swaps two rows' positions, in registers and in the list of rows
// by position that warp 0 hands over with the multipliers (double-buffered, so
// one barrier per column).  The pivot is the largest |a| by integer keys, ties to
// the smaller position as in LAPACK.  The column itself is not written back (L is
// not stored, and U needs only the rows above).
// The loops are specialised by the number of register blocks: straight-line code
// for three of them in one loop made a column of the smallest systems 2.0k cycles,
// fetching instructions; 1.2k as it is.  Order 66: 126k cycles (153k with rows
// exchanged in memory between barriers), order 15 18k (31k).  Four trailing
// warps instead of seven, or several elements in flight per thread, are slower
// (order 66: 160-350k).
constexpr int LU_RPL = (IPM_MAXS + 31) / 32;   // register blocks of 32 positions
struct LuShared {
  double lb[2][IPM_MAXS];    // multipliers by position, of even and odd columns
  int rows[2][IPM_MAXS];     // row by position, after the exchange of even and odd columns
  int prow[IPM_MAXS];        // pivot rows
};
// warp 0's registers
struct LuRegs {
  double v[LU_RPL], l[LU_RPL];
  int row[LU_RPL], pr;
};

// warp 0: R.v holds column j at positions j.. (in NQ register blocks); its pivot,
// reciprocal, multipliers and the exchange of positions
template <int NQ>
__device__ __forceinline__ void lu_pick(LuRegs& R, LuShared& S, int j, int n, double* dinv,
                                        int* ok_out) {
  const int lane = threadIdx.x & 31, p0 = n - 1 - lane;
  // lane-local candidate: largest |a| key, smallest position among equal keys
  unsigned long long best = abs_key(R.v[0]);
  int bp = p0;
#pragma unroll
  for (int q = 1; q < NQ; ++q) {
    const unsigned long long k = abs_key(R.v[q]);
    if (p0 - 32 * q >= j && k >= best) { best = k; bp = p0 - 32 * q; }
  }
  // warp argmax by reduction instructions: high word, then low word among
  // the lanes holding the top high word, then the smallest position among ties
  const bool cand = bp >= j;
  const unsigned hi = (unsigned)(best >> 32), lo = (unsigned)best;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, cand ? hi : 0u);
  const bool th = cand && hi == mhi;
  const unsigned mlo = __reduce_max_sync(0xffffffffu, th ? lo : 0u);
  const int bi = (int)__reduce_min_sync(0xffffffffu, (th && lo == mlo) ? (unsigned)bp : 0x7fffffffu);
  const int bo = n - 1 - bi, jo = n - 1 - j;      // their owner lanes and blocks
  double bsel = R.v[0], jsel = R.v[NQ - 1];       // position j is in the last block
  int brow = R.row[0], jrow = R.row[NQ - 1];
#pragma unroll
  for (int q = 1; q < NQ; ++q)
    if (q == (bo >> 5)) { bsel = R.v[q]; brow = R.row[q]; }
  const double bv = __shfl_sync(0xffffffffu, bsel, bo & 31);
  R.pr = __shfl_sync(0xffffffffu, brow, bo & 31);
  jsel = __shfl_sync(0xffffffffu, jsel, jo & 31);
  jrow = __shfl_sync(0xffffffffu, jrow, jo & 31);
  const bool zero = (abs_key(bv) == 0ull);
  const double inv = recip_exact(zero ? 1.0 : bv);
  double* lj = S.lb[j & 1];
  int* rj = S.rows[j & 1];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int p = p0 - 32 * q;
    if (p == bi) { R.v[q] = jsel; R.row[q] = jrow; }
    R.l[q] = R.v[q] * inv;
    if (p > j) {
      lj[p] = R.l[q];
      rj[p] = R.row[q];
    }
  }
  if (lane == 0) {
    S.prow[j] = R.pr;
    dinv[j] = inv;
    if (zero) *ok_out = 0;
  }
}

// columns j = j0.. while at most 32 NQ positions (and more than 32 (NQ - 1)) lie
// behind them; returns the first column not done
template <int NQ>
__device__ __forceinline__ int lu_columns(double* A, int lda, double* b, int n, double* dinv,
                                          LuShared& S, LuRegs& R, int j0, int* ok_out) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int j = j0;
  for (; j < n - 1 - 32 * (NQ - 1); ++j) {
    if (wid == 0) {
      // column j+1 at positions j+1.. (all loads first), then its pivot
      const double* col = A + (j + 1) * lda;
      const double u = col[R.pr];
      double a[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) a[q] = (n - 1 - lane - 32 * q > j) ? col[R.row[q]] : 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) R.v[q] = a[q] - R.l[q] * u;
      lu_pick<NQ>(R, S, j + 1, n, dinv, ok_out);
    } else {
      const int pj = S.prow[j];
      const double* lj = S.lb[j & 1];
      const int* rj = S.rows[j & 1];
      double l[NQ];
      int r[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int p = n - 1 - lane - 32 * q;
        l[q] = (p > j) ? lj[p] : 0.0;
        r[q] = (p > j) ? rj[p] : -1;
      }
      // columns j+2.. dealt to warps 1..7, and b (forward elimination of the
      // right-hand side) as one more column to the warp with the fewest
      for (int c = j + 1 + wid; c <= n; c += IPM_BLOCK / 32 - 1) {
        double* col = (c < n) ? A + c * lda : b;
        const double u = col[pj];
        double x[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) x[q] = (r[q] >= 0) ? col[r[q]] : 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q)
          if (r[q] >= 0) col[r[q]] = x[q] - l[q] * u;
      }
    }
    __syncthreads();
  }
  return j;
}

// U x = b, columns j = j0 down to 32 (NQ - 1), by one warp: lane l keeps b at
// positions l, l + 32, l + 64 in br; x_j = b_j * (1 / u_jj) with the pivot
// reciprocal of the factorisation (as the multipliers), then every lane updates
// its positions above j, the block that holds position j - 1 first.
template <int NQ>
__device__ __forceinline__ int lu_back(const double* A, int lda, const double* dinv, LuRegs& R,
                                       int j0) {
  const int lane = threadIdx.x & 31;
  int j = j0;
  for (; j >= 32 * (NQ - 1); --j) {
    const double* colj = A + j * lda;
    double u[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) u[q] = (lane + 32 * q < j) ? colj[R.row[q]] : 0.0;
    const double bj = __shfl_sync(0xffffffffu, R.v[NQ - 1], j & 31) * dinv[j];
#pragma unroll
    for (int q = NQ - 1; q >= 0; --q) {
      const int i = lane + 32 * q;
      if (i == j) R.v[q] = bj;
      else if (i < j) R.v[q] -= u[q] * bj;
    }
  }
  return j;
}

__device__ void ipm_lu_solve(double* A, int lda, double* b, int n, double* dinv, int* ok_out) {
  static_assert(LU_RPL == 3, "register blocks");
  __shared__ LuShared S;
  const int tid = threadIdx.x, lane = tid & 31;
  LuRegs R;
  if (tid == 0) *ok_out = 1;
  __syncthreads();
  if (tid < 32) {
#pragma unroll
    for (int q = 0; q < LU_RPL; ++q) {
      R.row[q] = n - 1 - lane - 32 * q;
      R.v[q] = (R.row[q] >= 0) ? A[R.row[q]] : 0.0;
    }
    if (n > 64) lu_pick<3>(R, S, 0, n, dinv, ok_out);
    else if (n > 32) lu_pick<2>(R, S, 0, n, dinv, ok_out);
    else lu_pick<1>(R, S, 0, n, dinv, ok_out);
  }
  __syncthreads();
  int j = lu_columns<3>(A, lda, b, n, dinv, S, R, 0, ok_out);
  j = lu_columns<2>(A, lda, b, n, dinv, S, R, j, ok_out);
  j = lu_columns<1>(A, lda, b, n, dinv, S, R, j, ok_out);
  if (tid < 32) {
#pragma unroll
    for (int q = 0; q < LU_RPL; ++q) {
      R.row[q] = (lane + 32 * q < n) ? S.prow[lane + 32 * q] : 0;
      R.v[q] = (lane + 32 * q < n) ? b[R.row[q]] : 0.0;
    }
    j = lu_back<3>(A, lda, dinv, R, n - 1);
    j = lu_back<2>(A, lda, dinv, R, j);
    j = lu_back<1>(A, lda, dinv, R, j);
#pragma unroll
    for (int q = 0; q < LU_RPL; ++q) if (lane + 32 * q < n) b[lane + 32 * q] = R.v[q];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(IPM_BLOCK, 1) ipm_kernel(const __grid_constant__ IpmArgs A) {
  extern __shared__ double dyn[];
  __shared__ IpmShared sh;
  __shared__ IpmScal sc;
  __shared__ double grid[256];
  __shared__ int s_ok;
  __shared__ unsigned s_mask;
  if (A.skip && *A.skip) return;
  const int k = A.k, s = k * (k + 1) / 2, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* Q11 = dyn;            // s*s (mode 0)
  double* coeff = dyn + s * s;  // s*s
  double* sm = A.smalls;
  if (tid == 0) {
    int a = 0, o = 0;
    for (int b = 0; b < k; ++b)
      for (int c = 0; c <= b; ++c) {
        sh.bi[a] = b; sh.ci[a] = c;
        if (b != c) sh.cord[o++] = a;
        ++a;
      }
    for (int b = 0; b < k; ++b) sh.cord[o++] = b * (b + 1) / 2 + b;
  }
  const int ngrid = A.ipm_grid;
  for (int j = tid; j < ngrid && j < 256; j += IPM_BLOCK) grid[j] = pow(0.9, (double)j);
  __syncthreads();
  const double tr = A.trace_ub;
  const double tXb_raw = sm[A.o_sc + SC_TRXBAR];
  const double tX = (tXb_raw > 0.0) ? tXb_raw : tr;
  const double bpo = sm[A.o_sc + SC_BPO];
  for (int a = tid; a < s; a += IPM_BLOCK) sh.sI[a] = (sh.bi[a] == sh.ci[a]) ? 1.0 : 0.0;
  if (A.mode == 0) {
    const double rho = A.rho;
    const double* QB = sm + A.o_QB;
    const double qs = tr * tr / rho;
    for (int e = tid; e < s * s; e += IPM_BLOCK) Q11[e] = qs * QB[e];
    const double* GZ = sm + A.o_GZ;
    const double* GYmC = sm + A.o_GYmC;
    const double* GB = sm + A.o_GB;
    const double q12s = tr * tr / (rho * tX);
    for (int a = tid; a < s; a += IPM_BLOCK) {
      const int b = sh.bi[a], c = sh.ci[a];
      sh.q12[a] = q12s * svec_of(GZ, k, b, c);
      // svec(V^T (A*(y) - C - A*(b - ups)/rho) V)
      sh.h1[a] = tr * (svec_of(GYmC, k, b, c) - svec_of(GB, k, b, c) / rho);
    }
    if (tid == 0) {
      sc.q22 = (tr * tr / (rho * tX * tX)) * sm[A.o_sc + SC_ZZ];
      sc.h2 = (tr / tX) * (sm[A.o_sc + SC_ZY] - bpo - sm[A.o_sc + SC_ZBMU] / rho);
    }
  } else {
    const double* GYC = sm + A.o_GYC;  // V^T (A*(y_cand) - C) V
    for (int a = tid; a < s; a += IPM_BLOCK) {
      sh.h1[a] = tr * svec_of(GYC, k, sh.bi[a], sh.ci[a]);   // g_1
      sh.q12[a] = 0.0;
    }
    if (tid == 0) { sc.q22 = 0.0; sc.h2 = (tr / tX) * (sm[A.o_sc + SC_ZYC] - bpo); }   // g_2
  }
  // ---- initial point ----
  if (A.mode == 0) {
    const double* S0 = sm + A.o_Ssub;
    for (int e = tid; e < k * k; e += IPM_BLOCK) sh.S[e] = S0[e] / tr;
    if (tid == 0) sc.eta = (tX / tr) * sm[A.o_sc + SC_ETA_SUB];
  } else {
    for (int e = tid; e < k * k; e += IPM_BLOCK) {
      const int r = e / k, c = e - r * k;
      sh.S[e] = (r == c) ? 0.99 * (1.0 / (k + 1.0)) : 0.0;
    }
    if (tid == 0) sc.eta = (bpo == 0.0) ? 0.00001 : 0.99 * (1.0 / (k + 1.0));
  }
  __syncthreads();
  for (int a = tid; a < s; a += IPM_BLOCK) sh.sS[a] = svec_of(sh.S, k, sh.bi[a], sh.ci[a]);
  __syncthreads();
  const double q22 = sc.q22, h2 = sc.h2;
  double eta = sc.eta;
  // T_svec -> sh.ord (temporary)
  for (int a = tid; a < s; a += IPM_BLOCK) {
    if (A.mode == 0) {
      double v = 0.0;
      for (int b = 0; b < s; ++b) v += Q11[a * s + b] * sh.sS[b];
      sh.ord[a] = v + eta * sh.q12[a] + sh.h1[a];
    } else {
      sh.ord[a] = sh.h1[a];
    }
  }
  if (wid == 0) {
    const double d = wdot(sh.q12, sh.sS, s);
    if (lane == 0) sc.zeta = (A.mode == 0) ? (d + eta * q22 + h2) : h2;
  }
  __syncthreads();
  svec_inv_to(sh.ord, k, s, sh.bi, sh.ci, sh.T);
  __syncthreads();
  if (tid == 0) {
    double zeta = sc.zeta, vmax = zeta, vmin = zeta;
    for (int b = 0; b < k; ++b) { vmax = fmax(vmax, sh.T[b * k + b]); vmin = fmin(vmin, sh.T[b * k + b]); }
    double width = vmax - vmin;
    width = (width < 100.0) ? 100.0 : width;
    double omega = -1.01 * vmin;
    omega = (omega < width) ? width : omega;
    for (int b = 0; b < k; ++b) sh.T[b * k + b] += omega;
    sc.zeta = zeta + omega;
    sc.omega = omega;
    double trS = 0.0;
    for (int b = 0; b < k; ++b) trS += sh.S[b * k + b];
    sc.trS = trS;
    sc.step = 1.0;
    sc.it = 0;
  }
  __syncthreads();
  for (int a = tid; a < s; a += IPM_BLOCK) sh.sT[a] = svec_of(sh.T, k, sh.bi[a], sh.ci[a]);
  __syncthreads();
  if (wid == 0) {
    const double d = wdot(sh.sS, sh.sT, s);
    if (lane == 0)
      sc.mu = (d + sc.eta * sc.zeta + sc.omega * (1 - sc.trS - sc.eta)) / (2 * k + 4.0);
  }
  __syncthreads();
  const int maxit = A.max_iters;
  const double eps = A.eps;
  long long ph0 = 0, ph1 = 0, ph2 = 0, ph3 = 0, tclk = 0;
  while (true) {
    if (tid == 0) tclk = clock64();
    if (tid == 0) {
      const bool cont = (sc.it < maxit) &&
          ((A.mode == 0) ? (sc.mu > eps && sc.step > eps * eps) : (sc.mu > eps));
      sc.cont = cont;
    }
    __syncthreads();
    if (!sc.cont) break;
    const double mu = sc.mu, eta_ = sc.eta, zeta = sc.zeta, omega = sc.omega, tIS = sc.trS;
    // ---- Newton system ----
    // The step's scalar coefficients are chains of FP64 divisions of about 600
    // cycles each: the last warp forms them, independent quotients on lanes of
    // their own (k1, ze, mu/omega and mu/eta together, then 1/den and, for the
    // quadratic subproblem, t1 and t2, for the lower bound its coefficient and t1),
    // while the other warps form F1 = Q11 svec(S) + ...  They are read after the
    // barrier that precedes the inverse below.
    if (wid == IPM_BLOCK / 32 - 1) {
      double F2 = 0.0;
      if (A.mode == 0) {
        const double d = wdot(sh.q12, sh.sS, s);
        F2 = d + eta_ * q22 + h2;
        F2 = F2 + (-zeta + omega);
      }
      F2 = __shfl_sync(0xffffffffu, F2, 0);
      const double q4 = (lane == 0 ? 1 - tIS - eta_ : lane == 1 ? zeta : mu) /
                        ((lane & 1) ? eta_ : omega);
      const double k1 = __shfl_sync(0xffffffffu, q4, 0), ze = __shfl_sync(0xffffffffu, q4, 1);
      const double mow = __shfl_sync(0xffffffffu, q4, 2), moe = __shfl_sync(0xffffffffu, q4, 3);
      const double k2 = ze + q22;
      const double den = fma(k1, k2, 1.0);
      double num, dv;
      if (A.mode == 0) {
        const double lin = mow + tIS + eta_ - 1;
        num = (lane == 1) ? fma(k1, F2 - moe + zeta, lin)
            : (lane == 2) ? fma(-k2, lin, F2 - moe + zeta) : 1.0;
        dv = den;
      } else {
        num = (lane == 1) ? ze * (fma(-k1, moe - h2 - omega, mow) + tIS + eta_ - 1)
            : (lane == 2) ? ze : 1.0;
        dv = (lane == 1) ? fma(-k1, ze, -1.0) : (lane == 2) ? fma(k1, ze, 1.0) : den;
      }
      const double q3 = num / dv;
      const double t1 = __shfl_sync(0xffffffffu, q3, 1), t2 = __shfl_sync(0xffffffffu, q3, 2);
      if (lane == 0) {
        sc.k1 = k1; sc.k2 = k2; sc.den = den; sc.ze = ze;
        sc.F2 = F2;
        sc.mow = mow; sc.moe = moe;
        sc.rden = q3;
        sc.t1 = t1;
        if (A.mode == 0) {
          sc.t2 = t2;
        } else {
          sc.lbc = t2;
          sc.t2 = h2 - moe;
        }
      }
    }
    if (A.mode == 0) {
      cta_matvec3(Q11, sh.sS, s, sh.part3, sh.F1);
      for (int a = tid; a < s; a += IPM_BLOCK) {
        const double f = sh.F1[a] + eta_ * sh.q12[a] + sh.h1[a];
        sh.F1[a] = f + (-sh.sT[a] + omega * sh.sI[a]);
      }
    }
    // S^-1 (the reference's jnp.linalg.inv, solver/usbs.py:91)
    __syncthreads();
    const double k1 = sc.k1, k2 = sc.k2, den = sc.den, ze = sc.ze;
    {
      const bool okinv = cta_inverse(sh.S, k, sh.Si, coeff);
      if (!okinv && tid == 0) atomicOr(A.status, ST_SMALL_DENSE_FAIL);
    }
    __syncthreads();
    const double F2 = (A.mode == 0) ? sc.F2 : 0.0;
    for (int a = tid; a < s; a += IPM_BLOCK) sh.sSi[a] = svec_of(sh.Si, k, sh.bi[a], sh.ci[a]);
    // coefficient matrix, every entry computed (S^-1 is not exactly symmetric in
    // floating point; mirroring one triangle measurably degrades the Newton
    // steps once the system is ill-conditioned near the end of the IPM)
    const double lbc = (A.mode == 1) ? sc.lbc : 0.0;
    const double rden = sc.rden;
    if (A.mode == 0) {
      for (int a2 = tid; a2 < s; a2 += IPM_BLOCK) {
        sh.u2[a2] = k1 * sh.q12[a2] + sh.sI[a2];
        sh.w2[a2] = sh.q12[a2] - k2 * sh.sI[a2];
      }
      __syncthreads();
    }
    // every entry of the s x s matrix, flat over the CTA; columns in cord order
    // so that the off-diagonal / diagonal branch is uniform across most warps
    // (stored column-major for the LU: coeff[a2 * s + a] is row a, column a2;
    // consecutive threads take consecutive rows of one column)
    for (int e = tid; e < s * s; e += IPM_BLOCK) {
      const int ca = e / s, a = e - ca * s, a2 = sh.cord[ca];
      double v = symkron_sum(sh.T, sh.Si, k, sh.bi[a], sh.ci[a], sh.bi[a2], sh.ci[a2]);
      if (A.mode == 0) {
        v = Q11[a * s + a2] + v;
        v -= (sh.q12[a] * sh.u2[a2] + sh.sI[a] * sh.w2[a2]) * rden;
      } else {
        v += lbc * (sh.sI[a] * sh.sI[a2]);
      }
      coeff[a2 * s + a] = v;
    }
    __syncthreads();
    for (int a = tid; a < s; a += IPM_BLOCK) {
      double o;
      if (A.mode == 0) {
        o = -sh.F1[a] + mu * sh.sSi[a] - sh.sT[a];
        o += sc.t1 * sh.q12[a];
        o += sc.t2 * sh.sI[a];
      } else {
        o = sc.t1 * sh.sI[a];
        o += sc.t2 * sh.sI[a] - sh.h1[a];
        o += mu * sh.sSi[a];
      }
      sh.ord[a] = o;
    }
    __syncthreads();
    if (tid == 0) { const long long c = clock64(); ph0 += c - tclk; tclk = c; }
    ipm_lu_solve(coeff, s, sh.ord, s, sh.dinv, &s_ok);
    if (tid == 0) { const long long c = clock64(); ph1 += c - tclk; tclk = c; }
    if (tid == 0 && !s_ok) atomicOr(A.status, ST_SMALL_DENSE_FAIL);
    // sh.ord now holds dsS
    if (wid == 0) {
      double t1 = 0.0, t2 = 0.0, t3 = 0.0;
      for (int a = lane; a < s; a += 32) {
        const double x = sh.ord[a];
        if (A.mode == 0) {
          t1 += (k1 * sh.q12[a] + sh.sI[a]) * x;
          t2 += (sh.q12[a] - k2 * sh.sI[a]) * x;
          t3 += sh.q12[a] * x;
        } else {
          t1 += sh.sI[a] * x;
        }
      }
      t1 = warp_sum(t1);
      if (A.mode == 0) { t2 = warp_sum(t2); t3 = warp_sum(t3); }
      // (every lane the same, but for one quotient per lane)
      const double mow = sc.mow, moe = sc.moe;
      double d_eta, d_omega, d_zeta;
      if (A.mode == 0) {
        const double ne = fma(k1, -F2 + moe - zeta, -t1 - mow - tIS - eta_ + 1);
        const double no = fma(k2, mow + tIS + eta_ - 1, -F2 + moe - zeta) - t2;
        const double qd = (lane == 0 ? ne : no) / den;
        d_eta = __shfl_sync(0xffffffffu, qd, 0);
        d_omega = __shfl_sync(0xffffffffu, qd, 1);
        d_zeta = fma(d_eta, q22, t3) + d_omega + F2;
      } else {
        d_eta = (fma(-k1, moe - h2 - omega, t1) + mow + tIS + eta_ - 1) / fma(-k1, ze, -1.0);
        d_omega = fma(-ze, d_eta, moe);
        d_omega = d_omega + (-h2 - omega);
        d_zeta = d_omega - zeta + h2 + omega;
      }
      // step size from the linear variables (solver/usbs.py:128-132)
      const double qr = (lane == 0 ? d_eta : lane == 1 ? d_zeta : d_omega) /
                        (lane == 0 ? eta_ : lane == 1 ? zeta : omega);
      const double r = nanmin2(nanmin2(__shfl_sync(0xffffffffu, qr, 0),
                                       __shfl_sync(0xffffffffu, qr, 1)),
                               __shfl_sync(0xffffffffu, qr, 2));
      if (lane == 0) {
        sc.d_eta = d_eta; sc.d_omega = d_omega; sc.d_zeta = d_zeta;
        double st = -1.0 / r;
        if (!isnan(st) && st > 1.0) st = 1.0;
        sc.st = 0.99 * ((st <= 0.0) ? 1.0 : st);
      }
    }
    __syncthreads();
    const double d_eta = sc.d_eta, d_omega = sc.d_omega;
    if (A.mode == 0) {
      cta_matvec3(Q11, sh.ord, s, sh.part3, sh.dsT);
      for (int a = tid; a < s; a += IPM_BLOCK)
        sh.dsT[a] = sh.dsT[a] + d_eta * sh.q12[a] + d_omega * sh.sI[a] + sh.F1[a];
    } else {
      for (int a = tid; a < s; a += IPM_BLOCK)
        sh.dsT[a] = d_omega * sh.sI[a] - sh.sT[a] + sh.h1[a] + omega * sh.sI[a];
    }
    __syncthreads();
    svec_inv_to(sh.ord, k, s, sh.bi, sh.ci, sh.dS);
    svec_inv_to(sh.dsT, k, s, sh.bi, sh.ci, sh.dT);
    __syncthreads();
    // ---- line search over the grid 0.9^j (solver/usbs.py:134-154): the largest
    // grid step keeping S and T positive definite is the first positive-definite
    // grid index ----
    int firstS, firstT;
    {
      // PD-ness of A + a dA is monotone along the grid (the PD steps form an
      // interval containing 0), so after the first 16 points the first PD
      // index is bracketed by testing every 16th point, then resolved inside
      // the bracket: at most three rounds of 16 tests per matrix.
      const int half = tid >> 7, sub = (tid >> 3) & 15;
      auto gstep = [&](int j) { return (j < 256) ? grid[j] : pow(0.9, (double)j); };
      auto tests = [&](bool active, int j) {
        return pd_tests(sh.S, sh.dS, sh.T, sh.dT, k, s, sh.bi, sh.ci, active,
                        active ? gstep(j) : 0.0, coeff, &s_mask);
      };
      auto lowest = [](unsigned m) { return m ? __ffs(m) - 1 : -1; };
      const unsigned m1 = tests(sub < ngrid, sub);
      firstS = lowest(m1 & 0xffffu);
      firstT = lowest(m1 >> 16);
      if (ngrid > 16 && (firstS < 0 || firstT < 0)) {
        __syncthreads();
        const bool need2 = (half ? firstT : firstS) < 0;
        const unsigned m2 = tests(need2 && 16 + 16 * sub < ngrid, min(31 + 16 * sub, ngrid - 1));
        const int qS = lowest(m2 & 0xffffu), qT = lowest(m2 >> 16);
        if (m2) {
          __syncthreads();
          const int q = half ? qT : qS;
          const int j3 = 16 + 16 * max(q, 0) + sub, jq = min(31 + 16 * max(q, 0), ngrid - 1);
          const unsigned m3 = tests(need2 && q >= 0 && j3 <= jq, j3);
          const int fS = lowest(m3 & 0xffffu), fT = lowest(m3 >> 16);
          if (firstS < 0 && qS >= 0 && fS >= 0) firstS = 16 + 16 * qS + fS;
          if (firstT < 0 && qT >= 0 && fT >= 0) firstT = 16 + 16 * qT + fT;
        }
      }
    }
    if (wid == 0) {
      if (lane == 0) {
        const double cS = (firstS < 0) ? 0.0 : (firstS < 256 ? grid[firstS] : pow(0.9, (double)firstS));
        const double cT = (firstT < 0) ? 0.0 : (firstT < 256 ? grid[firstT] : pow(0.9, (double)firstT));
        const double cand = (cS < cT) ? cS : cT;
        double st = sc.st;
        st = (st < cand) ? st : cand;
        sc.st = st;
        sc.eta = eta_ + st * d_eta;
        sc.zeta = zeta + st * sc.d_zeta;
        sc.omega = omega + st * d_omega;
      }
    }
    __syncthreads();
    if (tid == 0) { const long long c = clock64(); ph2 += c - tclk; tclk = c; }
    const double st = sc.st;
    for (int e = tid; e < k * k; e += IPM_BLOCK) {
      sh.S[e] = sh.S[e] + st * sh.dS[e];
      sh.T[e] = sh.T[e] + st * sh.dT[e];
    }
    __syncthreads();
    for (int a = tid; a < s; a += IPM_BLOCK) {
      sh.sS[a] = svec_of(sh.S, k, sh.bi[a], sh.ci[a]);
      sh.sT[a] = svec_of(sh.T, k, sh.bi[a], sh.ci[a]);
    }
    __syncthreads();
    if (wid == 0) {
      const double d = wdot(sh.sS, sh.sT, s);
      if (lane == 0) {
        double trS = 0.0;
        for (int b = 0; b < k; ++b) trS += sh.S[b * k + b];
        double mun = (d + sc.eta * sc.zeta + sc.omega * (1 - trS - sc.eta)) / (2 * k + 4.0);
        mun *= (st > 0.2) ? (0.5 - 0.4 * st * st) : 1.0;
        if (!(isnan(mun) || mun <= mu)) mun = mu;
        if (A.dbg && sc.it < 128) {
          double* d = A.dbg + sc.it * 8;
          d[0] = mun; d[1] = st; d[2] = sc.eta; d[3] = sc.zeta; d[4] = sc.omega;
          d[5] = sc.d_eta; d[6] = sc.d_omega; d[7] = trS;
        }
        sc.mu = mun;
        sc.trS = trS;
        sc.step = st;
        sc.it = sc.it + 1;
      }
    }
    __syncthreads();
    if (tid == 0) { const long long c = clock64(); ph3 += c - tclk; }
  }
  if (tid == 0 && A.prof) {
    A.prof[0] += (double)ph0; A.prof[1] += (double)ph1; A.prof[2] += (double)ph2;
    A.prof[3] += (double)ph3;
  }
  // ---- outputs ----
  if (A.mode == 0) {
    for (int e = tid; e < k * k; e += IPM_BLOCK) sm[A.o_Sout + e] = tr * sh.S[e];
    if (tid == 0) {
      sm[A.o_sc + SC_ETA] = (tr / tX) * sc.eta;
      sm[A.o_sc + SC_QITERS] = sc.it;
    }
  } else {
    if (wid == 0) {
      const double g1S = wdot(sh.h1, sh.sS, s);
      if (lane == 0) {
        sm[A.o_sc + SC_LB] = sm[A.o_sc + SC_BYC] - g1S - sc.eta * h2;
        sm[A.o_sc + SC_LITERS] = sc.it;
      }
    }
  }
}

// eigh(S) and the quantities the outer iteration derives from it.  One warp.
__global__ void __launch_bounds__(IPM_BLOCK) eigS_kernel(EigSArgs A) {
  if (A.skip && *A.skip) return;
  constexpr int L = 16;                               // ld of the FP64 k x k blocks
  __shared__ double Sd[L * L], Z[L * L], R[L * L], S2[L * L], Wb[L * L], lam[L];
  __shared__ double GW[IPM_MAXK * IPM_MAXK];
  __shared__ float Af[2 * (L + 1) + L * L + L], Af2[2 * (L + 1) + L * L + L], Zf[L * (L + 1)];
  __shared__ float wf[L], redf[32];
  __shared__ int order[L];
  const int k = A.k, kc = A.k_curr, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* sm = A.smalls;
  const double* S = sm + A.o_Sout;
  // eigh(S) (solver/usbs.py:568): FP32 parallel Jacobi at order 16, refined to
  // FP64 accuracy by two Ogita-Aishima steps, then sorted ascending
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, c = e - r * k;
    Sd[r * L + c] = S[e];
    Af[r * (L + 1) + c] = (float)S[e];
  }
  __syncthreads();
  bool ok = cta_jacobi_f32<L>(Af, Af2, L + 1, k, wf, Zf, L + 1, redf);
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, c = e - r * k;
    Z[r * L + c] = (double)Zf[r * (L + 1) + c];
  }
  __syncthreads();
  cta_refine_eig(Sd, Z, R, S2, Wb, lam, k, L);
  cta_refine_eig(Sd, Z, R, S2, Wb, lam, k, L);
  if (tid < k) {
    const double v = lam[tid];
    int r = 0;
    for (int j = 0; j < k; ++j) {
      const double u = lam[j];
      r += (u < v || (u == v && j < tid)) ? 1 : 0;
    }
    order[r] = tid;
  }
  __syncthreads();
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, c = e - r * k;
    S2[r * L + c] = Z[r * L + order[c]];
  }
  double lv = (tid < k) ? lam[order[tid]] : 0.0;
  __syncthreads();
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, c = e - r * k;
    Z[r * L + c] = S2[r * L + c];
  }
  if (tid < k) lam[tid] = fmax(lv, 0.0);   // clip(eigvals, 0)
  if (!ok && tid == 0) atomicOr(A.status, ST_SMALL_DENSE_FAIL);
  __syncthreads();
  double* W = sm + A.o_W;
  double* Sp = sm + A.o_Splus;
  double* Scp = sm + A.o_Scplus;
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, c = e - r * k;
    W[e] = Z[r * L + c];
    double a = 0.0, b = 0.0;
    for (int j = 0; j < k; ++j) {
      const double t = Z[r * L + j] * lam[j] * Z[c * L + j];
      a += t;
      if (j < kc) b += t;
    }
    Sp[e] = a;
    Scp[e] = b;
  }
  // trace(F^T C F) = sum_j lam_j (W^T G_C W)_jj
  const double* GC = sm + A.o_GC;
  for (int e = tid; e < k * k; e += IPM_BLOCK) {
    const int r = e / k, j = e - r * k;
    double v = 0.0;
    for (int c = 0; c < k; ++c) v += GC[r * k + c] * Z[c * L + j];
    GW[e] = v;   // (G_C W)[r][j]
  }
  __syncthreads();
  if (wid == 0) {
    double pj = 0.0;
    if (lane < k) {
      for (int r = 0; r < k; ++r) pj += Z[r * L + lane] * GW[r * k + lane];
      pj *= lam[lane];
    }
    const double pall = warp_sum(pj);
    const double pcur = warp_sum(lane < kc ? pj : 0.0);
    const double lc = warp_sum(lane < kc ? lam[lane] : 0.0);
    if (lane == 0) {
      double trS = 0.0;
      for (int b = 0; b < k; ++b) trS += S[b * k + b];
      sm[A.o_sc + SC_TRS] = trS;
      sm[A.o_sc + SC_SUMLAMC] = lc;
      sm[A.o_sc + SC_PFULL] = pall;
      sm[A.o_sc + SC_PCUR] = pcur;
    }
  }
  // W_past = W[:, kc:]
  const int kp = k - kc;
  for (int e = tid; e < k * kp; e += IPM_BLOCK) {
    const int r = e / kp, c = e - r * kp;
    sm[A.o_Wpast + e] = Z[r * L + kc + c];
  }
  // M = S+ (V^T Omega), Mc = Sc+ (V^T Omega)    (k x ssk)
  if (A.ssk > 0) {
    __syncthreads();
    const double* VtO = sm + A.o_VtO;
    for (int e = tid; e < k * A.ssk; e += IPM_BLOCK) {
      const int r = e / A.ssk, c = e - r * A.ssk;
      double a = 0.0, b = 0.0;
      for (int j = 0; j < k; ++j) {
        a += Sp[r * k + j] * VtO[j * A.ssk + c];
        b += Scp[r * k + j] * VtO[j * A.ssk + c];
      }
      sm[A.o_M + e] = a;
      sm[A.o_Mc + e] = b;
    }
  }
}

// One pass of (shifted) Cholesky QR: R^T R = G (+ shift I), output R^-1
// (upper), one warp.  Column j of R: lanes i >= j form G_ji - sum_p R_pj R_pi,
// lane j's value gives r_jj = sqrt(.), the others are scaled by 1 / r_jj.
// R^-1 by back substitution with one lane per column (reciprocals of the
// diagonal computed once).
__global__ void cholqr_kernel(CholQRArgs A) {
  if (A.skip && *A.skip) return;
  __shared__ double R[IPM_MAXK * IPM_MAXK], Ri[IPM_MAXK * IPM_MAXK], rd[IPM_MAXK];
  const int k = A.k, lane = threadIdx.x;
  double* sm = A.smalls;
  const double* G = sm + A.o_G;
  double shift = 0.0;
  if (A.shifted) {
    double tr = 0.0;
    for (int b = 0; b < k; ++b) tr += G[b * k + b];
    // Fukaya et al. (SIAM J. Sci. Comput. 42(1), 2020): s = 11 (m n + n (n + 1)) u ||A||_2^2
    shift = 11.0 * ((double)A.n * k + (double)k * (k + 1)) * 1.1102230246251565e-16 * tr;
  }
  for (int e = lane; e < k * k; e += 32) R[e] = 0.0;
  __syncwarp();
  bool ok = true;
  for (int j = 0; j < k; ++j) {
    double v = 0.0;
    if (lane >= j && lane < k) {
      v = G[j * k + lane] + ((lane == j) ? shift : 0.0);
      for (int p = 0; p < j; ++p) v -= R[p * k + j] * R[p * k + lane];
    }
    double d = __shfl_sync(0xffffffffu, v, j);
    if (!(d > 0.0)) { ok = false; d = 1.0; }
    const double rjj = sqrt(d);
    const double inv = 1.0 / rjj;
    if (lane == j) { R[j * k + j] = rjj; rd[j] = inv; }
    else if (lane > j && lane < k) R[j * k + lane] = v * inv;
    __syncwarp();
  }
  if (lane < k) {
    const int c = lane;
    for (int r = k - 1; r >= 0; --r) {
      double v = (r == c) ? 1.0 : 0.0;
      for (int p = r + 1; p <= c; ++p) v -= R[r * k + p] * Ri[p * k + c];
      Ri[r * k + c] = (r > c) ? 0.0 : v * rd[r];
    }
  }
  if (!ok && lane == 0) atomicOr(A.status, ST_SMALL_DENSE_FAIL);
  __syncwarp();
  for (int e = lane; e < k * k; e += 32) sm[A.o_Rinv + e] = Ri[e];
}

// Q11, then the Newton matrix, whose room the inverse of S (4 k^2) and the line
// search (32 tests of s + IPM_MAXK) use before and after it
static size_t ipm_dyn_doubles(int k) {
  const size_t s = (size_t)k * (k + 1) / 2;
  size_t w = s * s;
  if (w < (size_t)4 * k * k) w = (size_t)4 * k * k;
  if (w < 32 * (s + IPM_MAXK)) w = 32 * (s + IPM_MAXK);
  return s * s + w;
}

int launch_ipm(const IpmArgs& a, cudaStream_t st) {
  const size_t dyn = ipm_dyn_doubles(a.k) * sizeof(double);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(ipm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(ipm_dyn_doubles(IPM_MAXK) * sizeof(double)));
    attr = true;
  }
  ipm_kernel<<<1, IPM_BLOCK, dyn, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("ipm launch: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// cta_inverse of one matrix: the inverse and whether every pivot was usable
__global__ void __launch_bounds__(IPM_BLOCK) selftest_inverse_kernel(
    int n, const double* __restrict__ A, double* __restrict__ Ainv, int* ok) {
  __shared__ double M[IPM_MAXK * IPM_MAXK], R[IPM_MAXK * IPM_MAXK], ws[4 * IPM_MAXK * IPM_MAXK];
  for (int e = threadIdx.x; e < n * n; e += IPM_BLOCK) M[e] = A[e];
  __syncthreads();
  const bool good = cta_inverse(M, n, R, ws);
  for (int e = threadIdx.x; e < n * n; e += IPM_BLOCK) Ainv[e] = R[e];
  if (threadIdx.x == 0) *ok = good ? 1 : 0;
}

int launch_selftest_inverse(int n, const double* A, double* Ainv, int* ok, cudaStream_t st) {
  selftest_inverse_kernel<<<1, IPM_BLOCK, 0, st>>>(n, A, Ainv, ok);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("selftest_inverse: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

int launch_eigS(const EigSArgs& a, cudaStream_t st) {
  eigS_kernel<<<1, IPM_BLOCK, 0, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("eigS launch: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

int launch_cholqr(const CholQRArgs& a, cudaStream_t st) {
  cholqr_kernel<<<1, 32, 0, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("cholqr launch: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

}  // namespace usbs
