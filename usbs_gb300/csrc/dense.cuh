// Small dense FP64 linear algebra executed by one warp or one CTA in shared
// memory: the projected Lanczos eigenproblem (m <= 32), the k x k bundle
// matrices (k <= 16) and the s x s IPM Newton systems (s <= 136).
//
// Methods (textbook, own code):
//  * symmetric eigensolver: Householder tridiagonalisation followed by the
//    implicit symmetric QR iteration with Wilkinson shift (Golub & Van Loan,
//    Matrix Computations, 4th ed., Alg. 8.3.1 and 8.3.3), eigenvectors
//    accumulated, eigenvalues sorted ascending;
//  * LU with partial pivoting and forward/back substitution (G&VL Alg. 3.4.1);
//  * Cholesky (G&VL Alg. 4.2.1) as the positive-definiteness test.
#pragma once
#include "common.cuh"

namespace usbs {

// Eigen-decomposition of the symmetric n x n matrix A (row-major, lda) by one
// warp.  On return w[0..n-1] holds the eigenvalues in ascending order and
// Z (row-major, ldz) the eigenvectors as columns.  A is destroyed.  Returns
// false if the QR iteration did not converge in 30 n sweeps.  n <= 32.
// VECTORS = false: the eigenvalues alone, by the same arithmetic (Z is not used).
template <bool VECTORS = true>
__device__ inline bool warp_syev(double* A, int lda, int n, double* w, double* Z, int ldz) {
  const int lane = threadIdx.x & 31;
  // Z = I
  if (VECTORS)
    for (int j = 0; j < n; ++j)
      if (lane < n) Z[lane * ldz + j] = (lane == j) ? 1.0 : 0.0;
  __syncwarp();
  // ---- Householder tridiagonalisation: A <- H A H, Z <- Z H ----
  for (int j = 0; j + 2 < n; ++j) {
    const int r0 = j + 1;  // reflector acts on rows/cols r0..n-1
    double xi = (lane > r0 && lane < n) ? A[lane * lda + j] : 0.0;
    double sigma = warp_sum(xi * xi);
    double alpha = A[r0 * lda + j];
    if (sigma == 0.0) continue;  // already tridiagonal in this column
    double nrm = sqrt(alpha * alpha + sigma);
    double v0 = (alpha <= 0.0) ? (alpha - nrm) : (-sigma / (alpha + nrm));
    double beta = 2.0 * v0 * v0 / (sigma + v0 * v0);
    // v (length n, zero outside r0..n-1), v[r0] = 1
    double vi = (lane == r0) ? 1.0 : ((lane > r0 && lane < n) ? xi / v0 : 0.0);
    // p = beta * A_sub v  (lane i computes component i); every lane shuffles
    double p = 0.0;
    for (int l = r0; l < n; ++l) {
      double vl = __shfl_sync(0xffffffffu, vi, l);
      if (lane >= r0 && lane < n) p += A[lane * lda + l] * vl;
    }
    p *= beta;
    double K = 0.5 * beta * warp_sum(p * vi);
    double wv = p - K * vi;
    __syncwarp();
    // A_sub -= v w^T + w v^T
    for (int l = r0; l < n; ++l) {
      double vl = __shfl_sync(0xffffffffu, vi, l);
      double wl = __shfl_sync(0xffffffffu, wv, l);
      if (lane >= r0 && lane < n) A[lane * lda + l] -= vi * wl + wv * vl;
    }
    __syncwarp();
    if (lane == r0) { A[r0 * lda + j] = nrm; A[j * lda + r0] = nrm; }
    if (lane > r0 && lane < n) { A[lane * lda + j] = 0.0; A[j * lda + lane] = 0.0; }
    // Z <- Z (I - beta v v^T): row i of Z: z_i -= beta (z_i . v) v^T, the rows'
    // dots 16 at a time by a butterfly whose payload halves (lanes 2 i and
    // 2 i + 1 end with row i's, summed as by a warp sum)
    for (int i0 = 0; VECTORS && i0 < n; i0 += 16) {
      double zr[16], x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        zr[i] = (lane < n && i0 + i < n) ? Z[(i0 + i) * ldz + lane] : 0.0;
        x[i] = (lane < n && i0 + i < n) ? zr[i] * vi : 0.0;
      }
#pragma unroll
      for (int h = 16, w = 8; w >= 1; h >>= 1, w >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < w) {
            const double send = up ? x[i] : x[i + w], keep = up ? x[i + w] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
          }
      }
      const double bz = beta * (x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1));
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const double b = __shfl_sync(0xffffffffu, bz, 2 * i);
        if (lane < n && i0 + i < n) Z[(i0 + i) * ldz + lane] = fma(-b, vi, zr[i]);
      }
    }
    __syncwarp();
  }
  // ---- implicit symmetric QR with Wilkinson shift on (d, e) ----
  // d/e held redundantly by all lanes in registers would need dynamic indexing;
  // keep them in A's diagonal / subdiagonal (shared memory), lane 0 writes.
  double* d = w;                 // eigenvalues end up here
  for (int i = lane; i < n; i += 32) d[i] = A[i * lda + i];
  __syncwarp();
  // subdiagonal e[i] = A[i+1][i] stored in A[(i+1)*lda + i]
  const double eps = 1.1102230246251565e-16;
  int iters = 0, maxit = 30 * n;
  int hi = n - 1;
  while (hi > 0) {
    // deflate the trailing off-diagonal if negligible
    {
      double e = A[hi * lda + hi - 1];
      if (fabs(e) <= eps * (fabs(d[hi - 1]) + fabs(d[hi])) || fabs(e) < 1e-300) {
        __syncwarp();
        if (lane == 0) A[hi * lda + hi - 1] = 0.0;
        __syncwarp();
        --hi;
        continue;
      }
    }
    // start p of the unreduced block ending at hi: the last negligible
    // subdiagonal below it (lane p looks at p, p - 1), which becomes zero
    int p = 0;
    {
      bool neg = false;
      if (lane >= 1 && lane < hi) {
        const double e = A[lane * lda + lane - 1];
        neg = fabs(e) <= eps * (fabs(d[lane - 1]) + fabs(d[lane])) || fabs(e) < 1e-300;
      }
      const unsigned nb = __ballot_sync(0xffffffffu, neg);
      if (nb) {
        p = 31 - __clz(nb);
        if (lane == p) A[p * lda + p - 1] = 0.0;
        __syncwarp();
      }
    }
    if (++iters > maxit) return false;
    // Wilkinson shift from the trailing 2x2
    double a1 = d[hi - 1], a2 = d[hi], b = A[hi * lda + hi - 1];
    double dd = 0.5 * (a1 - a2);
    double den = dd + copysign(hypot(dd, b), dd == 0.0 ? 1.0 : dd);
    double mu = a2 - b * b / den;
    double x = d[p] - mu, z = A[(p + 1) * lda + p];
    for (int k = p; k < hi; ++k) {
      double r = hypot(x, z);
      // (both quotients in one division, on even and odd lanes)
      const double cs = (r == 0.0) ? ((lane & 1) ? 0.0 : 1.0) : ((lane & 1) ? z : x) / r;
      const double c = __shfl_sync(0xffffffffu, cs, 0), s = __shfl_sync(0xffffffffu, cs, 1);
      double ak = d[k], ak1 = d[k + 1], bk = A[(k + 1) * lda + k];
      double f = (k + 1 < hi) ? A[(k + 2) * lda + k + 1] : 0.0;
      // new 2x2 block
      double nak = c * c * ak + 2.0 * c * s * bk + s * s * ak1;
      double nak1 = s * s * ak - 2.0 * c * s * bk + c * c * ak1;
      double nbk = c * s * (ak1 - ak) + (c * c - s * s) * bk;
      __syncwarp();
      if (lane == 0) {
        if (k > p) A[k * lda + k - 1] = r;   // e[k-1] after removing the bulge
        d[k] = nak;
        d[k + 1] = nak1;
        A[(k + 1) * lda + k] = nbk;
        if (k + 1 < hi) A[(k + 2) * lda + k + 1] = c * f;
      }
      // rotate eigenvector columns k, k+1: (Z P^T)
      if (VECTORS && lane < n) {
        double zk = Z[lane * ldz + k], zk1 = Z[lane * ldz + k + 1];
        Z[lane * ldz + k] = c * zk + s * zk1;
        Z[lane * ldz + k + 1] = -s * zk + c * zk1;
      }
      __syncwarp();
      if (k + 1 < hi) { x = nbk; z = s * f; }
    }
  }
  __syncwarp();
  // sort ascending (selection sort, swap columns of Z)
  for (int i = 0; i < n - 1; ++i) {
    int kmin = i;
    double vmin = d[i];
    for (int j = i + 1; j < n; ++j)
      if (d[j] < vmin) { vmin = d[j]; kmin = j; }
    if (kmin != i) {
      __syncwarp();
      double di = d[i];
      if (VECTORS && lane < n) {
        double t = Z[lane * ldz + i];
        Z[lane * ldz + i] = Z[lane * ldz + kmin];
        Z[lane * ldz + kmin] = t;
      }
      if (lane == 0) { d[kmin] = di; d[i] = vmin; }
      __syncwarp();
    }
  }
  return true;
}

// Rotation (c, s) that zeroes the (p, q) entry of the symmetric 2 x 2 block
// [[app, apq], [apq, aqq]] (Rutishauser's formulas).  Where |theta| >= 2^64 its
// square overflows and the formulas give t = 0 with theta's sign, c = 1: those
// lanes divide ones instead, because quotients with such operands leave the
// fast path of the division for the whole warp (late in a sweep most warps
// have such a pair).
__device__ __forceinline__ void jacobi_rot(float app, float aqq, float apq, float& c, float& sn) {
  c = 1.0f;
  sn = 0.0f;
  if (apq != 0.0f) {
    float d = aqq - app, e = 2.0f * apq;
    const bool big = fabsf(d) >= 0x1p64f * fabsf(e);
    const float sgn = copysignf(1.0f, e) * d;      // theta's sign
    if (big) { d = 1.0f; e = 1.0f; }
    const float theta = d / e;
    float t = 1.0f / (fabsf(theta) + sqrtf(theta * theta + 1.0f));
    t = copysignf(big ? 0.0f : t, big ? sgn : theta);
    c = rsqrtf(t * t + 1.0f);
    sn = t * c;
  }
}

// a x - b y and a x + b y with the second product rounded (the choice is spelt
// out so that the result does not depend on the code around it).
__device__ __forceinline__ float rot_sub(float a, float x, float b, float y) {
  return __fmaf_rn(a, x, -__fmul_rn(b, y));
}
__device__ __forceinline__ float rot_add(float a, float x, float b, float y) {
  return __fmaf_rn(a, x, __fmul_rn(b, y));
}

// Pair i (0 <= i < M/2) of rounds r = 0, 1, ... of the round-robin ("chess
// tournament") order, p < q: index 0 stays, 1..M-1 rotate.  Pair 0 of round r
// is (0, 1 + r), pair i > 0 is {1 + (r + i) mod (M-1), 1 + (r - i) mod (M-1)}.
template <int M>
struct JacobiPair {
  int a, b;
  bool first;
  __device__ __forceinline__ explicit JacobiPair(int i)
      : a(1 + i), b(1 + (M - 1 - i) % (M - 1)), first(i == 0) {}
  __device__ __forceinline__ int p() const { return first ? 0 : min(a, b); }
  __device__ __forceinline__ int q() const { return max(a, b); }
  __device__ __forceinline__ void next() {
    a = (a == M - 1) ? 1 : a + 1;
    b = (b == M - 1) ? 1 : b + 1;
  }
};

// Cyclic parallel Jacobi eigensolver (float) for a symmetric n x n matrix, run
// by a CTA of 8 warps at order M (32 or 16; indices >= n
// are padding that couples to nothing): M/2 disjoint rotations per round in
// round-robin order, sweeps until the off-diagonal Frobenius norm is below
// 4 eps ||A||_F.
// One CTA barrier per round: A is double-buffered (a round reads one buffer
// and writes the other), and every warp forms the round's M/2 rotations itself
// (lane l: pair l mod M/2, which is also the column pair of its block).  Thread
// (I, J) maps the 2 x 2 block of pairs (I, J) through the row rotation of I
// and the column rotation of J (the pairs are disjoint, so the block depends
// only on itself).  The eigenvectors are kept transposed (row p of Z is vector
// p): a warp rotates those of its own row pairs, conflict-free.  A round is
// bound by the rotation's chain of two divisions and two roots (about 310
// cycles) and by instruction issue: everything that does not depend on the
// rotation is loaded before it, and the indices and rotations of the row pairs
// come by shuffle from the lanes that hold them.
// A and A2 (row-major, lda >= M, each with room for 2 lda + n M floats) are
// destroyed; w receives the eigenvalues ascending, Z (row-major, ldz >= M) the
// eigenvectors as columns.  Returns false (uniformly) if 20 sweeps do not
// converge.  red needs 2 floats.
template <int M>
__device__ inline bool cta_jacobi_f32(float* A, float* A2, int lda, int n, float* w, float* Z,
                                      int ldz, float* red) {
  static_assert(M == 16 || M == 32, "order 16 or 32");
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
  constexpr int H = M / 2;
  for (int e = tid; e < M * M; e += nt) {
    const int i = e / M, j = e % M;
    Z[i * ldz + j] = (i == j) ? 1.0f : 0.0f;
    if (i >= n || j >= n) A[i * lda + j] = 0.0f;
  }
  __syncthreads();
  if (wid == 0) {
    float fro = 0.0f;
    for (int i = 0; i < M; ++i) { const float a = (lane < M) ? A[i * lda + lane] : 0.0f; fro += a * a; }
    fro = warp_sum(fro);
    if (lane == 0) red[0] = fro * (4.0f * 1.2e-7f) * (4.0f * 1.2e-7f);
  }
  float* cur = A;
  float* nxt = A2;
  bool ok = false;
  const int I = ((32 / H) * wid + lane / H) % H;
  const int z0 = ((32 / H) * wid + lane / M) % H, z1 = (z0 + 32 / M) % H, zr = lane % M;
  const bool own = tid < H * H;          // whole warps
  JacobiPair<M> pj(lane % H);
  __syncthreads();
  const float tol2 = red[0];
  for (int sweep = 0; sweep < 20; ++sweep) {
    if (wid == 0) {
      float off = 0.0f;
      for (int i = 0; i < M; ++i) {
        const float a = (lane < M && lane != i) ? cur[i * lda + lane] : 0.0f;
        off += a * a;
      }
      off = warp_sum(off);
      if (lane == 0) red[1] = off;
    }
    __syncthreads();
    if (red[1] <= tol2) { ok = true; break; }
    for (int r = 0; r < M - 1; ++r) {
      if (own) {
        const int p2 = pj.p(), q2 = pj.q(), pq = p2 | (q2 << 16);
        const float* dp = cur + p2 * lda;
        const float dpp = dp[p2], dpq = dp[q2], dqq = cur[q2 * lda + q2];
        const int w0 = __shfl_sync(0xffffffffu, pq, z0), w1 = __shfl_sync(0xffffffffu, pq, z1);
        int wi;
        if constexpr (M == 32) wi = (lane < 16) ? w0 : w1;
        else wi = __shfl_sync(0xffffffffu, pq, I);
        const int p = (wi & 0xffff) * lda, q = (wi >> 16) * lda;
        const float app = cur[p + p2], apq = cur[p + q2];
        const float aqp = cur[q + p2], aqq = cur[q + q2];
        float* zp0 = Z + (w0 & 0xffff) * ldz + zr;
        float* zq0 = Z + (w0 >> 16) * ldz + zr;
        float* zp1 = Z + (w1 & 0xffff) * ldz + zr;
        float* zq1 = Z + (w1 >> 16) * ldz + zr;
        const float vp0 = *zp0, vq0 = *zq0, vp1 = *zp1, vq1 = *zq1;
        float c2, s2;
        jacobi_rot(dpp, dqq, dpq, c2, s2);
        const float c0 = __shfl_sync(0xffffffffu, c2, z0), s0 = __shfl_sync(0xffffffffu, s2, z0);
        const float c1 = __shfl_sync(0xffffffffu, c2, z1), s1 = __shfl_sync(0xffffffffu, s2, z1);
        float c, sn;
        if constexpr (M == 32) {
          c = (lane < 16) ? c0 : c1;
          sn = (lane < 16) ? s0 : s1;
        } else {
          c = __shfl_sync(0xffffffffu, c2, I);
          sn = __shfl_sync(0xffffffffu, s2, I);
        }
        // rows
        const float bpp = rot_sub(c, app, sn, aqp), bpq = rot_sub(c, apq, sn, aqq);
        const float bqp = rot_add(sn, app, c, aqp), bqq = rot_add(sn, apq, c, aqq);
        // columns
        nxt[p + p2] = rot_sub(c2, bpp, s2, bpq);
        nxt[p + q2] = rot_add(s2, bpp, c2, bpq);
        nxt[q + p2] = rot_sub(c2, bqp, s2, bqq);
        nxt[q + q2] = rot_add(s2, bqp, c2, bqq);
        *zp0 = rot_sub(c0, vp0, s0, vq0);
        *zq0 = rot_add(s0, vp0, c0, vq0);
        *zp1 = rot_sub(c1, vp1, s1, vq1);
        *zq1 = rot_add(s1, vp1, c1, vq1);
        pj.next();
      }
      __syncthreads();
      float* t = cur;
      cur = nxt;
      nxt = t;
    }
  }
  // eigenvalues from the diagonal, sorted ascending with their vectors: each
  // value's rank (ties by index) is its position; the spare buffer's first
  // row holds the values, its second the ranks, the rest the old Z
  float* wv = nxt;
  int* rk = (int*)(nxt + lda);
  if (tid < M) wv[tid] = (tid < n) ? cur[tid * lda + tid] : 0.0f;
  __syncthreads();
  if (tid < n) {
    const float v = wv[tid];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const float u = wv[j];
      r += (u < v || (u == v && j < tid)) ? 1 : 0;
    }
    rk[tid] = r;
    w[r] = v;
  }
  __syncthreads();
  // the vectors in their order, as columns: Z[:, rank[c]] = vector c
  float* zs = nxt + 2 * lda;   // n x n, stride M
  for (int e = tid; e < n * n; e += nt) {
    const int c = e / n, i = e - (e / n) * n;
    zs[c * M + i] = Z[c * ldz + i];
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, c = e - (e / n) * n;
    Z[i * ldz + rk[c]] = zs[c * M + i];
  }
  __syncthreads();
  return ok;
}

// 2 (sqrt(sum sa) + sqrt(sum aa) sqrt(sum rr)) over the CTA's threads, of which
// those at or past `count` hold zeros.  The sums are block_sum's (warps in
// order; warps of zeros add nothing), but only warps with values take part, the
// three run on three lanes, and so do the square roots: as three block_sums by
// every thread they took the SM's FP64 unit 8k cycles.
__device__ __forceinline__ double cta_refine_delta(double sa, double aa, double rr, int count) {
  __shared__ double part[3][32], out;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = min((int)(blockDim.x >> 5), (count + 31) / 32);
  if (wid < nw) {
    sa = warp_sum(sa);
    aa = warp_sum(aa);
    rr = warp_sum(rr);
    if (lane == 0) { part[0][wid] = sa; part[1][wid] = aa; part[2][wid] = rr; }
  }
  __syncthreads();
  if (wid == 0) {
    double s = 0.0;
    if (lane < 3)
      for (int w = 0; w < nw; ++w) s += part[lane][w];
    s = sqrt(s);
    const double r1 = __shfl_sync(0xffffffffu, s, 1), r2 = __shfl_sync(0xffffffffu, s, 2);
    if (lane == 0) out = 2.0 * (s + r1 * r2);
  }
  __syncthreads();
  return out;
}

// One step of the iterative refinement of a symmetric eigen-decomposition of
// Ogita & Aishima ("Iterative refinement for symmetric eigenvalue
// decomposition", Japan J. Indust. Appl. Math. 35, 2018), FP64, whole CTA.
//   R = I - X^T X,  S = X^T A X,  lam_i = S_ii / (1 - R_ii),
//   E_ij = (S_ij + lam_j R_ij) / (lam_j - lam_i)  if |lam_i - lam_j| > delta,
//          R_ij / 2                                 otherwise,
//   X <- X + X E.
// A, X, R, S, W: n x n row-major with leading dimension ld (shared memory);
// A is multiplied as a dense matrix.  lam receives the refined eigenvalues.
__device__ inline void cta_refine_eig(const double* A, double* X, double* R, double* S,
                                      double* W, double* lam, int n, int ld) {
  const int tid = threadIdx.x, nt = blockDim.x;
  // W = A X
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    double v = 0.0;
    for (int l = 0; l < n; ++l) {
      const double a = A[i * ld + l];
      if (a != 0.0) v += a * X[l * ld + j];
    }
    W[i * ld + j] = v;
  }
  __syncthreads();
  // R = I - X^T X,  S = X^T W
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    double r = 0.0, s = 0.0;
    for (int l = 0; l < n; ++l) {
      r += X[l * ld + i] * X[l * ld + j];
      s += X[l * ld + i] * W[l * ld + j];
    }
    R[i * ld + j] = ((i == j) ? 1.0 : 0.0) - r;
    S[i * ld + j] = s;
  }
  __syncthreads();
  if (tid < n) lam[tid] = S[tid * ld + tid] / (1.0 - R[tid * ld + tid]);
  __syncthreads();
  // delta = 2 (||S - diag(lam)||_F + ||A||_F ||R||_F)
  double sa = 0.0, aa = 0.0, rr = 0.0;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    const double d = S[i * ld + j] - ((i == j) ? lam[i] : 0.0);
    sa += d * d;
    aa += A[i * ld + j] * A[i * ld + j];
    rr += R[i * ld + j] * R[i * ld + j];
  }
  const double delta = cta_refine_delta(sa, aa, rr, n * n);
  // E into W
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    const double dl = lam[j] - lam[i];
    W[i * ld + j] = (fabs(dl) > delta) ? (S[i * ld + j] + lam[j] * R[i * ld + j]) / dl
                                       : 0.5 * R[i * ld + j];
  }
  __syncthreads();
  // X <- X + X E   (result into S, then copied back)
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    double v = 0.0;
    for (int l = 0; l < n; ++l) v += X[i * ld + l] * W[l * ld + j];
    S[i * ld + j] = X[i * ld + j] + v;
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    X[i * ld + j] = S[i * ld + j];
  }
  __syncthreads();
}

}  // namespace usbs
