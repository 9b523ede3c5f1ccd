// Thick-restart Lanczos (smallest eigenpairs) as one cooperative launch.
//
// Reference: solver/lanczos.py:80-236 (restart loop, CGS2 full
// reorthogonalisation, arrowhead projected matrix, gap-ratio restart choice).
//
// Layout and schedule.  The CTAs of the launch are split into teams, one team
// per problem.  A team owns a contiguous range of 256-row tiles of its problem;
// every phase below walks the same tiles, so a CTA only ever reads and writes
// its own rows of Q and of the work vectors, except for the SpMV gathers of x
// (read through L2 with ld.global.cg after a team barrier).  One Lanczos step i
// is three phases separated by team barriers:
//   A  y = Op x  (CSR, `lanes` threads per row) fused with h1 = Q[:, :i+1]^T y
//   B  q1 = y - Q h1, fused with h2 = Q^T q1
//   C  q2 = q1 - Q h2, fused with ||q2||^2
// The normalisation q2 / beta is folded into the next phase A (x = v * 1/beta),
// which also stores Q[:, i+1] for its rows.  Partial sums go to a per-team
// [pass][cta][column] buffer and every CTA reduces them in the same fixed order,
// so all CTAs hold bit-identical alpha/beta and take identical branches.
// At a restart CTA 0 builds the arrowhead matrix and runs the FP64 warp
// eigensolver; after a barrier every CTA rotates its rows of Q by the saved
// Ritz vectors.
#include <stdlib.h>
#include <map>
#include <mutex>
#include "common.cuh"
#include "dense.cuh"
#include "internal.h"

namespace usbs {

constexpr int LZ_BLOCK = 256;
constexpr int LZ_NW = LZ_BLOCK / 32;
constexpr int MAX_TEAMS = 48;
constexpr int MP1 = MAXM + 1;

constexpr int LZ_XS_BYTES = 160 * 1024;   // dynamic shared memory for a staged x

struct StreamCtl;

template <typename VT>
struct TeamDesc {
  int n, ld, m, num_desired, max_restarts, lanes, first_cta, nctas, xsmem;
  int ldv;               // stride of vbuf's vectors: n rounded up to 32, whatever ld is
  long long nnz;
  double tol;
  const int* rowptr;
  const int* col;
  const VT* val;
  VT* Q;                 // the caller's basis, ld x (m+1) column-major
  // working basis: element (c, row) at Qw[qix(c, row)] (here always Q:
  // tile stride LZ_BLOCK, column stride ld)
  VT* Qw;
  long long qts, qcs;    // tile and column strides (elements)
  // stream path: the operator in a sliced-ELL layout built on the device (rows
  // of each 256-row window sorted by length, 32-row slices, each slice
  // holding at most wcap entries per row; longer rows finish from the CSR)
  int wcap;
  int* sl_ptr;           // slice s: entries [sl_ptr[s], sl_ptr[s + 1]), column-major
  unsigned char* sl_row; // sorted position -> row offset inside its window
  int* sl_col;
  VT* sl_val;
  VT* vbuf;              // 3 flat vectors: two work vectors, then Q[:, k] of the cycle
  double* part;
  double* Ybuf;
  double* alpha;
  double* beta;
  int* ctl;
  unsigned int* bar;
  int* status;
  StreamCtl* resume;     // wave path: the loop state the team kernel continues from (else null)
};

// Loop state of the stream and wave paths (see there).
struct __align__(16) StreamCtl {
  int i, k, bd, cur;           // step, saved vectors, breakdown pending, work vector in use
  int stop, rot, stepped;      // ST_RUN, ...; rotation pending; the finished cycle had steps
  int restarts, breakdowns, steps, sum_nv, sum_kn, nconv;
  unsigned ticket[3];          // last-CTA tickets of B, C and the rotation
  unsigned dticket[4];         // of A2's column groups
  int breakdowns0, steps0, sum_nv0;   // the counters at the cycle's start
  double invb;                 // 1 / beta of the latest unnormalised vector
  double h1[MP1], h2[MP1];
  double alpha[MAXM], beta[MAXM];
  unsigned long long cyc[4];   // wave path: cycles of CTA 0 in the reductions and phases A, B, C
};
// stop: the loop runs; has ended; (wave path) goes on in the team kernel
enum { ST_RUN = 0, ST_ENDED = 1, ST_HANDED = 2 };

template <typename VT>
__device__ __forceinline__ size_t qix(const TeamDesc<VT>& P, int c, int row) {
  return (size_t)(row / LZ_BLOCK) * (size_t)P.qts + (size_t)c * (size_t)P.qcs +
         (size_t)(row % LZ_BLOCK);
}

template <typename VT>
struct TeamBatch {
  int count;
  TeamDesc<VT> t[MAX_TEAMS];
};

template <typename VT>
struct LzShared {
  union {
    struct {                     // Lanczos step phases
      double ys[LZ_BLOCK];
      double wred[LZ_NW][MP1];
    } st;
    struct {                     // restart on CTA 0 (T, X, R, S, W row-major, ld MP1)
      double T[MAXM * MP1];
      double X[MAXM * MP1];
      double R[MAXM * MP1];      // float copy of T during the Jacobi sweeps
      double S[MAXM * MP1];      // float eigenvectors during the Jacobi sweeps
      double W[MAXM * MP1];
    } rs;
    VT Ys[MAXM * MAXM];          // saved Ritz vectors, every CTA, after the restart barrier
    double red4[4][MP1];         // cluster reduction: the four level-two sums
  } u;
  double h[MP1];
  double bnorm;                  // cluster kernel: sqrt(h[0]) of a norm reduction ...
  VT hv[MP1];                    // h in the vector type, converted once per reduction (16-byte aligned)
  VT binv;                       // ... and 1 / bnorm in the vector type
  double alpha[MAXM];
  double beta[MAXM];
  double ritz[MAXM];
  double red[LZ_NW];
  float wf[MAXM], redf[32];
  int order[MAXM];
  int k_next, nconv;
  long long eig_cycles;          // cycles in the projected eigensolver (thread 0)
};

// acc[c] (c < nv) summed over the CTA, written to out[c * R] (column-major
// [column][cta] partial layout, so the team reduction reads each column in one
// coalesced load).  Columns 0..31 are reduced across each warp by one
// butterfly reduce-scatter (lane c ends with column c), column 32 by a warp sum.
template <typename SH, typename AT>
__device__ __forceinline__ void block_reduce_cols(AT* acc, int nv, SH& sh, double* out,
                                                  int R) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (nv == 1) {
    const AT v = warp_sum(acc[0]);
    if (lane == 0) sh.u.st.wred[wid][0] = (double)v;
  } else {
    const AT extra = (nv > 32) ? warp_sum(acc[32]) : (AT)0;
    const AT v = warp_reduce_scatter32(acc);
    sh.u.st.wred[wid][lane] = (double)v;
    if (lane == 0 && nv > 32) sh.u.st.wred[wid][32] = (double)extra;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < nv; c += LZ_BLOCK) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < LZ_NW; ++w) s += sh.u.st.wred[w][c];
    out[(size_t)c * R] = s;
  }
}

// h[c] = sum over the team's CTAs of part_pass[c][r], identical order in every
// CTA.  Warp 0 issues all loads (lane l takes CTAs l, l+32, ...), then one
// butterfly reduce-scatter leaves column c in lane c.
template <typename VT>
__device__ __forceinline__ void reduce_part(const double* part_pass, int R, int nv,
                                            LzShared<VT>& sh) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    if (nv == 1) {
      double a = 0.0;
      for (int r = lane; r < R; r += 32) a += __ldcg(part_pass + r);
      a = warp_sum(a);
      if (lane == 0) { sh.h[0] = a; sh.hv[0] = (VT)a; }
    } else {
      double acc[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) acc[c] = 0.0;
      double extra = 0.0;
      for (int r = lane; r < R; r += 32) {
#pragma unroll
        for (int c = 0; c < 32; ++c)
          if (c < nv) acc[c] += __ldcg(part_pass + (size_t)c * R + r);
        if (nv > 32) extra += __ldcg(part_pass + (size_t)32 * R + r);
      }
      extra = warp_sum(extra);
      const double v = warp_reduce_scatter32(acc);
      if (lane < nv) { sh.h[lane] = v; sh.hv[lane] = (VT)v; }
      if (lane == 0 && nv > 32) { sh.h[32] = extra; sh.hv[32] = (VT)extra; }
    }
  }
  __syncthreads();
}

// SpMV of one 256-row tile, L lanes per row: sh.u.st.ys[r] = (Op x)[base + r].
// Groups of up to 4 passes issue their rowptr loads, then their first col/val
// loads, before any result is used: two dependent L2 round trips per group
// instead of two per pass.
template <typename VT, int L, typename SH>
__device__ __forceinline__ void spmv_tile(const TeamDesc<VT>& P, SH& sh, int base,
                                          const VT* xsrc, const VT* xs, bool use_xs) {
  typedef typename Acc<VT>::type AT;
  constexpr int GPP = LZ_BLOCK / L;
  constexpr int CH = L < 4 ? L : 4;          // passes whose loads are issued together
  const int tid = threadIdx.x, g = tid / L, lig = tid - (tid / L) * L;
#pragma unroll 1
  for (int q0 = 0; q0 < L; q0 += CH) {
    int pb[CH], pe[CH];
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      const int row = base + (q0 + q) * GPP + g;
      pb[q] = 0; pe[q] = 0;
      if (row < P.n) { pb[q] = P.rowptr[row] + lig; pe[q] = P.rowptr[row + 1]; }
    }
    int c0[CH];
    VT v0[CH];
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      c0[q] = 0; v0[q] = (VT)0;
      if (pb[q] < pe[q]) { c0[q] = P.col[pb[q]]; v0[q] = P.val[pb[q]]; }
    }
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      AT s = (AT)v0[q] * (AT)(use_xs ? xs[c0[q]] : __ldcg(xsrc + c0[q]));
      for (int p = pb[q] + L; p < pe[q]; p += L)
        s += (AT)P.val[p] * (AT)(use_xs ? xs[P.col[p]] : __ldcg(xsrc + P.col[p]));
#pragma unroll
      for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lig == 0) sh.u.st.ys[(q0 + q) * GPP + g] = (double)s;
    }
  }
}

// Phase A: y = Op (xsrc * xscale) for own rows -> vout, acc[c] = Q[:, c] . y (c <= i).
// If wq, also stores Q[:, i] = xsrc * xscale for own rows.
template <typename VT>
__device__ void phase_spmv(const TeamDesc<VT>& P, LzShared<VT>& sh, int t0, int t1, int i,
                           const VT* xsrc, VT xscale, bool wq, VT* vout, double* part_out) {
  typedef typename Acc<VT>::type AT;
  AT acc[MP1];
#pragma unroll
  for (int c = 0; c < MP1; ++c) acc[c] = (AT)0;
  const int tid = threadIdx.x, L = P.lanes, gpp = LZ_BLOCK / L;
  const int g = tid / L, lig = tid - g * L;
  const size_t ld = (size_t)P.ld;
  // small vectors: stage x once in shared memory so the gathers skip L2
  extern __shared__ __align__(16) unsigned char lz_dyn[];
  VT* xs = (VT*)lz_dyn;
  const bool use_xs = P.xsmem != 0;
  if (use_xs) {
    // 16-byte loads, several in flight per thread (xsrc is one of vbuf's vectors,
    // 128-byte aligned)
    constexpr int VE = 16 / (int)sizeof(VT);
    const int n16 = P.n / VE;
    const uint4* src = (const uint4*)xsrc;
    uint4* dst = (uint4*)xs;
    int j = tid;
    for (; j + 3 * LZ_BLOCK < n16; j += 4 * LZ_BLOCK) {
      const uint4 a = __ldcg(src + j), b = __ldcg(src + j + LZ_BLOCK),
                  c = __ldcg(src + j + 2 * LZ_BLOCK), d = __ldcg(src + j + 3 * LZ_BLOCK);
      dst[j] = a; dst[j + LZ_BLOCK] = b; dst[j + 2 * LZ_BLOCK] = c; dst[j + 3 * LZ_BLOCK] = d;
    }
    for (; j < n16; j += LZ_BLOCK) dst[j] = __ldcg(src + j);
    for (int r = n16 * VE + tid; r < P.n; r += LZ_BLOCK) xs[r] = __ldcg(xsrc + r);
    __syncthreads();
  }
  (void)gpp; (void)g; (void)lig;
  for (int tile = t0; tile < t1; ++tile) {
    const int base = tile * LZ_BLOCK;
    switch (L) {
      case 1: spmv_tile<VT, 1>(P, sh, base, xsrc, xs, use_xs); break;
      case 2: spmv_tile<VT, 2>(P, sh, base, xsrc, xs, use_xs); break;
      case 4: spmv_tile<VT, 4>(P, sh, base, xsrc, xs, use_xs); break;
      case 8: spmv_tile<VT, 8>(P, sh, base, xsrc, xs, use_xs); break;
      case 16: spmv_tile<VT, 16>(P, sh, base, xsrc, xs, use_xs); break;
      default: spmv_tile<VT, 32>(P, sh, base, xsrc, xs, use_xs); break;
    }
    __syncthreads();
    const int row = base + tid;
    if (row < P.n) {
      const VT y = (VT)sh.u.st.ys[tid] * xscale;
      vout[row] = y;
      VT xn = (VT)0;
      if (wq) {
        xn = __ldcg(xsrc + row) * xscale;
        P.Qw[qix(P, i, row)] = xn;
      }
#pragma unroll
      for (int c = 0; c < MP1; ++c) {
        if (c <= i) {
          const VT qc = (wq && c == i) ? xn : P.Qw[qix(P, c, row)];
          acc[c] += (AT)qc * (AT)y;
        }
      }
    }
    __syncthreads();
  }
  block_reduce_cols(acc, i + 1, sh, part_out, P.nctas);
}

// Breakdown pass a: buf = hash_normal(key) for own rows, acc[c] = Q[:, c] . buf (c < nv)
template <typename VT, typename SH>
__device__ void phase_random(const TeamDesc<VT>& P, SH& sh, int t0, int t1, int nv,
                             uint64_t key, VT* buf, double* part_out) {
  typedef typename Acc<VT>::type AT;
  AT acc[MP1];
#pragma unroll
  for (int c = 0; c < MP1; ++c) acc[c] = (AT)0;
  const size_t ld = (size_t)P.ld;
  for (int tile = t0; tile < t1; ++tile) {
    const int row = tile * LZ_BLOCK + threadIdx.x;
    if (row < P.n) {
      const VT r = (VT)hash_normal(key, (uint64_t)row);
      buf[row] = r;
#pragma unroll
      for (int c = 0; c < MP1; ++c)
        if (c < nv) acc[c] += (AT)P.Qw[qix(P, c, row)] * (AT)r;
    }
  }
  block_reduce_cols(acc, nv, sh, part_out, P.nctas);
}

// Phase B: buf -= Q h (c < nv); acc[c] = Q[:, c] . buf
template <typename VT, typename SH>
__device__ void phase_update_dot(const TeamDesc<VT>& P, SH& sh, int t0, int t1, int nv,
                                 VT* buf, double* part_out) {
  typedef typename Acc<VT>::type AT;
  AT acc[MP1];
#pragma unroll
  for (int c = 0; c < MP1; ++c) acc[c] = (AT)0;
  const size_t ld = (size_t)P.ld;
  for (int tile = t0; tile < t1; ++tile) {
    const int row = tile * LZ_BLOCK + threadIdx.x;
    if (row < P.n) {
      VT qr[MP1];
      VT s = (VT)0;
#pragma unroll
      for (int c = 0; c < MP1; ++c) {
        if (c < nv) {
          qr[c] = P.Qw[qix(P, c, row)];
          s += qr[c] * sh.hv[c];
        }
      }
      const VT q1 = buf[row] - s;
      buf[row] = q1;
#pragma unroll
      for (int c = 0; c < MP1; ++c)
        if (c < nv) acc[c] += (AT)qr[c] * (AT)q1;
    }
  }
  block_reduce_cols(acc, nv, sh, part_out, P.nctas);
}

// Phase C: buf -= Q h (c < nv); part_out[0] = sum buf^2 over own rows
template <typename VT, typename SH>
__device__ void phase_update_norm(const TeamDesc<VT>& P, SH& sh, int t0, int t1, int nv,
                                  VT* buf, double* part_out) {
  typedef typename Acc<VT>::type AT;
  AT nrm = (AT)0;
  const size_t ld = (size_t)P.ld;
  for (int tile = t0; tile < t1; ++tile) {
    const int row = tile * LZ_BLOCK + threadIdx.x;
    if (row < P.n) {
      VT s = (VT)0;
#pragma unroll
      for (int c = 0; c < MP1; ++c)
        if (c < nv) s += P.Qw[qix(P, c, row)] * sh.hv[c];
      const VT q2 = buf[row] - s;
      buf[row] = q2;
      nrm += (AT)q2 * (AT)q2;
    }
  }
  AT one[MP1];
  one[0] = nrm;
  block_reduce_cols(one, 1, sh, part_out, P.nctas);
}

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(const void* p, unsigned rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// Reads of a peer's (or the own) shared memory written before the last cluster
// barrier.  volatile keeps them after that barrier and in order among
// themselves; without a memory clobber plain loads may be issued around them.
__device__ __forceinline__ float cl_ld(uint32_t a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ double cl_ld(uint32_t a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void cl_st(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// M[i][j] = v in every CTA's copy of M (the CTAs' shared memory is laid out alike)
__device__ __forceinline__ void cl_share(double* p, int C, double v) {
  for (int r = 0; r < C; ++r) cl_st(cl_map(p, r), v);
}

// cta_refine_eig (dense.cuh) with its four n x n products and the quotients E
// dealt out over the C CTAs of the cluster, which all hold the same A, X and
// lam: each CTA forms n^2 / C entries, as cta_refine_eig forms them, and writes
// them to every CTA.  The products are 4 n^3 FP64 FMAs at 2 per clock and SM:
// done by every CTA redundantly they took 170k cycles per step (n = 32).
__device__ inline void cl_refine_eig(const double* A, double* X, double* R, double* S, double* W,
                                     double* lam, int n, int ld, int rank, int C) {
  const int tid = threadIdx.x, nt = blockDim.x, nn = n * n;
  const int e0 = nn * rank / C, e1 = nn * (rank + 1) / C;
  // W = A X
  for (int e = e0 + tid; e < e1; e += nt) {
    const int i = e / n, j = e - i * n;
    double v = 0.0;
    for (int l = 0; l < n; ++l) {
      const double a = A[i * ld + l];
      if (a != 0.0) v += a * X[l * ld + j];
    }
    cl_share(W + i * ld + j, C, v);
  }
  cl_sync();
  // R = I - X^T X and S = X^T W, one of the two per thread
  for (int e = 2 * e0 + tid; e < 2 * e1; e += nt) {
    const bool second = e >= e0 + e1;
    const int f = second ? e - e1 : e - e0;
    const int i = f / n, j = f - i * n;
    const double* B = second ? W : X;
    double r = 0.0;
    for (int l = 0; l < n; ++l) r += X[l * ld + i] * B[l * ld + j];
    if (second) cl_share(S + i * ld + j, C, r);
    else cl_share(R + i * ld + j, C, ((i == j) ? 1.0 : 0.0) - r);
  }
  cl_sync();
  if (tid < n) lam[tid] = S[tid * ld + tid] / (1.0 - R[tid * ld + tid]);
  __syncthreads();
  // delta = 2 (||S - diag(lam)||_F + ||A||_F ||R||_F)
  double sa = 0.0, aa = 0.0, rr = 0.0;
  for (int e = tid; e < nn; e += nt) {
    const int i = e / n, j = e - i * n;
    const double d = S[i * ld + j] - ((i == j) ? lam[i] : 0.0);
    sa += d * d;
    aa += A[i * ld + j] * A[i * ld + j];
    rr += R[i * ld + j] * R[i * ld + j];
  }
  const double delta = cta_refine_delta(sa, aa, rr, nn);
  // E into W (every CTA is past its last read of the old W)
  for (int e = e0 + tid; e < e1; e += nt) {
    const int i = e / n, j = e - i * n;
    const double dl = lam[j] - lam[i];
    cl_share(W + i * ld + j, C,
             (fabs(dl) > delta) ? (S[i * ld + j] + lam[j] * R[i * ld + j]) / dl
                                : 0.5 * R[i * ld + j]);
  }
  cl_sync();
  // X <- X + X E   (result into S, then copied back)
  for (int e = e0 + tid; e < e1; e += nt) {
    const int i = e / n, j = e - i * n;
    double v = 0.0;
    for (int l = 0; l < n; ++l) v += X[i * ld + l] * W[l * ld + j];
    cl_share(S + i * ld + j, C, X[i * ld + j] + v);
  }
  cl_sync();
  for (int e = tid; e < nn; e += nt) {
    const int i = e / n, j = e - i * n;
    X[i * ld + j] = S[i * ld + j];
  }
  __syncthreads();
}

// Key whose unsigned order is the order of finite or infinite doubles (-0 = +0).
__device__ __forceinline__ unsigned long long order_key(double x) {
  const long long b = __double_as_longlong(x == 0.0 ? 0.0 : x);
  return (unsigned long long)b ^ (b < 0 ? ~0ull : 0x8000000000000000ull);
}

// order[] = the positions a selection sort of v[0..m-1] (ascending, the first of
// equal values at each step, by swaps) ends with.  Warp 0, lane p at position p,
// integer keys: the comparisons stay off the FP64 pipe, where one thread's
// loop of them took tens of thousands of cycles.  NaNs take the plain loop.
__device__ __forceinline__ void select_order(const double* v, int m, int* order) {
  const int lane = threadIdx.x;
  if (lane >= 32) return;
  const bool in = lane < m;
  if (__any_sync(0xffffffffu, in && isnan(v[in ? lane : 0]))) {
    if (lane == 0) {
      for (int i = 0; i < m; ++i) order[i] = i;
      for (int i = 0; i < m - 1; ++i) {
        int kmin = i;
        for (int j = i + 1; j < m; ++j)
          if (v[order[j]] < v[order[kmin]]) kmin = j;
        const int t = order[i]; order[i] = order[kmin]; order[kmin] = t;
      }
    }
    return;
  }
  const unsigned long long key = in ? order_key(v[lane]) : ~0ull;
  unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  int idx = lane;
  for (int i = 0; i < m - 1; ++i) {
    const bool c = in && lane >= i;
    const unsigned mhi = __reduce_min_sync(0xffffffffu, c ? hi : 0xffffffffu);
    const bool th = c && hi == mhi;
    const unsigned mlo = __reduce_min_sync(0xffffffffu, th ? lo : 0xffffffffu);
    const int k = __ffs(__ballot_sync(0xffffffffu, th && lo == mlo)) - 1;
    const int src = (lane == i) ? k : (lane == k) ? i : lane;
    hi = __shfl_sync(0xffffffffu, hi, src);
    lo = __shfl_sync(0xffffffffu, lo, src);
    idx = __shfl_sync(0xffffffffu, idx, src);
  }
  if (in) order[lane] = idx;
}

// CTA 0 of a team: projected eigenproblem and thick-restart selection
// (solver/lanczos.py:128-168, 202-221).  k = number of saved vectors of the
// finished cycle, beta_last = beta[m-1].
// LOCAL_YS: every CTA of a cluster (rank of C) runs this on identical inputs to
// identical results (the FP64 refinement's products shared out) and keeps the saved Ritz vectors in sh.u.Ys; only the CTA
// with write_out set stores alpha/beta/ctl.  Otherwise (team kernel) the Ritz
// vectors go through P.Ybuf.
template <bool LOCAL_YS, typename VT, typename D>
__device__ void restart_select(const D& P, LzShared<VT>& sh, int k, bool write_out = true,
                               int rank = 0, int C = 1) {
  const int m = P.m, tid = threadIdx.x;
  double* T = sh.u.rs.T;
  double* X = sh.u.rs.X;
  float* Tf = (float*)sh.u.rs.R;
  float* Zf = (float*)sh.u.rs.S;
  for (int e = tid; e < m * m; e += LZ_BLOCK) {
    const int r = e / m, c = e - r * m;
    double v = 0.0;
    if (r == c) v = sh.alpha[r];
    else if (c == k && r < k) v = sh.beta[r];
    else if (r == k && c < k) v = sh.beta[c];
    else if (c == r + 1 && r >= k) v = sh.beta[r];
    else if (r == c + 1 && c >= k) v = sh.beta[c];
    T[r * MP1 + c] = v;
    Tf[r * MP1 + c] = (float)v;
  }
  __syncthreads();
  // eigh(T) (solver/lanczos.py:203): FP32 parallel Jacobi by the CTA ...
  {
    const long long c0 = clock64();
    const bool ok = cta_jacobi_f32<32>(Tf, (float*)sh.u.rs.W, MP1, m, sh.wf, Zf, MP1, sh.redf);
    if (tid == 0) sh.eig_cycles += clock64() - c0;
    if (!ok && tid == 0) atomicOr(P.status, ST_SMALL_DENSE_FAIL);
  }
  for (int e = tid; e < m * m; e += LZ_BLOCK) {
    const int r = e / m, c = e - r * m;
    X[r * MP1 + c] = (double)Zf[r * MP1 + c];
  }
  if (tid < m) sh.ritz[tid] = (double)sh.wf[tid];
  __syncthreads();
  if (sizeof(VT) == 8) {
    // ... refined to FP64 accuracy by two Ogita-Aishima steps, then re-sorted
    // (a peer may still run its Jacobi sweeps in the buffers the refinement shares)
    if constexpr (LOCAL_YS) cl_sync();
    for (int it = 0; it < 2; ++it) {
      if constexpr (LOCAL_YS)
        cl_refine_eig(T, X, sh.u.rs.R, sh.u.rs.S, sh.u.rs.W, sh.ritz, m, MP1, rank, C);
      else
        cta_refine_eig(T, X, sh.u.rs.R, sh.u.rs.S, sh.u.rs.W, sh.ritz, m, MP1);
    }
    select_order(sh.ritz, m, sh.order);
    __syncthreads();
    double* Sx = sh.u.rs.S;
    for (int e = tid; e < m * m; e += LZ_BLOCK) {
      const int r = e / m, c = e - r * m;
      Sx[r * MP1 + c] = X[r * MP1 + sh.order[c]];
    }
    double rv = (tid < m) ? sh.ritz[sh.order[tid]] : 0.0;
    __syncthreads();
    for (int e = tid; e < m * m; e += LZ_BLOCK) {
      const int r = e / m, c = e - r * m;
      X[r * MP1 + c] = Sx[r * MP1 + c];
    }
    if (tid < m) sh.ritz[tid] = rv;
    __syncthreads();
  }
  const double* Z = X;
  if (tid < 32) {
    // lane c: Ritz pair c.  The residual tests, the gap ratios (one FP64
    // division each) and the finiteness test run side by side; as one thread's
    // loop they took about 25k cycles per restart.
    const int lane = tid;
    const bool in = lane < m;
    // a NaN / Inf in the projected matrix (e.g. from a non-finite operator)
    // ends the call after this restart with ST_NONFINITE
    const bool fin = !in || (isfinite(sh.alpha[lane]) && isfinite(sh.beta[lane]));
    const double bl = sh.beta[m - 1];
    const bool open = in && !(bl * fabs(Z[(m - 1) * MP1 + lane]) < P.tol);
    const unsigned ob = __ballot_sync(0xffffffffu, open);
    const int nconv = ob ? __ffs(ob) - 1 : m;
    const int delta = min(m - P.num_desired, 2 * (m - nconv) / 5);
    const double lt = sh.ritz[min(nconv, m - 1)];
    double g = 0.0;
    if (in) {
      const int kr = lane + delta;
      if (kr <= m) g = (sh.ritz[lane] - lt) / (sh.ritz[min(kr, m - 1)] - lt);
    }
    // first NaN, else the first largest ratio
    const unsigned nb = __ballot_sync(0xffffffffu, in && isnan(g));
    const unsigned long long key = order_key(g);
    const unsigned hi = in ? (unsigned)(key >> 32) : 0u, lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const bool th = in && hi == mhi;
    const unsigned mlo = __reduce_max_sync(0xffffffffu, th ? lo : 0u);
    const unsigned tb = __ballot_sync(0xffffffffu, th && lo == mlo);
    const int kl = nb ? __ffs(nb) - 1 : __ffs(tb) - 1;
    const int kright = kl + delta;
    const bool keep = in && (kl >= lane || kright < lane);
    const unsigned kb = __ballot_sync(0xffffffffu, keep);
    const unsigned below = (1u << lane) - 1u;
    const int kn = __popc(kb);
    if (in) sh.order[keep ? __popc(kb & below) : kn + lane - __popc(kb & below)] = lane;
    const bool bad = !__all_sync(0xffffffffu, fin);
    if (lane == 0) {
      if (bad) atomicOr(P.status, ST_NONFINITE);
      sh.k_next = kn;
      sh.nconv = nconv;
    }
  }
  __syncthreads();
  const int kn = sh.k_next;
  const double bl = sh.beta[m - 1];
  if constexpr (LOCAL_YS) {
    // sh.u.Ys overlays sh.u.rs.T only (T is no longer needed; Z lives in X)
    for (int e = tid; e < m * MAXM; e += LZ_BLOCK) {
      const int j = e / MAXM, c = e - j * MAXM;
      sh.u.Ys[e] = (c < kn) ? (VT)Z[j * MP1 + sh.order[c]] : (VT)0;
    }
  } else {
    for (int e = tid; e < m * m; e += LZ_BLOCK) {
      const int j = e / m, c = e - j * m;
      P.Ybuf[j * m + c] = Z[j * MP1 + sh.order[c]];
    }
  }
  __syncthreads();
  if (tid < m) {
    const int c = tid;
    const double a = (c < kn) ? sh.ritz[sh.order[c]] : 0.0;
    const double b = (c < kn) ? bl * Z[(m - 1) * MP1 + sh.order[c]] : 0.0;
    sh.alpha[c] = a;
    sh.beta[c] = b;
    if (write_out) {
      P.alpha[c] = a;
      P.beta[c] = b;
    }
  }
  if (tid == 0 && write_out) {
    P.ctl[0] = kn;
    P.ctl[1] = sh.nconv;
  }
  __syncthreads();
}

template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK, 1)
lanczos_team_kernel(const __grid_constant__ TeamBatch<VT> batch) {
  __shared__ LzShared<VT> sh;
  int team = 0;
  for (int t = 1; t < batch.count; ++t)
    if ((int)blockIdx.x >= batch.t[t].first_cta) team = t;
  const TeamDesc<VT>& P = batch.t[team];
  const int rank = (int)blockIdx.x - P.first_cta, R = P.nctas;
  const int tid = threadIdx.x;
  TeamBarrier bar{P.bar, R, P.status};
  auto team_sync = [&]() -> bool { return bar.sync(); };
  const int n = P.n, m = P.m;
  const size_t ld = (size_t)P.ld;
  const int ntiles = (n + LZ_BLOCK - 1) / LZ_BLOCK;
  const int t0 = (int)((long long)ntiles * rank / R);
  const int t1 = (int)((long long)ntiles * (rank + 1) / R);
  // [pass][column][cta] partial sums
  double* part0 = P.part;
  double* part1 = P.part + (size_t)R * MP1;
  double* part2 = P.part + (size_t)2 * R * MP1;

  int k = 0, nconv = 0, restart = 0, breakdowns = 0, steps = 0, sum_nv = 0, sum_kn = 0;
  long long clk_start = clock64(), clk_restart = 0;
  // rank-0 phase accounting: [0] barrier waits, [1] team reductions, [2..4] phases A..C
  long long tp[5] = {0, 0, 0, 0, 0}, tmark = clock64();
  const bool timing = (rank == 0 && tid == 0);
#define LZ_MARK(slot)                                   \
  do {                                                  \
    if (timing) {                                       \
      const long long _c = clock64();                   \
      tp[slot] += _c - tmark;                           \
      tmark = _c;                                       \
    }                                                   \
  } while (0)
  if (rank == 0 && tid < MAXM) { sh.alpha[tid] = 0.0; sh.beta[tid] = 0.0; }
  if (tid == 0) sh.eig_cycles = 0;
  if (const StreamCtl* rs = P.resume) {
    // after the wave path's cycles: its state at the start of a cycle, or its end
    k = rs->k; nconv = rs->nconv; restart = rs->restarts;
    breakdowns = rs->breakdowns0; steps = rs->steps0; sum_nv = rs->sum_nv0; sum_kn = rs->sum_kn;
    if (rank == 0 && tid < MAXM) { sh.alpha[tid] = rs->alpha[tid]; sh.beta[tid] = rs->beta[tid]; }
    if (timing) {
      clk_restart = (long long)P.ctl[6] << 10;
      sh.eig_cycles = (long long)P.ctl[15] << 10;
      clk_start -= clk_restart;
      for (int j = 0; j < 4; ++j) {
        tp[1 + j] = (long long)rs->cyc[j];
        clk_start -= tp[1 + j];
      }
    }
    if (rs->stop == ST_ENDED) {
      if (timing) {
        P.ctl[7] = (int)((clock64() - clk_start) >> 10);
        for (int j = 0; j < 5; ++j) P.ctl[8 + j] = (int)(tp[j] >> 10);
      }
      return;
    }
  }
  // the start vector Q[:, k]: flat copy for the first cycle's gathers
  VT* xk = P.vbuf + 2 * (size_t)P.ldv;
  for (int tile = t0; tile < t1; ++tile) {
    const int row = tile * LZ_BLOCK + tid;
    if (row < n) xk[row] = P.Q[(size_t)k * ld + row];
  }
  __syncthreads();
  if (!team_sync()) return;
  int prev = 0;          // vbuf slot holding the latest unnormalised vector
  VT invb = (VT)1;       // its normalisation
  while (nconv < P.num_desired && restart < P.max_restarts) {
    int cur = 0;
    for (int i = k; i < m; ++i) {
      const VT* xsrc;
      bool wq;
      if (i == k) {
        xsrc = xk;       // = Q[:, k]
        invb = (VT)1;
        wq = false;
      } else {
        reduce_part(part2, R, 1, sh);
        const double b = sqrt(sh.h[0]);
        if (rank == 0 && tid == 0) sh.beta[i - 1] = b;
        if (b < 1e-15) {
          // Krylov space exhausted: random vector orthogonalised twice
          // against Q[:, :i] (solver/lanczos.py:107-117)
          ++breakdowns;
          VT* buf = P.vbuf + (size_t)prev * P.ldv;
          phase_random(P, sh, t0, t1, i, (uint64_t)i, buf, part0 + rank);
          if (!team_sync()) return;
          reduce_part(part0, R, i, sh);
          phase_update_dot(P, sh, t0, t1, i, buf, part1 + rank);
          if (!team_sync()) return;
          reduce_part(part1, R, i, sh);
          phase_update_norm(P, sh, t0, t1, i, buf, part2 + rank);
          if (!team_sync()) return;
          reduce_part(part2, R, 1, sh);
          invb = (VT)(1.0 / sqrt(sh.h[0]));
        } else {
          invb = (VT)(1.0 / b);
        }
        xsrc = P.vbuf + (size_t)prev * P.ldv;
        wq = true;
      }
      VT* vout = P.vbuf + (size_t)cur * P.ldv;
      LZ_MARK(1);
      phase_spmv(P, sh, t0, t1, i, xsrc, invb, wq, vout, part0 + rank);
      LZ_MARK(2);
      if (!team_sync()) return;
      LZ_MARK(0);
      reduce_part(part0, R, i + 1, sh);
      LZ_MARK(1);
      const double h1i = sh.h[i];
      phase_update_dot(P, sh, t0, t1, i + 1, vout, part1 + rank);
      LZ_MARK(3);
      if (!team_sync()) return;
      LZ_MARK(0);
      reduce_part(part1, R, i + 1, sh);
      LZ_MARK(1);
      if (rank == 0 && tid == 0) sh.alpha[i] = h1i + sh.h[i];
      phase_update_norm(P, sh, t0, t1, i + 1, vout, part2 + rank);
      LZ_MARK(4);
      if (!team_sync()) return;
      LZ_MARK(0);
      prev = cur;
      cur ^= 1;
      ++steps;
      sum_nv += i + 1;
    }
    // ---- restart ----
    const bool stepped = (k < m);
    if (stepped) {
      reduce_part(part2, R, 1, sh);
      const double b = sqrt(sh.h[0]);
      if (rank == 0 && tid == 0) sh.beta[m - 1] = b;
      if (b < 1e-15) {
        ++breakdowns;
        VT* buf = P.vbuf + (size_t)prev * P.ldv;
        phase_random(P, sh, t0, t1, m, (uint64_t)m, buf, part0 + rank);
        if (!team_sync()) return;
        reduce_part(part0, R, m, sh);
        phase_update_dot(P, sh, t0, t1, m, buf, part1 + rank);
        if (!team_sync()) return;
        reduce_part(part1, R, m, sh);
        phase_update_norm(P, sh, t0, t1, m, buf, part2 + rank);
        if (!team_sync()) return;
        reduce_part(part2, R, 1, sh);
        invb = (VT)(1.0 / sqrt(sh.h[0]));
      } else {
        invb = (VT)(1.0 / b);
      }
    }
    __syncthreads();
    if (rank == 0) {
      const long long c0 = clock64();
      restart_select<false>(P, sh, k);
      clk_restart += clock64() - c0;
    }
    if (!team_sync()) return;
    if (__ldcg(P.status) & ST_NONFINITE) { ++restart; break; }
    const int kn = __ldcg(P.ctl + 0);
    nconv = __ldcg(P.ctl + 1);
    for (int e = tid; e < m * MAXM; e += LZ_BLOCK) {
      const int j = e / MAXM, c = e - j * MAXM;
      sh.u.Ys[e] = (c < kn) ? (VT)__ldcg(P.Ybuf + j * m + c) : (VT)0;
    }
    __syncthreads();
    const VT* lastv = P.vbuf + (size_t)prev * P.ldv;
    for (int tile = t0; tile < t1; ++tile) {
      const int row = tile * LZ_BLOCK + tid;
      if (row < n) {
        VT qr[MAXM];
#pragma unroll
        for (int j = 0; j < MAXM; ++j) qr[j] = (j < m) ? P.Qw[qix(P, j, row)] : (VT)0;
        const VT xl = stepped ? lastv[row] * invb : P.Qw[qix(P, m, row)];
        for (int c = 0; c < kn; ++c) {
          if (c >= m) break;
          VT s = (VT)0;
#pragma unroll
          for (int j = 0; j < MAXM; ++j)
            if (j < m) s += qr[j] * sh.u.Ys[j * MAXM + c];
          P.Qw[qix(P, c, row)] = s;
        }
        P.Qw[qix(P, kn, row)] = xl;
        if (kn != m) P.Qw[qix(P, m, row)] = xl;
        xk[row] = xl;
      }
    }
    k = kn;
    sum_kn += kn;
    ++restart;
    if (!team_sync()) return;
    if (timing) tmark = clock64();   // restart time is reported separately (ctl[6])
  }
  if (rank == 0 && tid == 0) {
    P.ctl[2] = restart;
    P.ctl[3] = breakdowns;
    P.ctl[4] = steps;
    P.ctl[6] = (int)(clk_restart >> 10);
    P.ctl[7] = (int)((clock64() - clk_start) >> 10);
    for (int j = 0; j < 5; ++j) P.ctl[8 + j] = (int)(tp[j] >> 10);
    P.ctl[13] = sum_nv;
    P.ctl[14] = sum_kn;
    P.ctl[15] = (int)(sh.eig_cycles >> 10);
    if (restart == 0) P.ctl[0] = 0;
  }
}

// ---------------------------------------------------------------- stream path
// Problems whose x does not fit in shared memory (n * sizeof(VT) > 160 KB) run
// as a sequence of ordinary full-GPU launches instead of one cooperative
// launch: every Lanczos step is
//   A1  y = Op x for one 256-row window per CTA on a sliced-ELL copy of the
//       operator built at the call's start, x = v * 1/beta folded in; also
//       stores Q[:, i] = x                           (no partial sums)
//   A2  h1 = Q[:, :i+1]^T y                          (partials, last-CTA sum)
//   B   q1 = y - Q h1,  h2 = Q^T q1                  (partials, last-CTA sum)
//   C   q2 = q1 - Q h2, ||q2||^2                     (partials, last-CTA sum)
// and a restart is one CTA's projected eigensolve and selection followed by a
// full-GPU rotation of the basis.  A kernel boundary is the grid-wide
// barrier, so no CTA ever waits on another and the kernels may share the GPU
// with other work.  Each CTA writes its partial sums to [column][cta]; the
// last CTA to finish (an atomic ticket after a fence) sums them in CTA order,
// so the result does not depend on which CTA is last.  The loop state lives
// in a device control block (StreamCtl) that only those last CTAs and the
// restart kernel write: every kernel of a step reads the same state at its
// start and derives the same mode (step, breakdown replacement, or nothing
// to do), so the host enqueues a cycle's launches without reading anything
// back, and reads the block once per restart.
template <typename VT>
struct StShared {
  union {
    struct {
      double ys[LZ_BLOCK];
      double wred[LZ_NW][MP1];
    } st;
    __align__(16) VT Ys[MAXM * MAXM];
  } u;
  double h[MP1];
  VT hv[MP1];
  int last;
};

enum { SM_SKIP = 0, SM_STEP = 1, SM_BREAKDOWN = 2 };

// the step's mode from the control block's first eight ints (i, k, bd, cur,
// stop, rot, ...; the same in every kernel of a step), read as two 16-byte
// loads in one round trip
__device__ __forceinline__ int st_mode_of(int4 a, int4 b, int m, int* i, int* nv, int* buf) {
  const int ii = a.x, bd = a.z, cur = a.w, stop = b.x, rot = b.y;
  *i = ii;
  if (stop || rot) return SM_SKIP;
  if (bd) { *nv = ii; *buf = cur ^ 1; return SM_BREAKDOWN; }
  if (ii < m) { *nv = ii + 1; *buf = cur; return SM_STEP; }
  return SM_SKIP;
}
// What the solve's own kernels write (the control block, the basis, the work vectors)
// is read by ordinary loads (ld_seen) after st_pdl_prologue, which makes the writes of the
// kernels before visible: an early-started kernel's life overlaps theirs, and the
// read-only path (__ldg) holds only for data that no one writes during it.  The
// ordinary loads may use the L1 as well.  (Through L2 alone, every warp of every
// CTA would queue on the control block's line.)  They are volatile asm without a
// memory clobber: nothing moves them before the prologue or a barrier, and the
// compiler may issue them ahead of stores to other vectors, as it does with __ldg.
__device__ __forceinline__ float ld_seen(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_seen(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_seen(const int* p) {
  int v;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_seen(const float2* p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_seen(const float4* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_seen(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_seen(const int4* p) {
  int4 v;
  asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ int st_mode(const StreamCtl* c, int m, int* i, int* nv, int* buf) {
  const int4* p = (const int4*)c;
  return st_mode_of(ld_seen(p), ld_seen(p + 1), m, i, nv, buf);
}

// Programmatic dependent launch: each stream kernel lets the next one in the
// stream launch as soon as all of its own CTAs have started, then waits until
// the previous kernel has finished and its writes are visible.  The next
// kernel's launch thus overlaps this one's tail; no data is read early.
__device__ __forceinline__ void st_pdl_prologue() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ticket of the last CTA: true in every thread of the CTA that finished last
// (its partial sums, fenced by their writers, are then visible to it)
template <typename SH>
__device__ __forceinline__ bool st_last_cta(unsigned* ticket, SH& sh) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sh.last = (atomicAdd(ticket, 1u) == gridDim.x - 1) ? 1 : 0;
  __syncthreads();
  if (sh.last) __threadfence();
  return sh.last != 0;
}

// h[c] = sum over the R CTAs of part[c][r], c < nv: warp w takes columns
// w, w + 8, ...; lane l sums CTAs l, l + 64, ... and l + 32, l + 96, ... in order,
// then a butterfly.  A column's loads are issued sixteen at a time, the next
// sixteen before these are added: the last CTA works alone here, and a load in
// front of every pair of FP64 adds made its sum (25 columns of 489 partials at
// n = 10^6) half of the dots' kernel.
template <typename VT, typename SH>
__device__ __forceinline__ void st_reduce(const double* part, int R, int nv, SH& sh) {
  constexpr int B = 16;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nb = (R + 32 * B - 1) / (32 * B);       // batches per column
  auto fetch = [&](int c, int b, double (&v)[B]) {
    const double* p = part + (size_t)c * R;
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int r = lane + 32 * (b * B + u);
      v[u] = (c < nv && r < R) ? __ldcg(p + r) : 0.0;
    }
  };
  double v[B], a0 = 0.0, a1 = 0.0;
  int c = w, b = 0;
  fetch(c, b, v);
  while (c < nv) {
    double x[B];
#pragma unroll
    for (int u = 0; u < B; ++u) x[u] = v[u];
    const int cn = (b + 1 < nb) ? c : c + LZ_NW, bn = (b + 1 < nb) ? b + 1 : 0;
    fetch(cn, bn, v);
    // (warp-uniform ends: rows past R hold zeros, which add nothing)
    const int left = (R - 32 * b * B + 31) / 32;
#pragma unroll
    for (int u = 0; u < B; u += 2) {
      if (u < left) a0 += x[u];
      if (u + 1 < left) a1 += x[u + 1];
    }
    if (bn == 0) {
      const double a = warp_sum(a0 + a1);
      if (lane == 0) { sh.h[c] = a; sh.hv[c] = (VT)a; }
      a0 = a1 = 0.0;
    }
    c = cn;
    b = bn;
  }
  __syncthreads();
}

// ---- vector helpers of the Q-streaming kernels ----
// 4 consecutive rows of a column (16-byte aligned: ld is a multiple of 32 and
// the first row a multiple of 4); rows at or past n read as 0.  The basis is
// read through the L1, the work vectors, which B and C update, through L2.
template <typename VT> struct Row4 { VT v[4]; };
template <typename VT, bool L1 = true>
__device__ __forceinline__ Row4<VT> ld4(const VT* p, int r4, int n) {
  Row4<VT> o;
  if (r4 + 4 <= n) {
    if constexpr (sizeof(VT) == 4) {
      const float4 a = L1 ? ld_seen((const float4*)(p + r4)) : __ldcg((const float4*)(p + r4));
      o.v[0] = a.x; o.v[1] = a.y; o.v[2] = a.z; o.v[3] = a.w;
    } else {
      const double2 a = L1 ? ld_seen((const double2*)(p + r4)) : __ldcg((const double2*)(p + r4));
      const double2 b =
          L1 ? ld_seen((const double2*)(p + r4 + 2)) : __ldcg((const double2*)(p + r4 + 2));
      o.v[0] = a.x; o.v[1] = a.y; o.v[2] = b.x; o.v[3] = b.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o.v[j] = (r4 + j < n) ? (L1 ? ld_seen(p + r4 + j) : __ldcg(p + r4 + j)) : (VT)0;
  }
  return o;
}
template <typename VT>
__device__ __forceinline__ void st4(VT* p, int r4, int n, const Row4<VT>& o) {
  if (r4 + 4 <= n) {
    if constexpr (sizeof(VT) == 4) {
      *(float4*)(p + r4) = make_float4(o.v[0], o.v[1], o.v[2], o.v[3]);
    } else {
      *(double2*)(p + r4) = make_double2(o.v[0], o.v[1]);
      *(double2*)(p + r4 + 2) = make_double2(o.v[2], o.v[3]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (r4 + j < n) p[r4 + j] = o.v[j];
  }
}

constexpr int ST_ROWS = 4 * LZ_BLOCK;   // rows of one chunk (4 per thread)
// column loads issued before any is used: 128 bytes per thread either way
template <typename VT> constexpr int st_batch() { return sizeof(VT) == 4 ? 8 : 4; }

// s = sum_{c < nv} Q[r4.., c] * hv[c] for a thread's 4 rows, in column
// order, st_batch() column loads in flight at a time
template <typename VT>
__device__ __forceinline__ Row4<VT> st_combine(const VT* Q, size_t ld, int r4, int n, int nv,
                                               const VT* hv) {
  constexpr int NB = st_batch<VT>();
  Row4<VT> s;
#pragma unroll
  for (int j = 0; j < 4; ++j) s.v[j] = (VT)0;
#pragma unroll 1
  for (int c0 = 0; c0 < nv; c0 += NB) {
    Row4<VT> q[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (c0 + b < nv) q[b] = ld4(Q + (size_t)(c0 + b) * ld, r4, n);
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (c0 + b < nv) {
        const VT h = hv[c0 + b];
#pragma unroll
        for (int j = 0; j < 4; ++j) s.v[j] += q[b].v[j] * h;
      }
  }
  return s;
}

// out[c * R] = sum over the CTA's threads of sacc[c][t], c < nv: warp w takes
// columns w, w + 8, ...; lane l sums threads l, l + 32, ... in order
template <typename AT>
__device__ __forceinline__ void st_block_cols(const AT* sacc, int nv, double* out, int R) {
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = w; c < nv; c += LZ_NW) {
    AT a = (AT)0;
#pragma unroll
    for (int k = 0; k < LZ_BLOCK / 32; ++k) a += sacc[c * LZ_BLOCK + lane + 32 * k];
    a = warp_sum(a);
    if (lane == 0) out[(size_t)c * R] = (double)a;
  }
}

// the per-thread dot accumulators of B (dynamic shared memory)
template <typename VT>
constexpr size_t st_sacc_bytes() {
  return (size_t)MP1 * LZ_BLOCK * sizeof(typename Acc<VT>::type);
}

// chunk range [c0, c1) of ST_ROWS-row chunks of this CTA
__device__ __forceinline__ void st_chunks(int n, int* c0, int* c1) {
  const int nch = (n + ST_ROWS - 1) / ST_ROWS, R = gridDim.x;
  *c0 = (int)((long long)nch * blockIdx.x / R);
  *c1 = (int)((long long)nch * (blockIdx.x + 1) / R);
}

// ---- the stream path's operator layout (built once per call) ----
// Rows of each 256-row window are ordered by length (longest first, then by
// row) and cut into 32-row slices; slice s keeps entry k of its lane-th row at
// sl_ptr[s] + 32 k + lane for k below the slice's width (its longest row's
// length, at most wcap; shorter rows are padded with column 0, value 0; rows
// longer than wcap finish from the CSR).  Three launches: the order and the
// widths per window, a prefix sum of the slice sizes, the entries.
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) st_sell_order_kernel(
    const __grid_constant__ TeamDesc<VT> P) {
  __shared__ int len[LZ_BLOCK];
  __shared__ int order[LZ_BLOCK];
  const int w0 = blockIdx.x * LZ_BLOCK, tid = threadIdx.x, r = w0 + tid;
  const int rows = min(LZ_BLOCK, P.n - w0);
  len[tid] = (r < P.n) ? P.rowptr[r + 1] - P.rowptr[r] : -1;
  __syncthreads();
  if (tid < rows) {
    const int mine = len[tid];
    int rank = 0;
    for (int j = 0; j < rows; ++j) {
      const int lj = len[j];
      rank += (lj > mine || (lj == mine && j < tid)) ? 1 : 0;
    }
    order[rank] = tid;
  }
  __syncthreads();
  // thread p: sorted position p of the window (slice p / 32, lane p % 32).  A
  // slice that exists (s < ceil(n / 32)) has a real row at its first position.
  const int p = tid, s = blockIdx.x * (LZ_BLOCK / 32) + p / 32, lane = p & 31;
  if (s >= (P.n + 31) / 32) return;
  const int lr = (p < rows) ? order[p] : p;      // padding lanes: unused positions
  P.sl_row[32 * s + lane] = (unsigned char)lr;
  if (lane == 0) P.sl_ptr[s + 1] = 32 * min(len[order[p]], P.wcap);
}

// sl_ptr[1..ns] (slice sizes) -> offsets, sl_ptr[0] = 0; one CTA of 1024
__global__ void __launch_bounds__(1024) st_sell_scan_kernel(int ns, int* sl_ptr) {
  __shared__ int part[1024];
  const int tid = threadIdx.x, per = (ns + 1023) / 1024;
  const int t0 = min(tid * per, ns), t1 = min(t0 + per, ns);
  int sum = 0;
  for (int i = t0; i < t1; ++i) sum += sl_ptr[i + 1];
  part[tid] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int v = tid >= off ? part[tid - off] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  int base = tid ? part[tid - 1] : 0;
  for (int i = t0; i < t1; ++i) {
    base += sl_ptr[i + 1];
    sl_ptr[i + 1] = base;
  }
  if (tid == 0) sl_ptr[0] = 0;
}

template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) st_sell_fill_kernel(
    const __grid_constant__ TeamDesc<VT> P) {
  const int w0 = blockIdx.x * LZ_BLOCK, p = threadIdx.x;
  const int s = blockIdx.x * (LZ_BLOCK / 32) + p / 32, lane = p & 31;
  if (s >= (P.n + 31) / 32) return;
  const int base = P.sl_ptr[s], w = (P.sl_ptr[s + 1] - base) >> 5;
  const int r = w0 + P.sl_row[32 * s + lane];
  const int b = (r < P.n) ? P.rowptr[r] : 0;
  const int lenr = (r < P.n) ? P.rowptr[r + 1] - b : 0;
  int* cdst = P.sl_col + base + lane;
  VT* vdst = P.sl_val + base + lane;
  for (int k = 0; k < w; ++k) {
    const bool e = k < lenr;
    cdst[32 * k] = e ? P.col[b + k] : 0;
    vdst[32 * k] = e ? P.val[b + k] : (VT)0;
  }
}

// A1: y = Op x on the sliced-ELL layout, one CTA per window, one warp per
// slice, lane = row: the first 16 entries' column / value loads, then their x
// gathers, all in flight at once.  Step: vbuf[cur] = Op x with x = (i == k ?
// Q[:, k] : vbuf[cur ^ 1] / beta), and Q[:, i] = x when i > k.  Breakdown:
// vbuf[cur ^ 1] = a Gaussian vector keyed by i (the replacement of
// solver/lanczos.py:107-117).  x is gathered through the L1.
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK, 8) st_sell_spmv_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  typedef typename Acc<VT>::type AT;
  __shared__ VT ys[LZ_BLOCK];
  // every load that depends on no other is issued first: the control block,
  // the slice's width and row map
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = blockIdx.x * (LZ_BLOCK / 32) + warp;
  const bool has = s < (P.n + 31) / 32;
  const int4 ca = ld_seen((const int4*)ctl), cb = ld_seen((const int4*)ctl + 1);
  const double invb_d = ld_seen(&ctl->invb);
  const int sb = has ? __ldg(P.sl_ptr + s) : 0;
  const int width = has ? (__ldg(P.sl_ptr + s + 1) - sb) >> 5 : 0;
  const int lr = has ? (int)__ldg(P.sl_row + 32 * s + lane) : 0;
  int i, nv, buf;
  const int mode = st_mode_of(ca, cb, P.m, &i, &nv, &buf);
  if (mode == SM_SKIP) return;
  const size_t ld = (size_t)P.ld;
  const int w0 = blockIdx.x * LZ_BLOCK, row = w0 + threadIdx.x;
  if (mode == SM_BREAKDOWN) {
    if (row < P.n) P.vbuf[(size_t)buf * P.ldv + row] = (VT)hash_normal((uint64_t)i, (uint64_t)row);
    return;
  }
  const int k = ca.y;
  const bool wq = i > k;
  const VT xscale = wq ? (VT)invb_d : (VT)1;
  const VT* x = wq ? P.vbuf + (size_t)(buf ^ 1) * P.ldv : P.Q + (size_t)k * ld;
  const VT xrow = (wq && row < P.n) ? ld_seen(x + row) : (VT)0;
  if (has) {
    const int* cp = P.sl_col + sb + lane;
    const VT* vp = P.sl_val + sb + lane;
    constexpr int PF = 16;
    int c[PF];
    VT v[PF], xv[PF];
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      c[u] = (u < width) ? __ldg(cp + 32 * u) : 0;
      v[u] = (u < width) ? __ldg(vp + 32 * u) : (VT)0;
    }
#pragma unroll
    for (int u = 0; u < PF; ++u) xv[u] = (u < width) ? ld_seen(x + c[u]) : (VT)0;
    AT acc = (AT)0;
#pragma unroll
    for (int u = 0; u < PF; ++u) acc += (AT)v[u] * (AT)xv[u];
    for (int u = PF; u < width; ++u) acc += (AT)__ldg(vp + 32 * u) * (AT)ld_seen(x + __ldg(cp + 32 * u));
    const int r = w0 + lr;
    if (r < P.n && width == P.wcap) {
      // the rest of a row longer than the slice capacity
      const int e = P.rowptr[r + 1];
      for (int q = P.rowptr[r] + P.wcap; q < e; ++q)
        acc += (AT)__ldg(P.val + q) * (AT)ld_seen(x + __ldg(P.col + q));
    }
    ys[lr] = (VT)acc;
  }
  __syncthreads();
  if (row < P.n) {
    P.vbuf[(size_t)buf * P.ldv + row] = ys[threadIdx.x] * xscale;
    if (wq) P.Q[(size_t)i * ld + row] = xrow * xscale;
  }
}

// A2: h1[c] = Q[:, c] . v for c < nv (v = the step's y, or the breakdown vector).
// The grid is DOT_G x R: the R row blocks of the partial sums, each shared by DOT_G
// CTAs that take columns g, g + DOT_G, ...  One CTA per row block left SMs with
// three or four of them (489 blocks at n = 10^6) and one CTA to add all columns'
// partials at the end; a group's last CTA adds its own columns.
constexpr int DOT_G = 4, DOT_U = MAXM / DOT_G;
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) st_dot_kernel(const __grid_constant__ TeamDesc<VT> P,
                                                           StreamCtl* ctl) {
  st_pdl_prologue();
  typedef typename Acc<VT>::type AT;
  __shared__ int last;
  __shared__ AT sacc[DOT_U * LZ_BLOCK];
  int i, nv, buf;
  if (st_mode(ctl, P.m, &i, &nv, &buf) == SM_SKIP) return;
  const int R = gridDim.x / DOT_G, g = blockIdx.x % DOT_G, rb = blockIdx.x / DOT_G;
  const int mine = (nv - g + DOT_G - 1) / DOT_G;            // columns g, g + DOT_G, ... < nv
  if (mine <= 0) return;
  const size_t ld = (size_t)P.ld;
  const int nch = (P.n + ST_ROWS - 1) / ST_ROWS;
  const int c0 = (int)((long long)nch * rb / R), c1 = (int)((long long)nch * (rb + 1) / R);
  const VT* v = P.vbuf + (size_t)buf * P.ldv;
  AT acc[DOT_U];
#pragma unroll
  for (int u = 0; u < DOT_U; ++u) acc[u] = (AT)0;
  for (int ch = c0; ch < c1; ++ch) {
    const int r4 = ch * ST_ROWS + 4 * threadIdx.x;
    if (r4 < P.n) {
      constexpr int B = st_batch<VT>();
#pragma unroll
      for (int u0 = 0; u0 < DOT_U; u0 += B) {
        if (u0 < mine) {
          Row4<VT> q[B];
#pragma unroll
          for (int u = 0; u < B; ++u)
            if (u0 + u < mine) q[u] = ld4(P.Q + (size_t)(g + DOT_G * (u0 + u)) * ld, r4, P.n);
          const Row4<VT> x = ld4<VT, false>(v, r4, P.n);
#pragma unroll
          for (int u = 0; u < B; ++u)
            if (u0 + u < mine) {
              AT d = (AT)0;
#pragma unroll
              for (int j = 0; j < 4; ++j) d += (AT)q[u].v[j] * (AT)x.v[j];
              acc[u0 + u] += d;
            }
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < DOT_U; ++u)
    if (u < mine) sacc[u * LZ_BLOCK + threadIdx.x] = acc[u];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w < mine) {                                            // one column per warp
    AT s = (AT)0;
#pragma unroll
    for (int k = 0; k < LZ_BLOCK / 32; ++k) s += sacc[w * LZ_BLOCK + lane + 32 * k];
    s = warp_sum(s);
    if (lane == 0) P.part[(size_t)(g + DOT_G * w) * R + rb] = (double)s;
  }
  // the group's last CTA
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&ctl->dticket[g], 1u) == (unsigned)R - 1u) ? 1 : 0;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // st_reduce's sums of columns g + DOT_G w: lane l adds partials l, l + 64, ... and
  // l + 32, l + 96, ..., then a butterfly
  if (w < mine) {
    const double* p = P.part + (size_t)(g + DOT_G * w) * R;
    double a0 = 0.0, a1 = 0.0;
    for (int r0 = 0; r0 < R; r0 += 512) {
      double x[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int r = r0 + lane + 32 * u;
        x[u] = (r < R) ? __ldcg(p + r) : 0.0;
      }
      const int left = (R - r0 + 31) / 32;
#pragma unroll
      for (int u = 0; u < 16; u += 2) {
        if (u < left) a0 += x[u];
        if (u + 1 < left) a1 += x[u + 1];
      }
    }
    const double a = warp_sum(a0 + a1);
    if (lane == 0) ctl->h1[g + DOT_G * w] = a;
  }
  if (threadIdx.x == 0) ctl->dticket[g] = 0u;
}

// B, one pass over Q: each thread keeps its rows of the nv basis columns in
// registers (8-byte loads: two FP32 rows or one FP64 row), forms
// v -= Q h1, then h2 = Q^T v from the same registers.
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK, 2) st_update_dot1_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  typedef typename Acc<VT>::type AT;
  constexpr int RW = 8 / (int)sizeof(VT);           // rows per thread
  constexpr int CROWS = RW * LZ_BLOCK;              // rows per chunk
  __shared__ StShared<VT> sh;
  int i, nv, buf;
  const int mode = st_mode(ctl, P.m, &i, &nv, &buf);
  if (mode == SM_SKIP) return;
  const int R = gridDim.x, n = P.n;
  const size_t ld = (size_t)P.ld;
  for (int c = threadIdx.x; c < nv; c += LZ_BLOCK) sh.hv[c] = (VT)ld_seen(&ctl->h1[c]);
  extern __shared__ __align__(16) unsigned char st_dyn[];
  AT* sacc = (AT*)st_dyn;
  for (int c = 0; c < nv; ++c) sacc[c * LZ_BLOCK + threadIdx.x] = (AT)0;
  __syncthreads();
  const int nch = (n + CROWS - 1) / CROWS;
  const int c0 = (int)((long long)nch * blockIdx.x / R);
  const int c1 = (int)((long long)nch * (blockIdx.x + 1) / R);
  VT* v = P.vbuf + (size_t)buf * P.ldv;
  for (int ch = c0; ch < c1; ++ch) {
    const int r0 = ch * CROWS + RW * threadIdx.x;
    if (r0 >= n) continue;
    const bool full = r0 + RW <= n;
    VT q[MP1][RW];
#pragma unroll
    for (int c = 0; c < MP1; ++c)
      if (c < nv) {
        const VT* src = P.Q + (size_t)c * ld + r0;
        if constexpr (RW == 2) {
          if (full) {
            const float2 a = ld_seen((const float2*)src);
            q[c][0] = a.x; q[c][1] = a.y;
          } else {
            q[c][0] = ld_seen(src); q[c][1] = (VT)0;
          }
        } else {
          q[c][0] = ld_seen(src);
        }
      }
    VT x[RW], s[RW];
#pragma unroll
    for (int j = 0; j < RW; ++j) {
      x[j] = (r0 + j < n) ? __ldcg(v + r0 + j) : (VT)0;
      s[j] = (VT)0;
    }
#pragma unroll
    for (int c = 0; c < MP1; ++c)
      if (c < nv) {
        const VT h = sh.hv[c];
#pragma unroll
        for (int j = 0; j < RW; ++j) s[j] += q[c][j] * h;
      }
#pragma unroll
    for (int j = 0; j < RW; ++j) {
      x[j] -= s[j];
      if (r0 + j < n) v[r0 + j] = x[j];
    }
#pragma unroll
    for (int c = 0; c < MP1; ++c)
      if (c < nv) {
        AT d = (AT)0;
#pragma unroll
        for (int j = 0; j < RW; ++j) d += (AT)q[c][j] * (AT)x[j];
        sacc[c * LZ_BLOCK + threadIdx.x] += d;
      }
  }
  double* part = P.part + (size_t)MP1 * R;
  st_block_cols(sacc, nv, part + blockIdx.x, R);
  if (!st_last_cta(&ctl->ticket[0], sh)) return;
  st_reduce<VT>(part, R, nv, sh);
  for (int c = threadIdx.x; c < nv; c += LZ_BLOCK) ctl->h2[c] = sh.h[c];
  if (threadIdx.x == 0) {
    if (mode == SM_STEP) ctl->alpha[i] = __ldcg(&ctl->h1[i]) + sh.h[i];
    ctl->ticket[0] = 0u;
  }
}

// C: v -= Q h2 (c < nv), ||v||^2; the last CTA advances the loop state
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) st_update_norm_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  typedef typename Acc<VT>::type AT;
  __shared__ StShared<VT> sh;
  int i, nv, buf;
  const int mode = st_mode(ctl, P.m, &i, &nv, &buf);
  if (mode == SM_SKIP) return;
  const int R = gridDim.x;
  const size_t ld = (size_t)P.ld;
  for (int c = threadIdx.x; c < nv; c += LZ_BLOCK) sh.hv[c] = (VT)ld_seen(&ctl->h2[c]);
  __syncthreads();
  int c0, c1;
  st_chunks(P.n, &c0, &c1);
  VT* v = P.vbuf + (size_t)buf * P.ldv;
  AT nrm[MP1];
  nrm[0] = (AT)0;
  for (int ch = c0; ch < c1; ++ch) {
    const int r4 = ch * ST_ROWS + 4 * threadIdx.x;
    if (r4 >= P.n) continue;
    Row4<VT> x = ld4<VT, false>(v, r4, P.n);
    const Row4<VT> s = st_combine(P.Q, ld, r4, P.n, nv, sh.hv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x.v[j] -= s.v[j];
      nrm[0] += (AT)x.v[j] * (AT)x.v[j];
    }
    st4(v, r4, P.n, x);
  }
  double* part = P.part + (size_t)2 * MP1 * R;
  block_reduce_cols(nrm, 1, sh, part + blockIdx.x, R);
  if (!st_last_cta(&ctl->ticket[1], sh)) return;
  st_reduce<VT>(part, R, 1, sh);
  if (threadIdx.x == 0) {
    const double nrm2 = sh.h[0];
    if (mode == SM_STEP) {
      // solver/lanczos.py:95-105 and the breakdown test of :107
      const double b = sqrt(nrm2);
      ctl->beta[i] = b;
      ctl->steps += 1;
      ctl->sum_nv += i + 1;
      ctl->cur = buf ^ 1;
      ctl->i = i + 1;
      if (b < 1e-15) {
        ctl->bd = 1;
        ctl->breakdowns += 1;
      } else {
        ctl->invb = 1.0 / b;
      }
    } else {
      ctl->invb = 1.0 / sqrt(nrm2);
      ctl->bd = 0;
    }
    ctl->ticket[1] = 0u;
  }
}

// restart, one CTA: the projected eigenproblem and the thick-restart choice
// (solver/lanczos.py:128-168, 202-221) once the cycle's m steps are done
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK, 1) st_restart_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  __shared__ LzShared<VT> sh;
  const int m = P.m, tid = threadIdx.x;
  if (ctl->stop || ctl->rot) return;
  if (ctl->bd || ctl->i < m) {
    // a cycle of the wave path that breakdowns made longer than planned
    if (P.resume && tid == 0) ctl->stop = ST_HANDED;
    return;
  }
  if (tid == 0) sh.eig_cycles = 0;
  if (tid < m) { sh.alpha[tid] = ctl->alpha[tid]; sh.beta[tid] = ctl->beta[tid]; }
  __syncthreads();
  const int k = ctl->k;
  const long long c0 = clock64();
  restart_select<false>(P, sh, k);
  if (tid < m) { ctl->alpha[tid] = sh.alpha[tid]; ctl->beta[tid] = sh.beta[tid]; }
  if (tid == 0) {
    const int kn = sh.k_next;
    ctl->stepped = (k < m) ? 1 : 0;
    ctl->k = kn;
    ctl->nconv = sh.nconv;
    ctl->restarts += 1;
    ctl->sum_kn += kn;
    ctl->rot = 1;
    const bool bad = (*(volatile int*)P.status & ST_NONFINITE) != 0;
    if (bad || sh.nconv >= P.num_desired || ctl->restarts >= P.max_restarts)
      ctl->stop = ST_ENDED;
    P.ctl[2] = ctl->restarts;
    P.ctl[3] = ctl->breakdowns;
    P.ctl[4] = ctl->steps;
    P.ctl[6] += (int)((clock64() - c0) >> 10);
    P.ctl[13] = ctl->sum_nv;
    P.ctl[14] = ctl->sum_kn;
    P.ctl[15] += (int)(sh.eig_cycles >> 10);
  }
}

// restart rotation, full grid: Q[:, :kn] = Q[:, :m] Y, then Q[:, kn] (and
// Q[:, m]) = the last normalised vector (solver/lanczos.py:217-221)
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) st_rotate_kernel(const __grid_constant__ TeamDesc<VT> P,
                                                              StreamCtl* ctl) {
  st_pdl_prologue();
  __shared__ StShared<VT> sh;
  if (!ld_seen(&ctl->rot)) return;
  const int m = P.m, kn = ld_seen(&ctl->k);
  const bool stepped = ld_seen(&ctl->stepped) != 0;
  const VT invb = (VT)ld_seen(&ctl->invb);
  const size_t ld = (size_t)P.ld;
  const VT* lastv = P.vbuf + (size_t)(ld_seen(&ctl->cur) ^ 1) * P.ldv;
  for (int e = threadIdx.x; e < m * MAXM; e += LZ_BLOCK) {
    const int j = e / MAXM, c = e - j * MAXM;
    sh.u.Ys[e] = (c < kn) ? (VT)__ldcg(P.Ybuf + j * m + c) : (VT)0;
  }
  __syncthreads();
  const int R = gridDim.x, ntiles = (P.n + LZ_BLOCK - 1) / LZ_BLOCK;
  const int t0 = (int)((long long)ntiles * blockIdx.x / R);
  const int t1 = (int)((long long)ntiles * (blockIdx.x + 1) / R);
  for (int tile = t0; tile < t1; ++tile) {
    const int row = tile * LZ_BLOCK + threadIdx.x;
    if (row < P.n) {
      VT qr[MAXM];
#pragma unroll
      for (int j = 0; j < MAXM; ++j) qr[j] = (j < m) ? P.Q[(size_t)j * ld + row] : (VT)0;
      const VT xl = stepped ? lastv[row] * invb : P.Q[(size_t)m * ld + row];
      // four output columns per pass, their Y entries read together (Y is
      // zero past column kn, so the last pass may overrun kn harmlessly)
      for (int c0 = 0; c0 < kn; c0 += 4) {
        VT s[4] = {(VT)0, (VT)0, (VT)0, (VT)0};
#pragma unroll
        for (int j = 0; j < MAXM; ++j)
          if (j < m) {
            VT y4[4];
            if constexpr (sizeof(VT) == 4) {
              const float4 a = *(const float4*)&sh.u.Ys[j * MAXM + c0];
              y4[0] = a.x; y4[1] = a.y; y4[2] = a.z; y4[3] = a.w;
            } else {
              const double2 a = *(const double2*)&sh.u.Ys[j * MAXM + c0];
              const double2 b = *(const double2*)&sh.u.Ys[j * MAXM + c0 + 2];
              y4[0] = a.x; y4[1] = a.y; y4[2] = b.x; y4[3] = b.y;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += qr[j] * y4[u];
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (c0 + u < kn) P.Q[(size_t)(c0 + u) * ld + row] = s[u];
      }
      P.Q[(size_t)kn * ld + row] = xl;
      if (kn != m) P.Q[(size_t)m * ld + row] = xl;
    }
  }
  if (!st_last_cta(&ctl->ticket[2], sh)) return;
  if (threadIdx.x == 0) {
    ctl->i = kn;     // the next cycle starts from Q[:, kn]
    ctl->rot = 0;
    ctl->breakdowns0 = __ldcg(&ctl->breakdowns);
    ctl->steps0 = __ldcg(&ctl->steps);
    ctl->sum_nv0 = __ldcg(&ctl->sum_nv);
    ctl->ticket[2] = 0u;
  }
}

// ---------------------------------------------------------------- wave path
// A team-size problem (too large for one cluster, x of at most 160 KB) that has
// the GPU's launches to itself runs its first cycles as four ordinary launches
// per Lanczos step, like the stream path, with the team kernel's arithmetic:
//   A1  y = Op x, Q[:, i] = x
//   A2  partial h1 = Q^T y
//   B   q1 = y - Q h1, partial h2 = Q^T q1
//   C   q2 = q1 - Q h2, partial ||q2||^2, the step's state
// Every sum is the team kernel's: rank r of its R CTAs owns up to four 256-row
// tiles, thread t accumulates a column over row t of each in turn, and the R
// partial sums of a column are added by lanes r, r + 32, ... and a butterfly.  Here
// a rank is four CTAs (a cluster in B and C).  CTA j takes the rows of tile j for
// the updates, and columns j, j + 4, ... of the dots over all four tiles (their
// vector, in B, from the other CTAs' shared memory).  So four times as many
// SMs work, a step has four kernel boundaries where the team kernel has three
// grid barriers of about 20k cycles, and the results are the same bits.
// The host reads nothing back: a cycle's steps are bounded by the rule of the
// restart, so all launches are enqueued at once, those past the loop's end
// return, and a launch of the team kernel follows that continues from the
// control block: after breakdowns (which take slots of their own; it runs their
// cycle again from its start), or when there are more restarts than launches
// planned (see WV_LAUNCHES).
// ER n = 30,011 of degree 12, FP32, 10 restarts: 4.7 ms per call (14.4 as one
// cooperative launch of 30 CTAs, 5.3 with A1 and A2 as one kernel).
constexpr int WV_C = 4;                  // CTAs (tiles) per rank
constexpr int WV_U = 8;                  // columns per CTA: c = j + 4 u

// adds cycles to one of the control block's counters (CTA 0).  At a kernel's end, where
// no fence or cluster barrier has to wait for the atomic.
__device__ __forceinline__ void wv_count(StreamCtl* ctl, int what, long long cycles) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    atomicAdd(&ctl->cyc[what], (unsigned long long)cycles);
}

struct WvPlace { int rank, j, tile, t0, nt; };
template <typename VT>
__device__ __forceinline__ WvPlace wv_place(const TeamDesc<VT>& P) {
  WvPlace w;
  const int ntiles = (P.n + LZ_BLOCK - 1) / LZ_BLOCK;
  w.rank = blockIdx.x / WV_C;
  w.j = blockIdx.x % WV_C;               // (its rank in the cluster, where there is one)
  w.t0 = (int)((long long)ntiles * w.rank / P.nctas);
  w.nt = (int)((long long)ntiles * (w.rank + 1) / P.nctas) - w.t0;
  w.tile = w.t0 + w.j;
  return w;
}

template <typename VT>
struct WvShared {
  union {
    struct {
      double ys[LZ_BLOCK];
      double wred[LZ_NW][MP1];
    } st;
  } u;
  double h[MP1];
  __align__(16) VT hv[MP1 + 3];
  VT xv[LZ_BLOCK];                       // the tile's vector, read by the rank's other CTAs
  int last;
};

// sh.h[c], sh.hv[c] = sum over the R ranks of part[c][r], c < nv <= 32: warp w
// takes columns 4 w .. 4 w + 3
template <typename VT>
__device__ __forceinline__ void wv_reduce(const double* part, int R, int nv, WvShared<VT>& sh) {
  const int lane = threadIdx.x & 31, c0 = 4 * (threadIdx.x >> 5);
  if (c0 < nv) {
    double a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = 0.0;
    for (int r = lane; r < R; r += 32)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + u < nv) a[u] += __ldcg(part + (size_t)(c0 + u) * R + r);
#pragma unroll
    for (int h = 16, w = 2; w >= 1; h >>= 1, w >>= 1) {
      const bool up = (lane & h) != 0;
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (u < w) {
          const double send = up ? a[u] : a[u + w], keep = up ? a[u + w] : a[u];
          a[u] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    double v = a[0];
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) v += __shfl_xor_sync(0xffffffffu, v, h);
    const int c = c0 + (lane >> 3);
    if ((lane & 7) == 0 && c < nv) { sh.h[c] = v; sh.hv[c] = (VT)v; }
  }
  __syncthreads();
}

// this CTA's columns of the rank's rows (0 past nv or the last row)
template <typename VT>
__device__ __forceinline__ void wv_load(const TeamDesc<VT>& P, const WvPlace& w, int nv,
                                        VT (&q)[WV_C][WV_U]) {
#pragma unroll
  for (int t = 0; t < WV_C; ++t) {
    const int row = (w.t0 + t) * LZ_BLOCK + threadIdx.x;
    const bool in = t < w.nt && row < P.n;
#pragma unroll
    for (int u = 0; u < WV_U; ++u) {
      const int c = w.j + WV_C * u;
      q[t][u] = (in && c < nv) ? ld_seen(P.Q + (size_t)c * P.ld + row) : (VT)0;
    }
  }
}

// partial dots of the CTA's columns with the rank's vector y
template <typename VT>
__device__ __forceinline__ void wv_dots(const TeamDesc<VT>& P, const WvPlace& w, WvShared<VT>& sh,
                                        int nv, const VT (&q)[WV_C][WV_U], const VT (&y)[WV_C],
                                        double* part) {
  typedef typename Acc<VT>::type AT;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  AT acc[WV_U];
#pragma unroll
  for (int u = 0; u < WV_U; ++u) acc[u] = (AT)0;
#pragma unroll
  for (int t = 0; t < WV_C; ++t)
    if (t < w.nt && (w.t0 + t) * LZ_BLOCK + tid < P.n) {
#pragma unroll
      for (int u = 0; u < WV_U; ++u)
        if (w.j + WV_C * u < nv) acc[u] += (AT)q[t][u] * (AT)y[t];
    }
#pragma unroll
  for (int h = 16, x = WV_U / 2; x >= 1; h >>= 1, x >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int u = 0; u < WV_U / 2; ++u)
      if (u < x) {
        const AT send = up ? acc[u] : acc[u + x], keep = up ? acc[u + x] : acc[u];
        acc[u] = keep + __shfl_xor_sync(0xffffffffu, send, h);
      }
  }
  AT v = acc[0];
#pragma unroll
  for (int h = 2; h >= 1; h >>= 1) v += __shfl_xor_sync(0xffffffffu, v, h);
  if ((lane & 3) == 0) sh.u.st.wred[wid][lane >> 2] = (double)v;
  __syncthreads();
  const int c = w.j + WV_C * tid;
  if (tid < WV_U && c < nv) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < LZ_NW; ++k) s += sh.u.st.wred[k][tid];
    part[(size_t)c * P.nctas + w.rank] = s;
  }
}

// the thread's row of its tile: its vector entry and basis row, loaded before h is
// known, then x - sum_{c < nv} Q[row, c] h[c]
template <typename VT>
struct WvRow {
  VT x, q[MAXM];
  __device__ __forceinline__ void load(const TeamDesc<VT>& P, int row, bool in, int nv,
                                       const VT* v) {
    x = in ? __ldcg(v + row) : (VT)0;
#pragma unroll
    for (int c = 0; c < MAXM; ++c)
      q[c] = (in && c < nv) ? ld_seen(P.Q + (size_t)c * P.ld + row) : (VT)0;
  }
  __device__ __forceinline__ VT update(const WvShared<VT>& sh, int nv) const {
    VT s = (VT)0;
#pragma unroll
    for (int c = 0; c < MAXM; ++c)
      if (c < nv) s += q[c] * sh.hv[c];
    return x - s;
  }
};

// A1, 64 rows per CTA, L lanes per row (spmv_tile's sums).  Breakdown
// (solver/lanczos.py:107-117): the replacement vector in y's place.
constexpr int WV_ROWS = 64;
template <typename VT, int L>
__device__ __forceinline__ void wv_spmv_rows(const TeamDesc<VT>& P, const VT* x, VT xscale, VT* v) {
  typedef typename Acc<VT>::type AT;
  constexpr int GPP = LZ_BLOCK / L, NP = (WV_ROWS + GPP - 1) / GPP;
  const int g = threadIdx.x / L, lig = threadIdx.x - (threadIdx.x / L) * L;
  const int base = blockIdx.x * WV_ROWS;
  int pb[NP], pe[NP], c0[NP];
  VT v0[NP], x0[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int lr = q * GPP + g;
    pb[q] = pe[q] = 0;
    if (lr < WV_ROWS && base + lr < P.n) {
      pb[q] = __ldg(P.rowptr + base + lr) + lig;
      pe[q] = __ldg(P.rowptr + base + lr + 1);
    }
  }
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    c0[q] = 0;
    v0[q] = (VT)0;
    if (pb[q] < pe[q]) { c0[q] = __ldg(P.col + pb[q]); v0[q] = __ldg(P.val + pb[q]); }
  }
#pragma unroll
  for (int q = 0; q < NP; ++q) x0[q] = ld_seen(x + c0[q]);
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    AT s = (AT)v0[q] * (AT)x0[q];
    for (int p = pb[q] + L; p < pe[q]; p += L)
      s += (AT)__ldg(P.val + p) * (AT)ld_seen(x + __ldg(P.col + p));
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int lr = q * GPP + g;
    if (lig == 0 && lr < WV_ROWS && base + lr < P.n) v[base + lr] = (VT)s * xscale;
  }
}
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) wv_spmv_kernel(const __grid_constant__ TeamDesc<VT> P,
                                                           StreamCtl* ctl) {
  st_pdl_prologue();
  const long long clk = clock64();
  int i, nv, buf;
  const int mode = st_mode(ctl, P.m, &i, &nv, &buf);
  if (mode == SM_SKIP) return;
  const size_t ld = (size_t)P.ld;
  const int row = blockIdx.x * WV_ROWS + threadIdx.x;
  const bool own = threadIdx.x < WV_ROWS && row < P.n;
  VT* v = P.vbuf + (size_t)buf * P.ldv;
  if (mode == SM_BREAKDOWN) {
    if (own) v[row] = (VT)hash_normal((uint64_t)i, (uint64_t)row);
    return;
  }
  const int k = ld_seen(&ctl->k);
  const bool wq = i > k;
  const VT* x = wq ? P.vbuf + (size_t)(buf ^ 1) * P.ldv : P.Q + (size_t)k * ld;
  const VT xscale = wq ? (VT)ld_seen(&ctl->invb) : (VT)1;
  if (wq && own) P.Q[(size_t)i * ld + row] = ld_seen(x + row) * xscale;
  switch (P.lanes) {
    case 1: wv_spmv_rows<VT, 1>(P, x, xscale, v); break;
    case 2: wv_spmv_rows<VT, 2>(P, x, xscale, v); break;
    case 4: wv_spmv_rows<VT, 4>(P, x, xscale, v); break;
    case 8: wv_spmv_rows<VT, 8>(P, x, xscale, v); break;
    case 16: wv_spmv_rows<VT, 16>(P, x, xscale, v); break;
    default: wv_spmv_rows<VT, 32>(P, x, xscale, v); break;
  }
  wv_count(ctl, 1, clock64() - clk);
}

// A2
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) wv_dot_kernel(const __grid_constant__ TeamDesc<VT> P,
                                                          StreamCtl* ctl) {
  st_pdl_prologue();
  __shared__ WvShared<VT> sh;
  const long long clk = clock64();
  int i, nv, buf;
  if (st_mode(ctl, P.m, &i, &nv, &buf) == SM_SKIP) return;
  const WvPlace w = wv_place(P);
  const VT* v = P.vbuf + (size_t)buf * P.ldv;
  VT q[WV_C][WV_U], y[WV_C];
  wv_load(P, w, nv, q);
#pragma unroll
  for (int t = 0; t < WV_C; ++t) {
    const int row = (w.t0 + t) * LZ_BLOCK + threadIdx.x;
    y[t] = (t < w.nt && row < P.n) ? ld_seen(v + row) : (VT)0;
  }
  wv_dots(P, w, sh, nv, q, y, P.part);
  wv_count(ctl, 1, clock64() - clk);
}

// B
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) wv_update_dot_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  __shared__ WvShared<VT> sh;
  int i, nv, buf;
  if (st_mode(ctl, P.m, &i, &nv, &buf) == SM_SKIP) return;
  const WvPlace w = wv_place(P);
  const int tid = threadIdx.x, row = w.tile * LZ_BLOCK + tid;
  const bool in = w.j < w.nt && row < P.n;
  VT* v = P.vbuf + (size_t)buf * P.ldv;
  WvRow<VT> r;
  r.load(P, row, in, nv, v);
  const long long clk = clock64();
  wv_reduce(P.part, P.nctas, nv, sh);
  const long long clk_red = clock64();
  if (blockIdx.x == 0 && tid < nv) ctl->h1[tid] = sh.h[tid];
  if (in) {
    const VT x = r.update(sh, nv);
    v[row] = x;
    sh.xv[tid] = x;
  }
  VT q[WV_C][WV_U], y[WV_C];
  wv_load(P, w, nv, q);
  cl_sync();
#pragma unroll
  for (int t = 0; t < WV_C; ++t) {
    y[t] = (VT)0;
    if (t < w.nt) y[t] = cl_ld(cl_map(&sh.xv[tid], (unsigned)t), (VT)0);
  }
  wv_dots(P, w, sh, nv, q, y, P.part + (size_t)MP1 * P.nctas);
  cl_sync();       // no CTA leaves while another reads its vector
  wv_count(ctl, 0, clk_red - clk);
  wv_count(ctl, 2, clock64() - clk_red);
}

// C; the last rank to finish advances the state (solver/lanczos.py:95-105, and the
// breakdown test of :107)
template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK) wv_update_norm_kernel(
    const __grid_constant__ TeamDesc<VT> P, StreamCtl* ctl) {
  st_pdl_prologue();
  typedef typename Acc<VT>::type AT;
  __shared__ WvShared<VT> sh;
  int i, nv, buf;
  const int mode = st_mode(ctl, P.m, &i, &nv, &buf);
  if (mode == SM_SKIP) return;
  const WvPlace w = wv_place(P);
  const int tid = threadIdx.x, lane = tid & 31, row = w.tile * LZ_BLOCK + tid, R = P.nctas;
  const bool in = w.j < w.nt && row < P.n;
  VT* v = P.vbuf + (size_t)buf * P.ldv;
  WvRow<VT> r;
  r.load(P, row, in, nv, v);
  const long long clk = clock64();
  wv_reduce(P.part + (size_t)MP1 * R, R, nv, sh);
  const long long clk_red = clock64();
  if (in) {
    const VT x = r.update(sh, nv);
    v[row] = x;
    sh.xv[tid] = x;
  }
  cl_sync();
  AT nrm = (AT)0;
  if (w.j == 0) {
#pragma unroll
    for (int t = 0; t < WV_C; ++t)
      if (t < w.nt && (w.t0 + t) * LZ_BLOCK + tid < P.n) {
        const VT x = cl_ld(cl_map(&sh.xv[tid], (unsigned)t), (VT)0);
        nrm += (AT)x * (AT)x;
      }
  }
  cl_sync();
  if (w.j != 0) return;
  nrm = warp_sum(nrm);
  if (lane == 0) sh.u.st.wred[tid >> 5][0] = (double)nrm;
  __syncthreads();
  double* part = P.part + (size_t)2 * MP1 * R;
  if (tid == 0) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < LZ_NW; ++k) s += sh.u.st.wred[k][0];
    part[w.rank] = s;
    __threadfence();
    sh.last = (atomicAdd(&ctl->ticket[1], 1u) == (unsigned)R - 1u) ? 1 : 0;
    wv_count(ctl, 0, clk_red - clk);
    wv_count(ctl, 3, clock64() - clk_red);
    if (sh.last) __threadfence();
  }
  __syncthreads();
  if (!sh.last || tid >= 32) return;
  double a = 0.0;
  for (int r = lane; r < R; r += 32) a += __ldcg(part + r);
  a = warp_sum(a);
  if (lane == 0) {
    const double b = sqrt(a);
    if (mode == SM_STEP) {
      ctl->alpha[i] = __ldcg(&ctl->h1[i]) + sh.h[i];
      ctl->beta[i] = b;
      ctl->steps += 1;
      ctl->sum_nv += i + 1;
      ctl->cur = buf ^ 1;
      ctl->i = i + 1;
      if (b < 1e-15) {
        ctl->bd = 1;
        ctl->breakdowns += 1;
      } else {
        ctl->invb = 1.0 / b;
      }
    } else {
      ctl->invb = 1.0 / b;
      ctl->bd = 0;
    }
    ctl->ticket[1] = 0u;
  }
}

// ---------------------------------------------------------------- cluster path
// A problem of at most CL_MAX_CTAS x rc rows runs as one thread-block cluster.
// CTA r of the cluster owns rows [r rc, (r+1) rc) and keeps, for the whole
// eigsh call, its rows of the basis Q (column-major, stride rc), the two work
// vectors and, when it fits, its slice of the operator in shared memory.  The
// SpMV gathers x from the owner CTAs' shared memory (distributed shared memory,
// mapa + ld.shared::cluster; the address of each entry's row is formed once) or
// from a copy of all of x that each CTA makes per step (see the rule in the
// kernel); each phase's per-CTA partial sums are written to
// the CTA's own shared memory and, after a hardware cluster barrier, summed by
// every CTA over the cluster in the same fixed order, so all CTAs hold
// bit-identical coefficients and take identical branches.  The restart's
// projected eigenproblem is solved redundantly by every CTA (identical inputs,
// identical results), which needs no broadcast; its FP64 refinement is shared
// out.  A cluster is co-scheduled by the hardware, so there is no software
// barrier and no spin-wait.
// Bound by latency: FP32 torus n = 10^4 runs 19k cycles per step (SpMV and dots
// 5.9k, second projection 4.2k, norm pass 2.6k, reductions 4.5k, barriers 1.7k)
// and 153k per restart, 2.13 ms per call of 131 steps (3.53 ms with one
// gather, one column and one shuffle level at a time); FP64 ER n = 800 of
// degree 48 3.02 ms (8.25 ms).
constexpr int CL_MAX_CTAS = 16;

template <typename VT>
struct ClusterDesc {
  int n, ld, m, num_desired, max_restarts, lanes, rc, csr_cap;
  long long nnz;
  double tol;
  const int* rowptr;
  const int* col;
  const VT* val;
  VT* Q;
  double* alpha;
  double* beta;
  int* ctl;
  int* status;
};

template <typename VT>
struct ClusterBatch {
  int count, csize;
  ClusterDesc<VT> t[MAX_TEAMS];
};

// per-CTA shared-memory layout of the cluster kernel (byte offsets)
struct ClLayout {
  size_t q, vb, part, rp, cg, val, total;
};
__host__ __device__ inline size_t cl_al(size_t b) { return (b + 15) & ~(size_t)15; }
template <typename VT>
__host__ __device__ inline ClLayout cl_layout(int m, int rc, int csr_cap) {
  ClLayout L;
  L.q = 0;
  L.vb = L.q + cl_al((size_t)(m + 1) * rc * sizeof(VT));
  L.part = L.vb + cl_al((size_t)2 * rc * sizeof(VT));
  L.rp = L.part + cl_al((size_t)3 * MP1 * sizeof(double));
  L.cg = L.rp + cl_al((size_t)(rc + 1) * sizeof(int));
  L.val = L.cg + cl_al((size_t)csr_cap * sizeof(int));
  L.total = L.val + cl_al((size_t)csr_cap * sizeof(VT));
  return L;
}

// h[c] = sum over the cluster's CTAs r = 0..C-1 of part_r[c], c < nv, summed
// as a fixed pairwise tree over 16 slots (slots r >= C hold 0): level one adds
// slots r and r+8, level two r and r+4, level three r and r+2, level four r and
// r+1.  A warp gets one FP64 add per ~60 cycles, dependent or not, while the SM's
// FP64 unit takes one from any warp every 19, so warps 0..3 each form one
// level-two sum R_w = (v_w + v_{w+8}) + (v_{w+4} + v_{w+12}), and warp 0 then forms
// (R_0 + R_2) + (R_1 + R_3): the tree's association, spread over four warps.
// With norm set (nv = 1), lane 0 also forms sh.bnorm = sqrt(h[0]) and
// sh.binv = 1 / bnorm once for the CTA (FP64 square roots and divisions are
// long dependent chains on this part's narrow FP64 pipe).
static_assert(CL_MAX_CTAS == 16, "the reduction tree below is written for 16 slots");
template <typename VT>
__device__ __forceinline__ void cl_reduce(const double* part, int C, int nv, LzShared<VT>& sh,
                                          bool norm = false) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid < 4) {
    for (int c = lane; c < nv; c += 32) {
      const double a = (wid < C) ? cl_ld(cl_map(part + c, wid), 0.0) : 0.0;
      const double b = (wid + 8 < C) ? cl_ld(cl_map(part + c, wid + 8), 0.0) : 0.0;
      const double d = (wid + 4 < C) ? cl_ld(cl_map(part + c, wid + 4), 0.0) : 0.0;
      const double e = (wid + 12 < C) ? cl_ld(cl_map(part + c, wid + 12), 0.0) : 0.0;
      sh.u.red4[wid][c] = (a + b) + (d + e);
    }
  }
  __syncthreads();
  if (wid == 0) {
    for (int c = lane; c < nv; c += 32) {
      const double v = (sh.u.red4[0][c] + sh.u.red4[2][c]) + (sh.u.red4[1][c] + sh.u.red4[3][c]);
      sh.h[c] = v;
      sh.hv[c] = (VT)v;
      if (norm) {
        const double b = sqrt(v);
        sh.bnorm = b;
        sh.binv = (VT)(1.0 / b);
      }
    }
  }
  __syncthreads();
}

// The cluster kernel's dynamic shared memory as words of VT from its start (the
// basis comes first); every vector below is an offset from there, so that the
// accesses are shared-memory instructions with 32-bit addresses.
template <typename VT>
__device__ __forceinline__ VT* cl_dyn_words() {
  extern __shared__ __align__(16) unsigned char cl_dyn[];
  return (VT*)cl_dyn;
}

template <typename VT>
struct ClCtx {
  int rank, C, n, m, rc, r0, rows;
  int lanes, lp;        // accumulators per row of the SpMV, threads per row (lp <= lanes)
  bool staged;          // CSR slice in shared memory
  bool short_rows;      // not staged, few entries per lane: four rows at a time
  int rp, cg, vs;       // its row bounds (rows+1 ints, from the slice's start), columns, values
  int xs;               // the whole x, copied at the start of each SpMV (or -1)
  const int* g_rowptr;  // the operator in global memory (slices that do not fit)
  const int* g_col;
  const VT* g_val;
};

// Row sums of the SpMV.  A row's entries are dealt round-robin to `lanes`
// accumulators that are then added pairwise (distance lanes/2, ..., 1).  A row
// takes lp <= lanes threads, each with NL = lanes / lp of the accumulators in
// registers (thread t: t, t + lp, ...), so the first log2(NL) levels of the tree
// need no shuffle; the sums do not depend on lp.  lp is chosen so that one pass
// of the CTA covers its rows: with one row per warp (lanes = 32, 62 FP64 rows of
// 49 entries per CTA) the shuffle tree's FP64 adds took 50k cycles per step,
// because an FP64 warp instruction costs the SM's one unit 19 cycles however few
// lanes carry a row.
// XS: x is read from the CTA's copy and cg holds byte offsets in it; else cg
// holds the shared::cluster address of the entry's row in its owner's Q[:, 0].
template <typename VT, int NL, bool XS>
__device__ __forceinline__ VT cl_row_sum(const ClCtx<VT>& X, int lr, int lig, int xo) {
  typedef typename Acc<VT>::type AT;
  const int L = X.lanes, lp = X.lp;
  AT s[NL];
#pragma unroll
  for (int u = 0; u < NL; ++u) s[u] = (AT)0;
  if (lr < X.rows) {
    constexpr int B = NL < 8 ? NL : 8;           // entries in flight per round trip ...
    constexpr int U = NL < 8 ? 8 / NL : 1;       // ... over U trips round the accumulators
    if (NL > 1 || X.staged) {         // (in global memory lp = lanes: NL = 1)
      const VT* D = cl_dyn_words<VT>();
      const int* rp = cl_dyn_words<int>() + X.rp;
      const uint32_t* cg = cl_dyn_words<uint32_t>() + X.cg;
      const int e = rp[lr + 1];
      for (int p0 = rp[lr] + lig; p0 < e; p0 += U * L) {
#pragma unroll
        for (int b0 = 0; b0 < NL; b0 += B) {
          VT av[U * B], xv[U * B];
          uint32_t ad[U * B];
#pragma unroll
          for (int v = 0; v < U * B; ++v) {
            const int p = p0 + (v / B) * L + (b0 + v % B) * lp;
            ad[v] = (p < e) ? cg[p] : 0u;
            av[v] = (p < e) ? D[X.vs + p] : (VT)0;
          }
#pragma unroll
          for (int v = 0; v < U * B; ++v) {
            const int p = p0 + (v / B) * L + (b0 + v % B) * lp;
            if constexpr (XS) {
              xv[v] = *(const VT*)((const char*)(D + X.xs) + ad[v]);
            } else {
              xv[v] = (VT)0;
              if (p < e) xv[v] = cl_ld(ad[v] + xo * (int)sizeof(VT), (VT)0);
            }
          }
#pragma unroll
          for (int v = 0; v < U * B; ++v) {
            const int p = p0 + (v / B) * L + (b0 + v % B) * lp;
            if (p < e) s[b0 + v % B] += (AT)av[v] * (AT)xv[v];
          }
        }
      }
    } else if constexpr (NL == 1) {
      const int e = X.g_rowptr[X.r0 + lr + 1];
      for (int p0 = X.g_rowptr[X.r0 + lr] + lig; p0 < e; p0 += U * L) {
#pragma unroll
        for (int b0 = 0; b0 < NL; b0 += B) {
          VT av[U * B], xv[U * B];
          int gc[U * B];
#pragma unroll
          for (int v = 0; v < U * B; ++v) {
            const int p = p0 + (v / B) * L + (b0 + v % B) * lp;
            gc[v] = (p < e) ? X.g_col[p] : -1;
            av[v] = (p < e) ? X.g_val[p] : (VT)0;
          }
#pragma unroll
          for (int v = 0; v < U * B; ++v) {
            xv[v] = (VT)0;
            if (gc[v] >= 0) {
              if constexpr (XS) {
                xv[v] = cl_dyn_words<VT>()[X.xs + gc[v]];
              } else {
                const int o = gc[v] / X.rc;
                xv[v] = cl_ld(cl_map(cl_dyn_words<VT>() + xo + (gc[v] - o * X.rc), (unsigned)o), (VT)0);
              }
            }
          }
#pragma unroll
          for (int v = 0; v < U * B; ++v)
            if (gc[v] >= 0) s[b0 + v % B] += (AT)av[v] * (AT)xv[v];
        }
      }
    }
  }
#pragma unroll
  for (int o = NL / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int u = 0; u < o; ++u) s[u] += s[u + o];
  }
  AT r = s[0];
  for (int o = lp >> 1; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return (VT)r;
}

// Row sums of a slice in global memory with short rows (lp = lanes: one accumulator
// per thread): four rows per thread group at a time, whose bounds, first two entries
// and gathers are in flight together, so a group waits for three round trips to L2
// per four rows and for two more per further entry of a lane.  cl_row_sum takes one
// row at a time, three round trips for up to eight entries of a lane.
template <typename VT, bool XS>
__device__ __forceinline__ void cl_spmv_global(const ClCtx<VT>& X, int xo, VT xscale, int vout) {
  typedef typename Acc<VT>::type AT;
  constexpr int R = 4, U = 2;                      // rows, entries of each in flight
  const int L = X.lanes, gpp = LZ_BLOCK / L;
  const int g = threadIdx.x / L, lig = threadIdx.x & (L - 1);
  VT* D = cl_dyn_words<VT>();
  auto gather = [&](int gc) -> VT {
    if constexpr (XS) {
      return D[X.xs + gc];
    } else {
      const int o = gc / X.rc;
      return cl_ld(cl_map(D + xo + (gc - o * X.rc), (unsigned)o), (VT)0);
    }
  };
  for (int base = 0; base < X.rows; base += R * gpp) {
    int pb[R], pe[R], c[R][U];
    VT v[R][U], xv[R][U];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int lr = base + r * gpp + g;
      pb[r] = pe[r] = 0;
      if (lr < X.rows) {
        pb[r] = X.g_rowptr[X.r0 + lr] + lig;
        pe[r] = X.g_rowptr[X.r0 + lr + 1];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int p = pb[r] + u * L;
        c[r][u] = (p < pe[r]) ? X.g_col[p] : -1;
        v[r][u] = (p < pe[r]) ? X.g_val[p] : (VT)0;
      }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        xv[r][u] = (VT)0;
        if (c[r][u] >= 0) xv[r][u] = gather(c[r][u]);
      }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      AT s = (AT)0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c[r][u] >= 0) s += (AT)v[r][u] * (AT)xv[r][u];
      for (int p = pb[r] + U * L; p < pe[r]; p += L)
        s += (AT)X.g_val[p] * (AT)gather(X.g_col[p]);
      for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int lr = base + r * gpp + g;
      if (lig == 0 && lr < X.rows) D[vout + lr] = (VT)s * xscale;
    }
  }
}

// the same out of line.  In FP32 the staged path's kernel is then faster (torus
// n = 10^4: 2.13 against 2.23 ms per call, its second projection 4.2 against 5.5
// kilocycles per step), while slices in global memory lose up to a fifth of their
// SpMV (n = 7000 of degree 80: 62 against 51); in FP64 inline is the faster form
// (ER n = 800: 2.92 against 2.97 ms).
template <typename VT, bool XS>
__device__ __noinline__ void cl_spmv_global_call(const ClCtx<VT> X, int xo, VT xscale, int vout) {
  cl_spmv_global<VT, XS>(X, xo, xscale, vout);
}

// vout = Op x * xscale for own rows; x and vout are offsets, the gathers read the
// owner CTA's copy of x (or this CTA's copy of all of it)
template <typename VT, int NL, bool XS>
__device__ __forceinline__ void cl_spmv_rows(const ClCtx<VT>& X, int xo, VT xscale, int vout) {
  const int lp = X.lp, gpp = LZ_BLOCK / lp;
  const int g = threadIdx.x / lp, lig = threadIdx.x & (lp - 1);
  for (int base = 0; base < X.rows; base += gpp) {
    const VT s = cl_row_sum<VT, NL, XS>(X, base + g, lig, xo);
    if (lig == 0 && base + g < X.rows) cl_dyn_words<VT>()[vout + base + g] = s * xscale;
  }
}
template <typename VT, bool XS>
__device__ __forceinline__ void cl_spmv(const ClCtx<VT>& X, int xo, VT xscale, int vout) {
  if (X.short_rows) {
    if constexpr (sizeof(VT) == 4) cl_spmv_global_call<VT, XS>(X, xo, xscale, vout);
    else cl_spmv_global<VT, XS>(X, xo, xscale, vout);
    return;
  }
  switch (X.lanes / X.lp) {
    case 1: cl_spmv_rows<VT, 1, XS>(X, xo, xscale, vout); break;
    case 2: cl_spmv_rows<VT, 2, XS>(X, xo, xscale, vout); break;
    case 4: cl_spmv_rows<VT, 4, XS>(X, xo, xscale, vout); break;
    case 8: cl_spmv_rows<VT, 8, XS>(X, xo, xscale, vout); break;
    case 16: cl_spmv_rows<VT, 16, XS>(X, xo, xscale, vout); break;
    default: cl_spmv_rows<VT, 32, XS>(X, xo, xscale, vout); break;
  }
}

// xs = x: warps take blocks of 256 rows of one owner CTA (starting with the next
// CTA, so that the cluster's CTAs read from different peers), eight consecutive
// 32-word rows of loads in flight per warp
template <typename VT>
__device__ __forceinline__ void cl_stage_x(const ClCtx<VT>& X, int xo) {
  VT* D = cl_dyn_words<VT>();
  const int lane = threadIdx.x & 31, parts = (X.rc + 255) / 256;
  for (int id = threadIdx.x >> 5; id < X.C * parts; id += LZ_NW) {
    const int part = id / X.C;
    int o = X.rank + 1 + id - part * X.C;
    if (o >= X.C) o -= X.C;
    const int j0 = part * 256 + lane, rows = min(X.rc, X.n - o * X.rc);
    const uint32_t src = cl_map(D + xo + j0, (unsigned)o);
    VT v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      v[u] = (VT)0;
      if (j0 + 32 * u < rows) v[u] = cl_ld(src + 32 * u * (int)sizeof(VT), (VT)0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + 32 * u < rows) D[X.xs + o * X.rc + j0 + 32 * u] = v[u];
  }
}

// Columns c0 .. c0 + CW - 1 of the partial dots of one row-warp: acc[c] over its
// rows, then summed across the warp by a butterfly whose payload halves while
// more than one column is left (distance 16, 8, 4, 2, 1: the association of a
// plain warp sum), to sh.u.st.wred[rw][c].
template <int CW, typename VT>
__device__ __forceinline__ void cl_warp_cols(typename Acc<VT>::type* acc, LzShared<VT>& sh,
                                             int rw, int c0) {
  typedef typename Acc<VT>::type AT;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 16, w = CW; h >= 1; h >>= 1) {
    if (w > 1) {
      w >>= 1;
      const bool up = (lane & h) != 0;
#pragma unroll
      for (int j = 0; j < CW / 2; ++j) {
        if (j < w) {
          const AT send = up ? acc[j] : acc[j + w];
          const AT keep = up ? acc[j + w] : acc[j];
          acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
      }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], h);
    }
  }
  constexpr int LPC = 32 / CW;                   // lanes that hold one column
  if (lane % LPC == 0) sh.u.st.wred[rw][c0 + lane / LPC] = (double)acc[0];
}

// out[c] = sum over the nrw row-warps, in their order, of wred[.][c], c < nv
template <typename VT>
__device__ __forceinline__ void cl_block_cols(LzShared<VT>& sh, int nrw, int nv, double* out) {
  __syncthreads();
  for (int c = threadIdx.x; c < nv; c += LZ_BLOCK) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < LZ_NW; ++w)
      if (w < nrw) s += sh.u.st.wred[w][c];
    out[c] = s;
  }
}

// A thread's rows are taken RT at a time (lr, lr + 256, ...).  In FP32 the loads
// and FMA chains of three rows overlap (CTAs of at most 256 rows: one); in FP64 the
// CTA's warps already keep the SM's FP64 unit busy (19 cycles per instruction).
template <typename VT> constexpr int cl_rt() { return sizeof(VT) == 4 ? 3 : 1; }

// G columns c0 .. of a thread's RT rows; with PART, those at or past nv as 0.
// Rows past the CTA's last are read too (whatever follows them in the layout;
// their results are not used): the row offsets stay immediates.
template <int RT, int G, bool PART, typename VT>
__device__ __forceinline__ void cl_ld_cols(const ClCtx<VT>& X, int lr, int c0, int nv,
                                           VT (&q)[RT][G]) {
  const VT* D = cl_dyn_words<VT>() + c0 * X.rc + lr;
#pragma unroll
  for (int c = 0; c < G; ++c) {
#pragma unroll
    for (int r = 0; r < RT; ++r)
      q[r][c] = (!PART || c0 + c < nv) ? D[c * X.rc + r * LZ_BLOCK] : (VT)0;
  }
}
template <typename VT>
__device__ __forceinline__ void cl_hv8(const LzShared<VT>& sh, int c0, VT (&h)[8]) {
  if constexpr (sizeof(VT) == 4) {
    const float4 a = *(const float4*)(sh.hv + c0), b = *(const float4*)(sh.hv + c0 + 4);
    h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w;
    h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
  } else {
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 a = *(const double2*)(sh.hv + c0 + c);
      h[c] = a.x; h[c + 1] = a.y;
    }
  }
}

// acc[c] += Q[lr, c] y over a thread's RT rows lr, lr + 256, ..., c < nv
template <int RT, bool PART, typename VT>
__device__ __forceinline__ void cl_dot8(const ClCtx<VT>& X, int lr, int g, int nv,
                                        const VT (&y)[RT], typename Acc<VT>::type* acc) {
  typedef typename Acc<VT>::type AT;
  VT q[RT][8];
  cl_ld_cols<RT, 8, PART>(X, lr, g, nv, q);
#pragma unroll
  for (int r = 0; r < RT; ++r)
    if (lr + r * LZ_BLOCK < X.rows) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (!PART || g + c < nv) acc[c] += (AT)q[r][c] * (AT)y[r];
    }
}
template <int RT, typename VT>
__device__ __forceinline__ void cl_dot_rows(const ClCtx<VT>& X, int lr, int nv, int vec,
                                            typename Acc<VT>::type* acc) {
  VT y[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) y[r] = cl_dyn_words<VT>()[vec + lr + r * LZ_BLOCK];
#pragma unroll
  for (int g = 0; g < 32; g += 8) {
    if (RT == 1 && g + 8 <= nv) cl_dot8<RT, false>(X, lr, g, nv, y, acc + g);
    else if (g < nv) cl_dot8<RT, true>(X, lr, g, nv, y, acc + g);
  }
}

// Partial dots Q[:, c] . vec, c < nv <= 32, over the CTA's rows.  Lane l of
// row-warp w accumulates rows 32 w + l, 32 w + l + 256, ...; CTAs with at most
// 128, 64 or 32 rows have 4, 2 or 1 row-warps and give each 2, 4 or 8 warps,
// which split the columns, so that all eight warps work.  vec may just have been
// written by other threads.
template <int CW, typename VT>
__device__ __forceinline__ void cl_dots_w(const ClCtx<VT>& X, LzShared<VT>& sh, int nv, int vec,
                                          double* part_out) {
  typedef typename Acc<VT>::type AT;
  constexpr int NRW = CW / 4;                    // row-warps: 8 CW / 32
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int rw = wid % NRW, c0 = (wid / NRW) * CW;
  AT acc[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) acc[c] = (AT)0;
  if (c0 < nv) {
    if constexpr (CW == 32) {
      constexpr int RT = cl_rt<VT>();
      for (int lr = threadIdx.x; lr - lane < X.rows; lr += RT * LZ_BLOCK) {
        if (RT > 1 && X.rows > LZ_BLOCK) cl_dot_rows<RT>(X, lr, nv, vec, acc);
        else cl_dot_rows<1>(X, lr, nv, vec, acc);
      }
    } else {
      const int lr = 32 * rw + lane;             // at most one row per lane
      if (lr < X.rows) {
        const VT y = cl_dyn_words<VT>()[vec + lr];
        VT q[1][CW];
        cl_ld_cols<1, CW, true>(X, lr, c0, nv, q);
#pragma unroll
        for (int c = 0; c < CW; ++c)
          if (c0 + c < nv) acc[c] += (AT)q[0][c] * (AT)y;
      }
    }
    cl_warp_cols<CW>(acc, sh, rw, c0);
  }
  cl_block_cols(sh, NRW, nv, part_out);
}
template <typename VT>
__device__ __forceinline__ void cl_dots(const ClCtx<VT>& X, LzShared<VT>& sh, int nv, int vec,
                                        double* part_out) {
  if (X.rows > 128) cl_dots_w<32>(X, sh, nv, vec, part_out);
  else if (X.rows > 64) cl_dots_w<16>(X, sh, nv, vec, part_out);
  else if (X.rows > 32) cl_dots_w<8>(X, sh, nv, vec, part_out);
  else cl_dots_w<4>(X, sh, nv, vec, part_out);
}

// Phase A: vout = Op (x * xscale) for own rows, partial Q[:, c] . vout (c <= i);
// if wq, Q[:, i] = x * xscale (own rows)
template <typename VT>
__device__ __forceinline__ void cl_phase_spmv(const ClCtx<VT>& X, LzShared<VT>& sh, int i, int xo,
                                              VT xscale, bool wq, int vout, double* part_out) {
  VT* D = cl_dyn_words<VT>();
  if (wq)
    for (int lr = threadIdx.x; lr < X.rows; lr += LZ_BLOCK) D[i * X.rc + lr] = D[xo + lr] * xscale;
  if (X.xs >= 0) {
    cl_stage_x(X, xo);
    __syncthreads();
    cl_spmv<VT, true>(X, xo, xscale, vout);
  } else {
    cl_spmv<VT, false>(X, xo, xscale, vout);
  }
  __syncthreads();
  cl_dots(X, sh, i + 1, vout, part_out);
}

template <typename VT>
__device__ void cl_phase_random(const ClCtx<VT>& X, LzShared<VT>& sh, int nv, uint64_t key,
                                int buf, double* part_out) {
  for (int lr = threadIdx.x; lr < X.rows; lr += LZ_BLOCK)
    cl_dyn_words<VT>()[buf + lr] = (VT)hash_normal(key, (uint64_t)(X.r0 + lr));
  __syncthreads();
  cl_dots(X, sh, nv, buf, part_out);
}

// x[r] = buf[.] - sum_{c < nv} Q[., c] hv[c] in column order for a thread's RT
// rows (lr, lr + 256, ...), written back to buf
template <int RT, bool PART, typename VT>
__device__ __forceinline__ void cl_combine8(const ClCtx<VT>& X, const LzShared<VT>& sh, int lr,
                                            int g, int nv, VT (&s)[RT]) {
  VT q[RT][8], h[8];
  cl_ld_cols<RT, 8, PART>(X, lr, g, nv, q);
  cl_hv8(sh, g, h);
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (!PART || g + c < nv) {
#pragma unroll
      for (int r = 0; r < RT; ++r) s[r] += q[r][c] * h[c];
    }
}
template <int RT, typename VT>
__device__ __forceinline__ void cl_combine(const ClCtx<VT>& X, const LzShared<VT>& sh, int nv,
                                           int lr, int buf, VT* x) {
  VT* D = cl_dyn_words<VT>() + buf + lr;
  VT s[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    s[r] = (VT)0;
    x[r] = D[r * LZ_BLOCK];
  }
  // one row: straight-line code for the groups of eight; three rows: a loop (a
  // third of the code, and the rows overlap as it is)
  if constexpr (RT == 1) {
#pragma unroll
    for (int g = 0; g < 32; g += 8) {
      if (g + 8 <= nv) cl_combine8<RT, false>(X, sh, lr, g, nv, s);
      else if (g < nv) cl_combine8<RT, true>(X, sh, lr, g, nv, s);
    }
  } else {
#pragma unroll 1
    for (int g = 0; g < nv; g += 8) cl_combine8<RT, true>(X, sh, lr, g, nv, s);
  }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    x[r] -= s[r];
    if (lr + r * LZ_BLOCK < X.rows) D[r * LZ_BLOCK] = x[r];
  }
}
// cl_combine of the rows that are left from lr on (at most RT), the squares of
// the results added to nrm
template <typename VT>
__device__ __forceinline__ void cl_update_rows(const ClCtx<VT>& X, const LzShared<VT>& sh, int nv,
                                               int lr, int buf, typename Acc<VT>::type& nrm) {
  typedef typename Acc<VT>::type AT;
  constexpr int RT = cl_rt<VT>();
  VT x[RT];
  if (RT > 1 && X.rows > LZ_BLOCK) cl_combine<RT>(X, sh, nv, lr, buf, x);
  else cl_combine<1>(X, sh, nv, lr, buf, x);
#pragma unroll
  for (int r = 0; r < RT; ++r)
    if (lr + r * LZ_BLOCK < X.rows) nrm += (AT)x[r] * (AT)x[r];
}

// Phase B: buf -= Q h (c < nv); partial Q[:, c] . buf
template <typename VT>
__device__ __forceinline__ void cl_phase_update_dot(const ClCtx<VT>& X, LzShared<VT>& sh, int nv,
                                                    int buf, double* part_out) {
  const int lane = threadIdx.x & 31;
  typename Acc<VT>::type unused = 0;
  for (int lr = threadIdx.x; lr - lane < X.rows; lr += cl_rt<VT>() * LZ_BLOCK)
    cl_update_rows(X, sh, nv, lr, buf, unused);
  __syncthreads();
  cl_dots(X, sh, nv, buf, part_out);
}

// Phase C: buf -= Q h (c < nv); part_out[0] = sum buf^2 over own rows
template <typename VT>
__device__ __forceinline__ void cl_phase_update_norm(const ClCtx<VT>& X, LzShared<VT>& sh, int nv,
                                                     int buf, double* part_out) {
  const int lane = threadIdx.x & 31;
  typename Acc<VT>::type nrm = 0;
  for (int lr = threadIdx.x; lr - lane < X.rows; lr += cl_rt<VT>() * LZ_BLOCK)
    cl_update_rows(X, sh, nv, lr, buf, nrm);
  nrm = warp_sum(nrm);
  if (lane == 0) sh.u.st.wred[threadIdx.x >> 5][0] = (double)nrm;
  cl_block_cols(sh, min(LZ_NW, (X.rows + 31) / 32), 1, part_out);
}

template <typename VT>
__global__ void __launch_bounds__(LZ_BLOCK, 1)
lanczos_cluster_kernel(const __grid_constant__ ClusterBatch<VT> batch) {
  __shared__ __align__(16) LzShared<VT> sh;
  const int C = batch.csize;
  const ClusterDesc<VT>& P = batch.t[blockIdx.x / C];
  const int rank = (int)cl_rank();
  const int tid = threadIdx.x;
  const int n = P.n, m = P.m, rc = P.rc;
  const size_t ld = (size_t)P.ld;
  const ClLayout Lo = cl_layout<VT>(m, rc, P.csr_cap);
  VT* D = cl_dyn_words<VT>();
  ClCtx<VT> X;
  X.rank = rank;
  X.C = C;
  X.n = n;
  X.m = m;
  X.rc = rc;
  X.r0 = rank * rc;
  X.rows = max(0, min(rc, n - X.r0));
  X.lanes = P.lanes;
  X.rp = (int)(Lo.rp / sizeof(int));
  X.cg = (int)(Lo.cg / sizeof(int));
  X.vs = (int)(Lo.val / sizeof(VT));
  X.g_rowptr = P.rowptr;
  X.g_col = P.col;
  X.g_val = P.val;
  const int vb = (int)(Lo.vb / sizeof(VT));        // the two work vectors
  double* part0 = cl_dyn_words<double>() + Lo.part / sizeof(double);
  double* part1 = part0 + MP1;
  double* part2 = part0 + 2 * MP1;
  // stage Q[:, 0] (the start vector) and, if it fits, the operator slice
  for (int lr = tid; lr < X.rows; lr += LZ_BLOCK) D[lr] = P.Q[X.r0 + lr];
  const int p0 = (X.rows > 0) ? P.rowptr[X.r0] : 0;
  const int p1 = (X.rows > 0) ? P.rowptr[X.r0 + X.rows] : 0;
  X.staged = (p1 - p0) <= P.csr_cap;
  // up to 3.5 entries per lane and row on average; kilocycles of a step's SpMV, 16
  // CTAs, four rows at a time (inlined) / one row at a time: ER n = 7000 of degree 80
  // (2.5 per lane) 52 / 71, n = 5000 of degree 100 (3.1) 46 / 54, of degree 130 (4.1) 59 / 55,
  // n = 4000 of degree 200 (6.3) 70 / 44
  X.short_rows = !X.staged && 2ll * (p1 - p0) <= 7ll * X.lanes * X.rows;
  X.lp = 1;
  // (a slice read from global memory keeps one thread per accumulator: its
  // consecutive entries are then consecutive lanes')
  while (2 * X.lp <= X.lanes && (!X.staged || 2 * X.lp * X.rows <= LZ_BLOCK)) X.lp *= 2;
  X.xs = -1;
  if (X.staged) {
    int* rp = cl_dyn_words<int>() + X.rp;
    uint32_t* cg = cl_dyn_words<uint32_t>() + X.cg;
    int remote = 0;
    for (int p = p0 + tid; p < p1; p += LZ_BLOCK) {
      const int gc = P.col[p];
      remote += (gc < X.r0 || gc >= X.r0 + X.rows) ? 1 : 0;
      cg[p - p0] = (uint32_t)gc;
      D[X.vs + p - p0] = P.val[p];
    }
    // (a CTA past the problem's last row has no rows, and r0 may be past n)
    for (int lr = tid; lr <= X.rows; lr += LZ_BLOCK)
      rp[lr] = (X.rows > 0) ? P.rowptr[X.r0 + lr] - p0 : 0;
    remote = (int)block_sum((double)remote, sh.red);
    // A copy of all of x where there is room for it and the rows' entries in
    // other CTAs number at least a quarter of it: the copy reads consecutive
    // words of its peers, the gather scattered ones.  Phase A in kilocycles per
    // step, copied / gathered (16 CTAs): ER n = 5000 degree 30 FP32 11.6 / 32,
    // degree 8 8.7 / 12.4, n = 9000 degree 6 11.2 / 15, n = 800 degree 48 FP64
    // 9.1 / 13; below the line, torus n = 2500 FP32 5.2 / 3.7 (few peers).
    const int used = (p1 - p0 + 3) & ~3;
    if (P.csr_cap - used >= n && 4 * remote >= n) X.xs = X.vs + used;
    for (int p = tid; p < p1 - p0; p += LZ_BLOCK) {
      const int gc = (int)cg[p], o = gc / rc;
      cg[p] = X.xs >= 0 ? (uint32_t)(gc * (int)sizeof(VT)) : cl_map(D + (gc - o * rc), (unsigned)o);
    }
  } else if ((size_t)P.csr_cap * (sizeof(int) + sizeof(VT)) >= (size_t)n * sizeof(VT)) {
    X.xs = (int)(Lo.cg / sizeof(VT));     // the operator stays in global memory: the room is x's
  }
  int k = 0, nconv = 0, restart = 0, breakdowns = 0, steps = 0, sum_nv = 0, sum_kn = 0;
  long long clk_start = clock64(), clk_restart = 0;
  long long tp[5] = {0, 0, 0, 0, 0}, tmark = clock64();
  const bool timing = (rank == 0 && tid == 0);
  if (tid < MAXM) { sh.alpha[tid] = 0.0; sh.beta[tid] = 0.0; }
  if (tid == 0) sh.eig_cycles = 0;
  __syncthreads();
  cl_sync();
  int prev = 0;
  VT invb = (VT)1;
  while (nconv < P.num_desired && restart < P.max_restarts) {
    int cur = 0;
    for (int i = k; i < m; ++i) {
      int xbase;
      bool wq;
      if (i == k) {
        xbase = k * rc;
        invb = (VT)1;
        wq = false;
      } else {
        cl_reduce(part2, C, 1, sh, true);
        const double b = sh.bnorm;
        if (tid == 0) sh.beta[i - 1] = b;
        if (b < 1e-15) {
          // Krylov space exhausted: random vector orthogonalised twice
          // against Q[:, :i] (solver/lanczos.py:107-117)
          ++breakdowns;
          const int buf = vb + prev * rc;
          cl_phase_random(X, sh, i, (uint64_t)i, buf, part0);
          cl_sync();
          cl_reduce(part0, C, i, sh);
          cl_phase_update_dot(X, sh, i, buf, part1);
          cl_sync();
          cl_reduce(part1, C, i, sh);
          cl_phase_update_norm(X, sh, i, buf, part2);
          cl_sync();
          cl_reduce(part2, C, 1, sh, true);
          invb = sh.binv;
        } else {
          invb = sh.binv;
        }
        xbase = vb + prev * rc;
        wq = true;
      }
      const int vout = vb + cur * rc;
      if (timing) { const long long c = clock64(); tp[1] += c - tmark; tmark = c; }
      cl_phase_spmv(X, sh, i, xbase, invb, wq, vout, part0);
      if (timing) { const long long c = clock64(); tp[2] += c - tmark; tmark = c; }
      cl_sync();
      if (timing) { const long long c = clock64(); tp[0] += c - tmark; tmark = c; }
      cl_reduce(part0, C, i + 1, sh);
      if (timing) { const long long c = clock64(); tp[1] += c - tmark; tmark = c; }
      const double h1i = sh.h[i];
      cl_phase_update_dot(X, sh, i + 1, vout, part1);
      if (timing) { const long long c = clock64(); tp[3] += c - tmark; tmark = c; }
      cl_sync();
      if (timing) { const long long c = clock64(); tp[0] += c - tmark; tmark = c; }
      cl_reduce(part1, C, i + 1, sh);
      if (timing) { const long long c = clock64(); tp[1] += c - tmark; tmark = c; }
      if (tid == 0) sh.alpha[i] = h1i + sh.h[i];
      cl_phase_update_norm(X, sh, i + 1, vout, part2);
      if (timing) { const long long c = clock64(); tp[4] += c - tmark; tmark = c; }
      cl_sync();
      if (timing) { const long long c = clock64(); tp[0] += c - tmark; tmark = c; }
      prev = cur;
      cur ^= 1;
      ++steps;
      sum_nv += i + 1;
    }
    // ---- restart ----
    const bool stepped = (k < m);
    if (stepped) {
      cl_reduce(part2, C, 1, sh, true);
      const double b = sh.bnorm;
      if (tid == 0) sh.beta[m - 1] = b;
      if (b < 1e-15) {
        ++breakdowns;
        const int buf = vb + prev * rc;
        cl_phase_random(X, sh, m, (uint64_t)m, buf, part0);
        cl_sync();
        cl_reduce(part0, C, m, sh);
        cl_phase_update_dot(X, sh, m, buf, part1);
        cl_sync();
        cl_reduce(part1, C, m, sh);
        cl_phase_update_norm(X, sh, m, buf, part2);
        cl_sync();
        cl_reduce(part2, C, 1, sh, true);
        invb = sh.binv;
      } else {
        invb = sh.binv;
      }
    }
    __syncthreads();
    const long long c0 = clock64();
    restart_select<true>(P, sh, k, /*write_out=*/rank == 0, rank, C);
    if (timing) clk_restart += clock64() - c0;
    // every CTA of the cluster found the same projected matrix, so all of
    // them see their own ST_NONFINITE here and leave together
    if (*(volatile int*)P.status & ST_NONFINITE) { ++restart; break; }
    const int kn = sh.k_next;
    nconv = sh.nconv;
    const VT* last = D + (stepped ? vb + prev * rc : m * rc);
    const VT lscale = stepped ? invb : (VT)1;
    for (int lr = tid; lr < X.rows; lr += LZ_BLOCK) {
      VT qr[MAXM];
#pragma unroll
      for (int j = 0; j < MAXM; ++j) qr[j] = (j < m) ? D[j * rc + lr] : (VT)0;
      const VT xl = last[lr] * lscale;
      // four output columns per pass, their Y entries read together (Y is zero
      // past column kn, so the last pass may overrun kn)
      for (int c0 = 0; c0 < kn; c0 += 4) {
        VT s[4] = {(VT)0, (VT)0, (VT)0, (VT)0};
#pragma unroll
        for (int j = 0; j < MAXM; ++j)
          if (j < m) {
            VT y4[4];
            if constexpr (sizeof(VT) == 4) {
              const float4 a = *(const float4*)&sh.u.Ys[j * MAXM + c0];
              y4[0] = a.x; y4[1] = a.y; y4[2] = a.z; y4[3] = a.w;
            } else {
              const double2 a = *(const double2*)&sh.u.Ys[j * MAXM + c0];
              const double2 b = *(const double2*)&sh.u.Ys[j * MAXM + c0 + 2];
              y4[0] = a.x; y4[1] = a.y; y4[2] = b.x; y4[3] = b.y;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += qr[j] * y4[u];
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (c0 + u < kn) D[(c0 + u) * rc + lr] = s[u];
      }
      D[kn * rc + lr] = xl;
      if (kn != m) D[m * rc + lr] = xl;
    }
    k = kn;
    sum_kn += kn;
    ++restart;
    __syncthreads();
    cl_sync();   // rotated rows visible to the next cycle's gathers
    if (timing) tmark = clock64();
  }
  // the basis back to global memory (own rows; untouched if no cycle ran)
  if (restart > 0) {
    for (int c = 0; c <= m; ++c)
      for (int lr = tid; lr < X.rows; lr += LZ_BLOCK)
        P.Q[(size_t)c * ld + X.r0 + lr] = D[c * rc + lr];
  }
  if (rank == 0 && tid == 0) {
    P.ctl[2] = restart;
    P.ctl[3] = breakdowns;
    P.ctl[4] = steps;
    P.ctl[6] = (int)(clk_restart >> 10);
    P.ctl[7] = (int)((clock64() - clk_start) >> 10);
    for (int j = 0; j < 5; ++j) P.ctl[8 + j] = (int)(tp[j] >> 10);
    P.ctl[13] = sum_nv;
    P.ctl[14] = sum_kn;
    P.ctl[15] = (int)(sh.eig_cycles >> 10);
    if (restart == 0) P.ctl[0] = 0;
  }
  cl_sync();   // no CTA leaves while a peer may still read its shared memory
}

// ---------------------------------------------------------------- host side

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

static thread_local int t_launches = 0;   // kernels the last lanczos_run launched (this thread)

// x of a team-kernel problem is staged in shared memory; larger problems take
// the stream path
static bool x_fits_smem(int n, size_t vt) { return (size_t)n * vt <= (size_t)LZ_XS_BYTES; }

// Workspace: 3 work vectors, [pass][column][cta] partials, the Ritz vectors and the
// barrier counters; the stream path adds its operator layout.  The stream and wave
// paths' control block lies behind the third pass's partials, which are one column
// (the sums of squares) of the MP1 that the pass has room for: from six CTAs
// on it needs no room of its own.
static int vec_stride(int n) { return (n + 31) & ~31; }
static size_t ctl_offset(int nctas) {      // in bytes from the partials' start
  return ((size_t)(2 * MP1 + 1) * nctas * sizeof(double) + 15) & ~(size_t)15;
}
static size_t part_bytes(int nctas, bool with_ctl) {
  const size_t p = (size_t)3 * nctas * MP1 * sizeof(double);
  const size_t c = ctl_offset(nctas) + sizeof(StreamCtl);
  return align256(with_ctl && c > p ? c : p);
}
static bool ctl_fits(int nctas) {          // without more room than the partials'
  return ctl_offset(nctas) + sizeof(StreamCtl) <= (size_t)3 * nctas * MP1 * sizeof(double);
}
// entries per row a stream-path slice holds (longer rows finish from the CSR)
static int sell_wcap(int n, long long nnz) {
  const long long avg = n > 0 ? (nnz + n - 1) / n : 1;
  const long long w = avg + avg / 2 + 2;
  return (int)(w < 4 ? 4 : (w > 64 ? 64 : w));
}
static size_t sell_bytes(int n, long long nnz, size_t vt) {
  const size_t ns = ((size_t)n + 31) / 32;
  return align256((ns + 1) * sizeof(int)) + align256(ns * 32) +
         align256(ns * 32 * (size_t)sell_wcap(n, nnz) * sizeof(int)) +
         align256(ns * 32 * (size_t)sell_wcap(n, nnz) * vt);
}

size_t lanczos_workspace_bytes(int n, long long nnz, int ld, int m, int prec, int nctas,
                               bool stream) {
  (void)m;
  const size_t vt = (prec == 64) ? 8 : 4;
  const bool strm = stream || !x_fits_smem(n, vt);
  size_t b = align256(3 * (size_t)ld * vt);
  b += part_bytes(nctas, strm);
  b += align256((size_t)MAXM * MAXM * sizeof(double));
  b += 256;  // barrier counters
  if (strm) b += sell_bytes(n, nnz, vt);
  return b;
}

int lanczos_lanes(int n, long long nnz) {
  const double avg = n > 0 ? (double)nnz / n : 1.0;
  int L = 1;
  while (L < 32 && L * 2 <= avg * 0.75 + 1) L *= 2;
  return L;
}

int lanczos_team_size(const DeviceInfo& di, int n, int prec, bool stream) {
  if (stream || !x_fits_smem(n, prec == 64 ? 8 : 4)) {
    // stream path: the grid of its partial-sum kernels, one wave
    const int tiles = (n + LZ_BLOCK - 1) / LZ_BLOCK;
    const int occ = (prec == 64) ? di.stream_occ64 : di.stream_occ32;
    const int g = di.sm_count * (occ > 0 ? occ : 1);
    return tiles < g ? tiles : g;
  }
  const int occ = (prec == 64) ? di.lanczos_occ64 : di.lanczos_occ32;
  // two SMs stay free for the single-CTA kernels that run beside the team
  const int maxc = (di.sm_count > 4 ? di.sm_count - 2 : di.sm_count) * (occ > 0 ? occ : 1);
  const int tiles = (n + LZ_BLOCK - 1) / LZ_BLOCK;
  // at least 4 tiles per CTA: small problems are latency bound, and every
  // extra CTA costs barrier arrivals and partial sums on each phase
  int want = (tiles + 3) / 4;
  // USBS_LANCZOS_CTAS overrides the team size (tuning experiments)
  static const int forced = [] {
    const char* e = getenv("USBS_LANCZOS_CTAS");
    return e ? atoi(e) : 0;
  }();
  if (forced > 0) want = forced;
  if (want > tiles) want = tiles;
  if (want > maxc) want = maxc;
  if (want < 1) want = 1;
  return want;
}

// team kernel: dynamic shared memory it may use (the staged x)
template <typename VT>
constexpr size_t tm_dyn_max() {
  return (227 * 1024 - sizeof(LzShared<VT>) - 1024) / 128 * 128;
}
static_assert(tm_dyn_max<double>() >= (size_t)LZ_XS_BYTES, "staged x must fit");

// a problem's descriptor for R CTAs (or ranks), with its part of the workspace;
// returns the workspace behind it
template <typename VT>
static char* fill_desc(TeamDesc<VT>& t, const LanczosProblem& p, int R, bool with_ctl) {
  memset(&t, 0, sizeof(t));
  t.n = p.n; t.ld = p.ld; t.ldv = vec_stride(p.n); t.m = p.m; t.num_desired = p.num_desired;
  t.max_restarts = p.max_restarts; t.tol = p.tol;
  t.lanes = lanczos_lanes(p.n, p.nnz);
  t.nctas = R;
  t.rowptr = p.rowptr; t.col = p.col; t.val = (const VT*)p.val;
  t.nnz = p.nnz;
  t.Q = (VT*)p.Q; t.Qw = t.Q; t.qts = LZ_BLOCK; t.qcs = p.ld;
  t.alpha = p.alpha; t.beta = p.beta; t.ctl = p.ctl; t.status = p.status;
  char* w = (char*)p.work;
  t.vbuf = (VT*)w; w += align256(3 * (size_t)t.ldv * sizeof(VT));
  t.part = (double*)w; w += part_bytes(R, with_ctl);
  t.Ybuf = (double*)w; w += align256((size_t)MAXM * MAXM * sizeof(double));
  t.bar = (unsigned int*)w; w += 256;
  return w;
}

template <typename VT>
static int run_typed(const DeviceInfo& di, const LanczosProblem* probs, int count,
                     cudaStream_t stream, StreamCtl* const* resume = nullptr) {
  const int occ = (sizeof(VT) == 8) ? di.lanczos_occ64 : di.lanczos_occ32;
  const int maxc = (di.sm_count > 4 ? di.sm_count - 2 : di.sm_count) * (occ > 0 ? occ : 1);
  for (int base = 0; base < count; base += MAX_TEAMS) {
    const int cnt = (count - base < MAX_TEAMS) ? (count - base) : MAX_TEAMS;
    TeamBatch<VT> batch;
    batch.count = cnt;
    int total = 0;
    int want[MAX_TEAMS];   // cnt <= MAX_TEAMS; no heap allocation on the launch path
    for (int i = 0; i < cnt; ++i) {
      want[i] = lanczos_team_size(di, probs[base + i].n, sizeof(VT) == 8 ? 64 : 32);
      total += want[i];
    }
    if (total > maxc) {
      // shrink teams proportionally so that every CTA is co-resident
      int tot2 = 0;
      for (int i = 0; i < cnt; ++i) {
        want[i] = (int)((long long)want[i] * maxc / total);
        if (want[i] < 1) want[i] = 1;
        tot2 += want[i];
      }
      if (tot2 > maxc) {
        set_error("lanczos: %d problems need more co-resident CTAs (%d) than the device holds (%d)",
                  cnt, tot2, maxc);
        return -3;
      }
      total = tot2;
    }
    int first = 0;
    size_t dyn = 0;
    for (int i = 0; i < cnt; ++i) {
      const LanczosProblem& p = probs[base + i];
      if (p.m > MAXM || p.m < 1 || p.n < 1 || p.ld < p.n) {
        set_error("lanczos: unsupported sizes n=%d ld=%d m=%d (m must be in [1, %d])", p.n,
                  p.ld, p.m, MAXM);
        return -2;
      }
      TeamDesc<VT>& t = batch.t[i];
      fill_desc(t, p, want[i], false);
      t.xsmem = ((size_t)p.n * sizeof(VT) <= (size_t)LZ_XS_BYTES) ? 1 : 0;
      if (t.xsmem && (size_t)p.n * sizeof(VT) > dyn) dyn = (size_t)p.n * sizeof(VT);
      t.first_cta = first;
      t.resume = resume ? resume[base + i] : nullptr;
      first += want[i];
      if (cudaMemsetAsync(t.bar, 0, 2 * sizeof(unsigned int), stream) != cudaSuccess ||
          (!t.resume &&
           cudaMemsetAsync(p.ctl, 0, 16 * sizeof(int), stream) != cudaSuccess)) {
        set_error("lanczos: memset failed");
        return -4;
      }
    }
    void* args[] = {(void*)&batch};
    static bool attr_set = false;
    if (!attr_set) {
      cudaFuncSetAttribute((const void*)lanczos_team_kernel<VT>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tm_dyn_max<VT>());
      attr_set = true;
    }
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)lanczos_team_kernel<VT>,
                                                dim3(total), dim3(LZ_BLOCK), args, dyn, stream);
    ++t_launches;
    if (e != cudaSuccess) {
      set_error("lanczos: cooperative launch of %d CTAs failed: %s", total,
                cudaGetErrorString(e));
      return -5;
    }
  }
  return 0;
}

// Row blocks per SM of the stream path's partial-sum kernels and the rotation (A2,
// B, C, rotation).  They fix which rows share a partial sum, and with that the
// last bits of every dot, so they are numbers of their own and not the kernels'
// occupancies (which they were when each row block was one CTA of one wave).
// Sets the dynamic shared memory limit of B on the way.
template <typename VT>
static const int* stream_occ() {
  static const int blocks[4] = {sizeof(VT) == 4 ? 4 : 3, 2, 4, sizeof(VT) == 4 ? 3 : 2};
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute((const void*)st_update_dot1_kernel<VT>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)st_sacc_bytes<VT>());
  });
  return blocks;
}
// the largest of them (sizes the partial-sum buffers)
int lanczos_stream_occupancy(int prec) {
  const int* o = prec == 64 ? stream_occ<double>() : stream_occ<float>();
  int b = 1;
  for (int j = 0; j < 4; ++j) b = o[j] > b ? o[j] : b;
  return b;
}

// Whether a problem runs on the wave path: a team-size problem whose ranks hold at
// most four tiles and whose workspace has room for the control block (six ranks; below
// that only what a batch with a larger problem, or a cluster that cannot be had,
// sends here), outside a stream capture (where a call stays one node).
template <typename VT>
static bool wave_fits(const LanczosProblem& p, int nctas, cudaStream_t stream) {
  if (p.m > MAXM || p.m < 1 || p.n < 1 || p.ld < p.n) return false;
  const int tiles = (p.n + LZ_BLOCK - 1) / LZ_BLOCK;
  if (nctas < 1 || (tiles + nctas - 1) / nctas > WV_C || !ctl_fits(nctas)) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) { cudaGetLastError(); return false; }
  return cs == cudaStreamCaptureStatusNone;
}

// a stream kernel launched with programmatic stream serialisation (see
// st_pdl_prologue)
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), bool early, int grid, int cluster,
                              size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(LZ_BLOCK);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)cluster;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Stream path of one problem.  The host enqueues a cycle's steps (m - i of
// them, one more after a breakdown), the restart and the rotation, then reads
// the control block back once (a synchronisation of `stream`) to learn where
// the next cycle starts and whether the loop has ended.  The loop state is
// on the device, so a step that is not needed only returns.
template <typename VT>
static int run_stream(const DeviceInfo& di, const LanczosProblem& p, cudaStream_t stream) {
  if (p.m > MAXM || p.m < 1 || p.n < 1 || p.ld < p.n) {
    set_error("lanczos: unsupported sizes n=%d ld=%d m=%d (m must be in [1, %d])", p.n, p.ld,
              p.m, MAXM);
    return -2;
  }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    set_error("lanczos: a problem of n=%d rows reads its loop state back once per restart and "
              "cannot run inside a stream capture", p.n);
    return -2;
  }
  // the stream path's kernels take four rows of a column as 16-byte words
  if ((((uintptr_t)p.Q | (size_t)p.ld * sizeof(VT)) & 15) != 0) {
    set_error("lanczos: n=%d rows need Q and its columns (ld=%d) on 16-byte boundaries", p.n, p.ld);
    return -2;
  }
  const int ntiles = (p.n + LZ_BLOCK - 1) / LZ_BLOCK;
  // partials per pass
  const int G = lanczos_team_size(di, p.n, sizeof(VT) == 8 ? 64 : 32, true);
  const int* occ = stream_occ<VT>();
  // each kernel: at most one wave, and every CTA the same number of row
  // chunks (A2 and C use 4 rows per thread, B 8 bytes per thread), so no
  // CTA runs a last chunk alone
  int g[4];
  for (int j = 0; j < 4; ++j) {
    const int rows = (j == 1) ? (8 / (int)sizeof(VT)) * LZ_BLOCK : (j == 3 ? LZ_BLOCK : ST_ROWS);
    const int nch = (p.n + rows - 1) / rows;
    int gmax = di.sm_count * occ[j];
    if (gmax > G) gmax = G;
    if (gmax < 1) gmax = 1;
    const int per = (nch + gmax - 1) / gmax;
    g[j] = (nch + per - 1) / per;
    if (g[j] < 1) g[j] = 1;
  }
  TeamDesc<VT> t;
  char* w = fill_desc(t, p, G, true);
  StreamCtl* ctl = (StreamCtl*)((char*)t.part + ctl_offset(G));
  const int ns = (p.n + 31) / 32;
  t.wcap = sell_wcap(p.n, p.nnz);
  if ((long long)ns * 32 * t.wcap > 0x7fffffffLL) {
    set_error("lanczos: n=%d is too large for the stream path's operator layout", p.n);
    return -2;
  }
  t.sl_ptr = (int*)w; w += align256((size_t)(ns + 1) * sizeof(int));
  t.sl_row = (unsigned char*)w; w += align256((size_t)ns * 32);
  t.sl_col = (int*)w; w += align256((size_t)ns * 32 * t.wcap * sizeof(int));
  t.sl_val = (VT*)w;
  st_sell_order_kernel<VT><<<ntiles, LZ_BLOCK, 0, stream>>>(t);
  st_sell_scan_kernel<<<1, 1024, 0, stream>>>(ns, t.sl_ptr);
  st_sell_fill_kernel<VT><<<ntiles, LZ_BLOCK, 0, stream>>>(t);
  t_launches += 3;
  if (cudaMemsetAsync(ctl, 0, sizeof(StreamCtl), stream) != cudaSuccess ||
      cudaMemsetAsync(p.ctl, 0, 16 * sizeof(int), stream) != cudaSuccess) {
    set_error("lanczos: memset failed");
    return -4;
  }
  if (p.max_restarts == 0 || p.num_desired < 1) return 0;   // no cycle runs
  StreamCtl h;
  int i_host = 0, bd_host = 0;
  for (int guard = 0;; ++guard) {
    if (guard > 4 * p.max_restarts + 16) {
      set_error("lanczos: the stream path did not finish its %d restarts", p.max_restarts);
      return -5;
    }
    const int slots = (p.m - i_host) + (bd_host ? 1 : 0);
    cudaError_t e = cudaSuccess;
    for (int j = 0; j < slots && e == cudaSuccess; ++j) {
      e = launch_pdl(st_sell_spmv_kernel<VT>, true, ntiles, 1, 0, stream, t, ctl);
      if (e == cudaSuccess)
        e = launch_pdl(st_dot_kernel<VT>, true, DOT_G * g[0], 1, 0, stream, t, ctl);
      if (e == cudaSuccess)
        e = launch_pdl(st_update_dot1_kernel<VT>, true, g[1], 1, st_sacc_bytes<VT>(), stream, t, ctl);
      if (e == cudaSuccess)
        e = launch_pdl(st_update_norm_kernel<VT>, true, g[2], 1, 0, stream, t, ctl);
    }
    if (e == cudaSuccess) e = launch_pdl(st_restart_kernel<VT>, true, 1, 1, 0, stream, t, ctl);
    if (e == cudaSuccess) e = launch_pdl(st_rotate_kernel<VT>, true, g[3], 1, 0, stream, t, ctl);
    t_launches += 4 * slots + 2;
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error("lanczos: stream-path launch failed: %s", cudaGetErrorString(e));
      return -5;
    }
    if (cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess) {
      set_error("lanczos: stream-path state read failed: %s",
                cudaGetErrorString(cudaGetLastError()));
      return -5;
    }
    if (h.stop) break;
    i_host = h.i;
    bd_host = h.bd;
  }
  return 0;
}

// Most launches a call enqueues for the wave path.  A stream's queue holds 1,024
// launches (1,020 behind a waiting stream return in 8 ms, 1,100 when it goes on), and a
// call that stays below returns at once however busy its stream is.  It is room for 18
// cycles of 32 vectors, or for 8 of each of two problems.
constexpr int WV_LAUNCHES = 980;

// Wave path of one problem over R ranks: enqueues the launches of its first cycles, at
// most `budget` of them.  *resume receives the control block from which the team
// kernel continues (untouched if no cycle is enqueued).  After a restart at most
// delta = min(m - num_desired, 2 m / 5) vectors are dropped (restart_select), so a
// cycle takes at most that many steps, the first one m.  A launch past the loop's end
// costs about 1 us: n = 30,011 converging at the first of ten restarts takes 1.5 ms, at
// the fifth 3.1 (1.1 and 2.8 with a host that reads the state back and stops; 2.9 and
// 8.2 on the team kernel alone).
// The rotation and the next cycle's first launch wait for the kernel before them to
// end: started early they and, each started by the one before it, the next step's
// kernels would hold the SMs through the one-CTA restart.  Eight streams at once: 13.3
// ms with n = 30,011 in FP32 (16.0 with both early, 13.8 with the rotation early), 17.9
// with n = 15,000 in FP64 (27, 19.2); one alone 5.0 either way, 7.5 (8.0, 7.8).
template <typename VT>
static int enqueue_wave(const LanczosProblem& p, int R, int budget, cudaStream_t stream,
                        StreamCtl** resume) {
  const int more = p.m - p.num_desired < 2 * p.m / 5 ? p.m - p.num_desired : 2 * p.m / 5;
  if (p.max_restarts < 1 || p.num_desired < 1 || more < 0 || 4 * p.m + 2 > budget) return 0;
  TeamDesc<VT> t;
  fill_desc(t, p, R, false);
  StreamCtl* ctl = (StreamCtl*)((char*)t.part + ctl_offset(R));
  t.resume = ctl;
  if (cudaMemsetAsync(ctl, 0, sizeof(StreamCtl), stream) != cudaSuccess ||
      cudaMemsetAsync(p.ctl, 0, 16 * sizeof(int), stream) != cudaSuccess) {
    set_error("lanczos: memset failed");
    return -4;
  }
  const int ntiles = (p.n + LZ_BLOCK - 1) / LZ_BLOCK;
  int used = 0;
  for (int c = 0; c < p.max_restarts; ++c) {
    const int slots = c ? more : p.m;
    if (used + 4 * slots + 2 > budget) break;
    cudaError_t e = cudaSuccess;
    for (int j = 0; j < slots && e == cudaSuccess; ++j) {
      e = launch_pdl(wv_spmv_kernel<VT>, j > 0, (p.n + WV_ROWS - 1) / WV_ROWS, 1, 0, stream, t, ctl);
      if (e == cudaSuccess) e = launch_pdl(wv_dot_kernel<VT>, true, WV_C * R, 1, 0, stream, t, ctl);
      if (e == cudaSuccess)
        e = launch_pdl(wv_update_dot_kernel<VT>, true, WV_C * R, WV_C, 0, stream, t, ctl);
      if (e == cudaSuccess)
        e = launch_pdl(wv_update_norm_kernel<VT>, true, WV_C * R, WV_C, 0, stream, t, ctl);
    }
    if (e == cudaSuccess) e = launch_pdl(st_restart_kernel<VT>, true, 1, 1, 0, stream, t, ctl);
    if (e == cudaSuccess) e = launch_pdl(st_rotate_kernel<VT>, false, ntiles, 1, 0, stream, t, ctl);
    used += 4 * slots + 2;
    if (e != cudaSuccess) {
      set_error("lanczos: wave-path launch failed: %s", cudaGetErrorString(e));
      return -5;
    }
  }
  t_launches += used;
  *resume = ctl;
  return 0;
}

// team-kernel problems (x staged in shared memory) in batched cooperative
// launches; larger ones one after another on the stream path
template <typename VT>
static int run_noncluster(const DeviceInfo& di, const LanczosProblem* probs, int count,
                          cudaStream_t stream) {
  LanczosProblem team[MAX_TEAMS];
  for (int base = 0; base < count; base += MAX_TEAMS) {
    const int cnt = (count - base < MAX_TEAMS) ? (count - base) : MAX_TEAMS;
    int nt = 0;
    for (int i = 0; i < cnt; ++i) {
      const LanczosProblem& p = probs[base + i];
      if (x_fits_smem(p.n, sizeof(VT)) && !p.no_coop) {
        team[nt++] = p;
      } else {
        const int rc = run_stream<VT>(di, p, stream);
        if (rc) return rc;
      }
    }
    if (nt) {
      // one or two team-size problems: their cycles one after another on the wave
      // path, with the team sizes, and so the results, of the shared launch that
      // follows.  ms for one, two, three and four on it alone / in a shared launch,
      // whose time hardly depends on their number: FP32 n = 30,011 5.0, 10.8, 14.6, 19.0 /
      // 14.8; FP64 n = 20,000 8.4, 17.8, 25.8, 34.5 / 21.5.  More, or teams shrunk to fit one launch, share it
      const int occ = (sizeof(VT) == 8) ? di.lanczos_occ64 : di.lanczos_occ32;
      const int maxc = (di.sm_count > 4 ? di.sm_count - 2 : di.sm_count) * (occ > 0 ? occ : 1);
      int want[MAX_TEAMS], total = 0;
      StreamCtl* resume[MAX_TEAMS] = {};
      for (int i = 0; i < nt; ++i) {
        want[i] = lanczos_team_size(di, team[i].n, sizeof(VT) == 8 ? 64 : 32);
        total += want[i];
      }
      for (int i = 0; i < nt && nt <= 2 && total <= maxc; ++i)
        if (wave_fits<VT>(team[i], want[i], stream)) {
          const int rc = enqueue_wave<VT>(team[i], want[i], WV_LAUNCHES / nt, stream, &resume[i]);
          if (rc) return rc;
        }
      const int rc = run_typed<VT>(di, team, nt, stream, resume);
      if (rc) return rc;
    }
  }
  return 0;
}

// shared memory left for the cluster kernel's dynamic layout
template <typename VT>
constexpr size_t cl_budget() { return 227 * 1024 - sizeof(LzShared<VT>) - 1024; }
// ---- cluster-size policy and its autotuner ----
// A launch's cluster size is ceil(n_max / target) CTAs (at most 16), for a
// target number of rows per CTA.  Each step's phases scale with the rows per
// CTA and its cluster reductions with the CTAs, and clusters of one launch
// (or of concurrent solves) compete for the SMs: on GB300 a lone problem runs
// fastest spread over 16 CTAs (FP32 n = 5000: 4.8 ms at 16 CTAs, 8.7 ms at 8 when
// the line was drawn), while 48 problems in one launch run fastest packed at 640
// rows per CTA (17 ms against 27 ms spread then; 8.5 ms packed now).  A caller that knows its launch shares the
// GPU (a solve service) passes its own rows per CTA in the problem; otherwise
// the class's measured choice is used (usbs_lanczos_autotune times the
// candidates on a caller's batch and records the fastest for its precision,
// batch and size class), else 64 rows per CTA for one problem and 640 for a
// batch.
constexpr int TUNE_NCAND = 5;
constexpr int TUNE_CAND[TUNE_NCAND] = {64, 128, 256, 640, 1280};
static std::mutex g_tune_mu;
static std::map<long long, int> g_tune;            // class key -> rows per CTA
static thread_local int t_forced_target = 0;       // set by the tuner while it measures

static int log2_bucket(long long v) {
  int b = 0;
  while (v > 1) { v >>= 1; ++b; }
  return b;
}
// class key: precision << 32 | floor(log2(problems)) << 16 | floor(log2(largest n))
static long long tune_key(int prec, int count, int nmax) {
  return ((long long)prec << 32) | ((long long)log2_bucket(count < 1 ? 1 : count) << 16) |
         log2_bucket(nmax);
}
static int cl_target(int prec, int count, int nmax, int requested) {
  if (t_forced_target) return t_forced_target;
  if (requested > 0) return requested;
  if (const char* e = getenv(prec == 64 ? "USBS_CL_TARGET64" : "USBS_CL_TARGET32"))
    if (atoi(e) >= 32) return atoi(e);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find(tune_key(prec, count, nmax));
    if (it != g_tune.end()) return it->second;
  }
  return count <= 1 ? 64 : 640;
}
static int cl_csize_for(int n, int target) {
  const int c = (n + target - 1) / target;
  return c < 1 ? 1 : (c > CL_MAX_CTAS ? CL_MAX_CTAS : c);
}
template <typename VT>
inline int cl_csize(int n) {
  return cl_csize_for(n, cl_target(sizeof(VT) == 8 ? 64 : 32, 1, n, 0));
}
template <typename VT>
static bool cl_fits(int n, int m) {
  const int csize = cl_csize<VT>(n);
  if (csize > CL_MAX_CTAS || m > MAXM || m < 1 || n < 1) return false;
  const int rc = (n + csize - 1) / csize;
  return cl_layout<VT>(m, rc, 0).total <= cl_budget<VT>();
}

int lanczos_kernel_kind(int n, int m, int prec) {
  static const int enabled = [] {
    const char* e = getenv("USBS_LANCZOS_CLUSTER");
    return e ? atoi(e) : 1;
  }();
  if (enabled && (prec == 64 ? cl_fits<double>(n, m) : cl_fits<float>(n, m))) return 1;
  return x_fits_smem(n, prec == 64 ? 8 : 4) ? 0 : 2;
}

// Cluster path: every problem of the launch as one cluster of `csize` CTAs.
// Returns 1 if the problems do not fit (the caller then runs the team kernel),
// 0 on success, negative on a launch error.
template <typename VT>
static int run_cluster(const LanczosProblem* probs, int count, cudaStream_t stream) {
  static const int enabled = [] {
    const char* e = getenv("USBS_LANCZOS_CLUSTER");   // 0 forces the team kernel
    return e ? atoi(e) : 1;
  }();
  if (!enabled || count < 1 || count > MAX_TEAMS) return 1;
  constexpr size_t BUDGET = cl_budget<VT>();
  int nmax = 1, req = 0;
  for (int i = 0; i < count; ++i) {
    nmax = probs[i].n > nmax ? probs[i].n : nmax;
    req = probs[i].rows_per_cta > req ? probs[i].rows_per_cta : req;
  }
  const int csize = cl_csize_for(nmax, cl_target(sizeof(VT) == 8 ? 64 : 32, count, nmax, req));
  if (csize > CL_MAX_CTAS) return 1;
  ClusterBatch<VT> batch;
  batch.count = count;
  size_t dyn = 0;
  // the largest operators first: clusters start in launch order and a long one
  // started last runs alone
  int order[MAX_TEAMS];
  for (int i = 0; i < count; ++i) {
    int j = i;
    for (; j > 0 && probs[order[j - 1]].nnz < probs[i].nnz; --j) order[j] = order[j - 1];
    order[j] = i;
  }
  for (int i = 0; i < count; ++i) {
    const LanczosProblem& p = probs[order[i]];
    if (p.m > MAXM || p.m < 1 || p.n < 1 || p.ld < p.n) return 1;
    const int rc = (p.n + csize - 1) / csize;
    const ClLayout base = cl_layout<VT>(p.m, rc, 0);
    if (base.total > BUDGET) return 1;
    // whatever is left holds the operator slice (else it is read from L2)
    const int cap = (int)((BUDGET - base.total) / (sizeof(int) + sizeof(VT))) - 8;
    ClusterDesc<VT>& t = batch.t[i];
    t.n = p.n; t.ld = p.ld; t.m = p.m; t.num_desired = p.num_desired;
    t.max_restarts = p.max_restarts; t.tol = p.tol; t.nnz = p.nnz;
    t.lanes = lanczos_lanes(p.n, p.nnz);
    t.rc = rc;
    t.csr_cap = cap > 0 ? cap : 0;
    t.rowptr = p.rowptr; t.col = p.col; t.val = (const VT*)p.val;
    t.Q = (VT*)p.Q; t.alpha = p.alpha; t.beta = p.beta; t.ctl = p.ctl; t.status = p.status;
    const size_t tot = cl_layout<VT>(p.m, rc, t.csr_cap).total;
    dyn = tot > dyn ? tot : dyn;
  }
  batch.csize = csize;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute((const void*)lanczos_cluster_kernel<VT>,
                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaFuncSetAttribute((const void*)lanczos_cluster_kernel<VT>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BUDGET);
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(csize * count));
  cfg.blockDim = dim3(LZ_BLOCK);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int nclusters = 0;
  cudaLaunchConfig_t qcfg = cfg;     // the query needs no stream (this one may be capturing)
  qcfg.stream = nullptr;
  if (cudaOccupancyMaxActiveClusters(&nclusters, (const void*)lanczos_cluster_kernel<VT>, &qcfg) !=
          cudaSuccess || nclusters < 1) {
    cudaGetLastError();
    return 1;
  }
  for (int i = 0; i < count; ++i) {
    if (cudaMemsetAsync(probs[i].ctl, 0, 16 * sizeof(int), stream) != cudaSuccess) {
      set_error("lanczos: memset failed");
      return -4;
    }
  }
  cudaError_t e = cudaLaunchKernelEx(&cfg, lanczos_cluster_kernel<VT>, batch);
  ++t_launches;
  if (e != cudaSuccess) {
    set_error("lanczos: cluster launch (%d x %d CTAs) failed: %s", count, csize,
              cudaGetErrorString(e));
    return -5;
  }
  return 0;
}

int lanczos_last_launches() { return t_launches; }

int lanczos_run(const DeviceInfo& di, const LanczosProblem* probs, int count, int prec,
                cudaStream_t stream) {
  t_launches = 0;
  if (prec == 64) {
    const int rc = run_cluster<double>(probs, count, stream);
    if (rc <= 0) return rc;
    return run_noncluster<double>(di, probs, count, stream);
  }
  if (prec == 32) {
    const int rc = run_cluster<float>(probs, count, stream);
    if (rc <= 0) return rc;
    return run_noncluster<float>(di, probs, count, stream);
  }
  set_error("lanczos: precision must be 32 or 64");
  return -2;
}

int lanczos_tune_candidates(int i) { return (i >= 0 && i < TUNE_NCAND) ? TUNE_CAND[i] : 0; }

void lanczos_force_target(int target) { t_forced_target = target; }

// cluster size a launch of `count` problems of at most nmax rows gets with `target`
int lanczos_cluster_size(int nmax, int target) { return cl_csize_for(nmax, target); }

void lanczos_tune_record(int prec, int count, int nmax, int target) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (target > 0) g_tune[tune_key(prec, count, nmax)] = target;
  else g_tune.erase(tune_key(prec, count, nmax));
}

int lanczos_tune_entries(long long* keys, int* targets, int cap) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  int i = 0;
  for (const auto& kv : g_tune) {
    if (i < cap) { keys[i] = kv.first; targets[i] = kv.second; }
    ++i;
  }
  return i;
}

void lanczos_tune_clear() {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune.clear();
}

int lanczos_occupancy(int prec) {
  // occupancy with the largest staged x, so any launch stays co-resident
  int occ = 0;
  if (prec == 64) {
    cudaFuncSetAttribute((const void*)lanczos_team_kernel<double>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tm_dyn_max<double>());
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, lanczos_team_kernel<double>, LZ_BLOCK,
                                                  tm_dyn_max<double>());
  } else {
    cudaFuncSetAttribute((const void*)lanczos_team_kernel<float>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tm_dyn_max<float>());
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, lanczos_team_kernel<float>, LZ_BLOCK,
                                                  tm_dyn_max<float>());
  }
  return occ;
}

}  // namespace usbs
