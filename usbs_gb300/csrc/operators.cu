// Problem-data callbacks on the device (reference: solver/utils.py:11-37 and the
// Lanczos operator of solver/lanczos.py:86-87).
//
// Triples (constraint c, row i, column j, value a) are kept in two sorted
// copies prepared once on the host: by constraint (for A(.), a segmented
// reduction per constraint) and by row (for A*(.), a segmented reduction per
// output row).  Neither kernel needs atomics, so every sum has a fixed order.
// The Lanczos operator C + A*(w) is assembled once per eigsh call onto the
// union of C's pattern and the triples' (i, j) positions; the solver's SpMV then
// reads one CSR matrix.
#include "common.cuh"
#include "internal.h"

namespace usbs {

// (float)x rounded to nearest even, on the integer pipes for results that are
// normal floats (or round to infinity): a conversion from FP64 takes the SM's FP64
// unit 19 cycles per warp, like any FP64 instruction.
__device__ __forceinline__ float to_float_rn(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long m = b & 0x7fffffffffffffffull;
  const unsigned ex = (unsigned)(m >> 52);
  if (ex - 897u > 253u && m != 0ull) return (float)x;      // subnormal float, overflow, Inf, NaN
  unsigned r = 0u;
  if (m) r = (unsigned)((m + 0x0fffffffull + ((m >> 29) & 1ull)) >> 29) - (896u << 23);
  return __uint_as_float(r | ((unsigned)(b >> 32) & 0x80000000u));
}
template <typename OT> __device__ __forceinline__ OT out_of(double v);
template <> __device__ __forceinline__ double out_of<double>(double v) { return v; }
template <> __device__ __forceinline__ float out_of<float>(double v) { return to_float_rn(v); }

// alpha x without an FP64 instruction where alpha is 1 or -1 (sgn = 0 or the sign
// bit; 1 otherwise), as the solvers' operators are
__device__ __forceinline__ double scaled(double alpha, unsigned long long sgn, double x) {
  return (sgn == 1ull) ? alpha * x
                       : __longlong_as_double(__double_as_longlong(x) ^ (long long)sgn);
}

static unsigned long long sign_of_scale(double alpha) {
  return (alpha == 1.0) ? 0ull : (alpha == -1.0) ? 1ull << 63 : 1ull;
}

// The kernels below count entries, rows and triples in unsigned: the entry points take
// up to 2^31 - 1 of them, and a position plus a grid's stride stays below 2^32.
constexpr int AS_BLOCK = 256;

// out = alpha_c C + A*(w) on the pattern.  Entries that no triple lands on (seven of
// eight on a degree-7 graph) need no FP64 arithmetic; the others are listed per
// block and taken by whole warps, because an FP64 instruction costs its warp the
// same however few lanes have such an entry.  n = 10^6, 8.1e6 entries, FP32 out:
// 50 us (87 with every entry scaled, added to and converted in place).
template <typename OT, int AS_PER>      // AS_PER pattern entries per thread and round
__global__ void __launch_bounds__(AS_BLOCK) assemble_kernel(
    unsigned nnz, const double* __restrict__ c_val, double alpha_c, unsigned long long sgn,
    const int* __restrict__ slot_ptr, const int* __restrict__ slot_tid,
    const int* __restrict__ con, const double* __restrict__ a, const double* __restrict__ w,
    OT* __restrict__ out) {
  __shared__ unsigned list[AS_BLOCK * AS_PER];
  __shared__ int count;
  const bool has_c = alpha_c != 0.0 && c_val;
  constexpr unsigned CH = AS_BLOCK * AS_PER;
  for (unsigned base = blockIdx.x * CH; base < nnz; base += gridDim.x * CH) {
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    double v[AS_PER];
    int n0[AS_PER], n1[AS_PER];
#pragma unroll
    for (int u = 0; u < AS_PER; ++u) {
      const unsigned p = base + u * AS_BLOCK + threadIdx.x;
      v[u] = (has_c && p < nnz) ? c_val[p] : 0.0;
      n0[u] = n1[u] = 0;
      if (w && p < nnz) { n0[u] = slot_ptr[p]; n1[u] = slot_ptr[p + 1]; }
    }
#pragma unroll
    for (int u = 0; u < AS_PER; ++u) {
      const unsigned p = base + u * AS_BLOCK + threadIdx.x;
      const bool more = n1[u] > n0[u];
      const unsigned mb = __ballot_sync(0xffffffffu, more);
      int at = 0;
      if (mb && (threadIdx.x & 31) == 0) at = atomicAdd(&count, __popc(mb));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(mb & ((1u << (threadIdx.x & 31)) - 1u));
      if (more) list[at] = p;
      else if (p < nnz) out[p] = out_of<OT>(has_c ? scaled(alpha_c, sgn, v[u]) : 0.0);
    }
    __syncthreads();
    const int cnt = count;
    for (int i = threadIdx.x; i < cnt; i += AS_BLOCK) {
      const unsigned p = list[i];
      double x = has_c ? scaled(alpha_c, sgn, c_val[p]) : 0.0;
      const int e = slot_ptr[p + 1];
      for (int q = slot_ptr[p]; q < e; ++q) {
        const int t = slot_tid[q];
        x += a[t] * w[con[t]];
      }
      out[p] = out_of<OT>(x);
    }
    __syncthreads();
  }
}

template <typename OT>
static void assemble_launch(int nnz, const double* c_val, double alpha_c, const int* slot_ptr,
                            const int* slot_tid, const int* con, const double* a, const double* w,
                            OT* out, cudaStream_t stream) {
  const unsigned long long sgn = sign_of_scale(alpha_c);
  // four entries per thread once that still fills the GPU twice over
  const int per = (nnz >= 152 * 2048) ? 4 : 1;
  const unsigned ch = AS_BLOCK * per, need = ((unsigned)nnz + ch - 1) / ch;
  const int blocks = (int)(need < 152 * 16 ? need : 152 * 16);
  if (per == 4)
    assemble_kernel<OT, 4><<<blocks, AS_BLOCK, 0, stream>>>(nnz, c_val, alpha_c, sgn, slot_ptr,
                                                            slot_tid, con, a, w, out);
  else
    assemble_kernel<OT, 1><<<blocks, AS_BLOCK, 0, stream>>>(nnz, c_val, alpha_c, sgn, slot_ptr,
                                                            slot_tid, con, a, w, out);
}

int assemble_operator(int nnz, const double* c_val, double alpha_c, const int* slot_ptr,
                      const int* slot_tid, const int* con, const double* a, const double* w,
                      void* op_val, int prec, cudaStream_t stream) {
  if (nnz <= 0) return 0;
  if (prec == 64)
    assemble_launch(nnz, c_val, alpha_c, slot_ptr, slot_tid, con, a, w, (double*)op_val, stream);
  else
    assemble_launch(nnz, c_val, alpha_c, slot_ptr, slot_tid, con, a, w, (float*)op_val, stream);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("assemble_operator: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// y[row] = sum_p val[p] x[col[p]], L lanes per row (vector CSR)
template <typename VT, int L>
__global__ void csr_spmv_kernel(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                                const VT* __restrict__ val, const VT* __restrict__ x,
                                VT* __restrict__ y) {
  const int lanes_total = gridDim.x * blockDim.x;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lig = gid % L;
  const int lane = threadIdx.x & 31;
  const unsigned gmask = (L == 32) ? 0xffffffffu : (((1u << L) - 1u) << (lane & ~(L - 1)));
  for (unsigned row = gid / L; row < (unsigned)n; row += lanes_total / L) {
    VT s = (VT)0;
    const unsigned e = rowptr[row + 1];
    for (unsigned p = rowptr[row] + lig; p < e; p += L) s += val[p] * x[col[p]];
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(gmask, s, o, L);
    if (lig == 0) y[row] = s;
  }
}

template <typename VT>
static void spmv_dispatch(int L, int blocks, int threads, cudaStream_t st, int n, const int* rp,
                          const int* c, const VT* v, const VT* x, VT* y) {
  switch (L) {
    case 1: csr_spmv_kernel<VT, 1><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
    case 2: csr_spmv_kernel<VT, 2><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
    case 4: csr_spmv_kernel<VT, 4><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
    case 8: csr_spmv_kernel<VT, 8><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
    case 16: csr_spmv_kernel<VT, 16><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
    default: csr_spmv_kernel<VT, 32><<<blocks, threads, 0, st>>>(n, rp, c, v, x, y); break;
  }
}

int csr_spmv(int n, long long nnz, const int* rowptr, const int* col, const void* val,
             const void* x, void* y, int prec, int sm_count, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int L = lanczos_lanes(n, nnz);
  const int threads = 256;
  long long need = ((long long)n * L + threads - 1) / threads;
  int blocks = (int)(need < (long long)sm_count * 8 ? need : (long long)sm_count * 8);
  if (blocks < 1) blocks = 1;
  if (prec == 64)
    spmv_dispatch<double>(L, blocks, threads, stream, n, rowptr, col, (const double*)val,
                          (const double*)x, (double*)y);
  else
    spmv_dispatch<float>(L, blocks, threads, stream, n, rowptr, col, (const float*)val,
                         (const float*)x, (float*)y);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("csr_spmv: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// y = (alpha_c C + A*(w)) x without storing the operator: each entry's value is
// formed as assemble_kernel forms it (rounded to VT), and the row is summed as
// csr_spmv_kernel sums it, so the result is that of the two kernels.  One apply
// then reads the pattern once and writes y, one launch: n = 10^6, 8.1e6 entries,
// FP32: 84 us (89 as two kernels); n = 800, degree 48, FP64: 16 us a call (37 as two
// launches and an allocation for the values).  (The Lanczos path applies one operator a hundred
// times and keeps the assembled values.)
template <typename VT, int L>
__global__ void __launch_bounds__(256) fused_apply_kernel(
    int n, const int* __restrict__ rowptr, const int* __restrict__ col,
    const double* __restrict__ c_val, double alpha_c, unsigned long long sgn,
    const int* __restrict__ slot_ptr, const int* __restrict__ slot_tid,
    const int* __restrict__ con, const double* __restrict__ a, const double* __restrict__ w,
    const VT* __restrict__ x, VT* __restrict__ y) {
  const bool has_c = alpha_c != 0.0 && c_val;
  const int lanes_total = gridDim.x * blockDim.x;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lig = gid % L;
  const int lane = threadIdx.x & 31;
  const unsigned gmask = (L == 32) ? 0xffffffffu : (((1u << L) - 1u) << (lane & ~(L - 1)));
  constexpr int U = 2;                             // entries in flight per lane
  for (unsigned row = gid / L; row < (unsigned)n; row += lanes_total / L) {
    VT s = (VT)0;
    const unsigned e = rowptr[row + 1];
    for (unsigned p0 = rowptr[row] + lig; p0 < e; p0 += U * L) {
      double v[U];
      VT xv[U];
      int b[U], f[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned p = min(p0 + u * L, e - 1);
        v[u] = has_c ? scaled(alpha_c, sgn, c_val[p]) : 0.0;
        xv[u] = x[col[p]];
        b[u] = f[u] = 0;
        if (w) { b[u] = slot_ptr[p]; f[u] = slot_ptr[p + 1]; }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (p0 + u * L < e) {
          for (int q = b[u]; q < f[u]; ++q) {
            const int t = slot_tid[q];
            v[u] += a[t] * w[con[t]];
          }
          s += out_of<VT>(v[u]) * xv[u];
        }
    }
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(gmask, s, o, L);
    if (lig == 0) y[row] = s;
  }
}

template <typename VT>
static void fused_dispatch(int L, int blocks, cudaStream_t st, int n, const int* rp, const int* c,
                           const double* cv, double alpha, unsigned long long sgn, const int* sp,
                           const int* sid, const int* con, const double* a, const double* w,
                           const VT* x, VT* y) {
  auto go = [&](auto kern) {
    kern<<<blocks, 256, 0, st>>>(n, rp, c, cv, alpha, sgn, sp, sid, con, a, w, x, y);
  };
  switch (L) {
    case 1: go(fused_apply_kernel<VT, 1>); break;
    case 2: go(fused_apply_kernel<VT, 2>); break;
    case 4: go(fused_apply_kernel<VT, 4>); break;
    case 8: go(fused_apply_kernel<VT, 8>); break;
    case 16: go(fused_apply_kernel<VT, 16>); break;
    default: go(fused_apply_kernel<VT, 32>); break;
  }
}

int fused_apply(int n, long long nnz, const int* rowptr, const int* col, const double* c_val,
                double alpha_c, const int* slot_ptr, const int* slot_tid, const int* con,
                const double* a, const double* w, const void* x, void* y, int prec, int sm_count,
                cudaStream_t stream) {
  if (n <= 0) return 0;
  const int L = lanczos_lanes(n, nnz);
  const unsigned long long sgn = sign_of_scale(alpha_c);
  const long long need = ((long long)n * L + 255) / 256;
  int blocks = (int)(need < (long long)sm_count * 32 ? need : (long long)sm_count * 32);
  if (blocks < 1) blocks = 1;
  if (prec == 64)
    fused_dispatch<double>(L, blocks, stream, n, rowptr, col, c_val, alpha_c, sgn, slot_ptr,
                           slot_tid, con, a, w, (const double*)x, (double*)y);
  else
    fused_dispatch<float>(L, blocks, stream, n, rowptr, col, c_val, alpha_c, sgn, slot_ptr,
                          slot_tid, con, a, w, (const float*)x, (float*)y);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("fused_apply: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// ------------------------------------------------------------------------
// Sliced-ELL operator apply.  Rows are grouped in windows of SELL_WIN = 256
// rows; inside a window they are sorted by length (longest first) and cut into
// 8 slices of 32 rows.  A slice stores its entries column-major (entry k of
// the slice's row r at sl_ptr[s] + 32 k + r), padded to the slice's longest
// row with column 0 and value 0.  One block per window, one warp per slice,
// lane = row: every load of col / val is a coalesced 128-byte line, and all of
// a row's loads are independent (no rowptr -> col -> x chain).  sl_row[32 s + r]
// is the row's position inside its window; results pass through shared memory
// so y is written in the original order, coalesced.
constexpr int SELL_WIN = 256;

template <typename VT>
__global__ void __launch_bounds__(SELL_WIN) sell_spmv_kernel(int n, const int* __restrict__ sl_ptr,
                                                           const int* __restrict__ col,
                                                           const VT* __restrict__ val,
                                                           const unsigned char* __restrict__ sl_row,
                                                           const VT* __restrict__ x,
                                                           VT* __restrict__ y) {
  __shared__ VT ys[SELL_WIN];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = blockIdx.x * (SELL_WIN / 32) + warp;
  const int w0 = blockIdx.x * SELL_WIN;
  const int nslices = (n + 31) / 32;
  VT acc = (VT)0;
  if (s < nslices) {
    const int base = sl_ptr[s], width = (sl_ptr[s + 1] - base) >> 5;
    const int* cp = col + base + lane;
    const VT* vp = val + base + lane;
    // the first SELL_PF entries of the row: every col / val load, then every
    // x gather, in flight at once; longer rows finish in a plain loop
    constexpr int SELL_PF = 16;
    int c[SELL_PF];
    VT v[SELL_PF], xv[SELL_PF];
#pragma unroll
    for (int u = 0; u < SELL_PF; ++u) {
      c[u] = (u < width) ? __ldg(cp + 32 * u) : 0;
      v[u] = (u < width) ? __ldg(vp + 32 * u) : (VT)0;
    }
#pragma unroll
    for (int u = 0; u < SELL_PF; ++u) xv[u] = (u < width) ? __ldg(x + c[u]) : (VT)0;
#pragma unroll
    for (int u = 0; u < SELL_PF; ++u) acc += v[u] * xv[u];
    for (int k = SELL_PF; k < width; ++k) acc += __ldg(vp + 32 * k) * __ldg(x + __ldg(cp + 32 * k));
    ys[sl_row[32 * s + lane]] = acc;
  }
  __syncthreads();
  const int r = w0 + threadIdx.x;
  if (r < n) y[r] = ys[threadIdx.x];
}

int sell_spmv(int n, const int* sl_ptr, const int* col, const void* val,
              const unsigned char* sl_row, const void* x, void* y, int prec, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int blocks = (n + SELL_WIN - 1) / SELL_WIN;
  if (prec == 64)
    sell_spmv_kernel<double><<<blocks, SELL_WIN, 0, stream>>>(n, sl_ptr, col, (const double*)val,
                                                            sl_row, (const double*)x, (double*)y);
  else
    sell_spmv_kernel<float><<<blocks, SELL_WIN, 0, stream>>>(n, sl_ptr, col, (const float*)val,
                                                           sl_row, (const float*)x, (float*)y);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("sell_spmv: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// Streaming reference for the SpMV's bandwidth: one pass over a (int4 words)
// and b (float4 words) with 16-byte loads, grid-stride, no gathers; block k
// writes the sum of the floats it read to out_sum[k] and the XOR of the words
// it read to out_xor[k].  Timed like the SpMV (one launch after an L2 flush),
// it shows what a kernel moving the same bytes can reach at that size.
__global__ void __launch_bounds__(256) stream_probe_kernel(long long na, const int4* __restrict__ a,
                                                           long long nb, const float4* __restrict__ b,
                                                           float* __restrict__ out_sum,
                                                           unsigned* __restrict__ out_xor) {
  __shared__ float ssum[8];
  __shared__ unsigned sxor[8];
  float acc = 0.f;
  unsigned x = 0u;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long nmax = na > nb ? na : nb;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nmax; i += stride) {
    if (i < na) {
      const int4 u = __ldg(a + i);
      x ^= (unsigned)u.x ^ (unsigned)u.y ^ (unsigned)u.z ^ (unsigned)u.w;
    }
    if (i < nb) {
      const float4 v = __ldg(b + i);
      acc += (v.x + v.y) + (v.z + v.w);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, o);
    x ^= __shfl_xor_sync(0xffffffffu, x, o);
  }
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { ssum[warp] = acc; sxor[warp] = x; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    unsigned u = 0u;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { t += ssum[w]; u ^= sxor[w]; }
    out_sum[blockIdx.x] = t;
    out_xor[blockIdx.x] = u;
  }
}

int stream_probe(long long a_words, const void* a, long long b_words, const void* b, int blocks,
                 float* out_sum, unsigned* out_xor, cudaStream_t stream) {
  if (blocks < 1) return 0;
  stream_probe_kernel<<<blocks, 256, 0, stream>>>(a_words, (const int4*)a, b_words,
                                                  (const float4*)b, out_sum, out_xor);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("stream_probe: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// dst[e] = src[map[e]] (0 where map[e] < 0): operator values from CSR to sliced-ELL order
template <typename VT>
__global__ void gather_values_kernel(long long total, const int* __restrict__ map,
                                     const VT* __restrict__ src, VT* __restrict__ dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int m = map[e];
    dst[e] = (m >= 0) ? src[m] : (VT)0;
  }
}

int gather_values(long long total, const int* map, const void* src, void* dst, int prec,
                  cudaStream_t stream) {
  if (total <= 0) return 0;
  long long b = (total + 255) / 256;
  const int blocks = (int)(b < 152 * 16 ? b : 152 * 16);
  if (prec == 64)
    gather_values_kernel<double><<<blocks, 256, 0, stream>>>(total, map, (const double*)src, (double*)dst);
  else
    gather_values_kernel<float><<<blocks, 256, 0, stream>>>(total, map, (const float*)src, (float*)dst);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("gather_values: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// a_t U[i_t, :] . U[j_t, :]
__device__ __forceinline__ double triple_value(unsigned t, const int* __restrict__ t_row,
                                               const int* __restrict__ t_col,
                                               const double* __restrict__ a,
                                               const double* __restrict__ U, int ldu, int k) {
  const int i = t_row[t], j = t_col[t];
  double d = 0.0;
  for (int q = 0; q < k; ++q) d += U[(size_t)q * ldu + i] * U[(size_t)q * ldu + j];
  return fma(a[t], d, 0.0);
}

// out[c] = sum_{t in constraint c} a_t * U[i_t, :] . U[j_t, :]: triples dealt to 32
// accumulators (every 32nd to the same one) that are added pairwise at distance
// 16, 8, 4, 2, 1.  Constraints of at most AO_SHORT triples take one thread each
// (its few accumulators in registers, the tree's additions of nothing left out),
// longer ones one warp.  With a warp for each of the QAP's 3.4e5 constraints, of
// mostly two triples, the FP64 unit added zeros: 170 us at l = 30, k = 2; 18 now.
constexpr int AO_SHORT = 8;
__global__ void __launch_bounds__(256) A_operator_kernel(
    int m, const int* __restrict__ con_ptr, const int* __restrict__ t_row,
    const int* __restrict__ t_col, const double* __restrict__ a, const double* __restrict__ U,
    int ldu, int k, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int total = gridDim.x * blockDim.x, warps = total >> 5;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x, wid = gid >> 5;
  // long constraints: each lane looks at one, far from its neighbours' (long ones
  // come in runs), and the warp takes those it found one by one
  for (long long c0 = wid; c0 < m; c0 += 32ll * warps) {
    const long long c = c0 + (long long)lane * warps;
    int b = 0, e = 0;
    if (c < m) { b = con_ptr[c]; e = con_ptr[c + 1]; }
    unsigned todo = __ballot_sync(0xffffffffu, e - b > AO_SHORT);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const unsigned tb = __shfl_sync(0xffffffffu, b, src), te = __shfl_sync(0xffffffffu, e, src);
      double s = 0.0;
      for (unsigned t = tb + lane; t < te; t += 32) {
        const int i = t_row[t], j = t_col[t];
        double d = 0.0;
        for (int q = 0; q < k; ++q) d += U[(size_t)q * ldu + i] * U[(size_t)q * ldu + j];
        s += a[t] * d;
      }
      s = warp_sum(s);
      if (lane == 0) out[c0 + (long long)src * warps] = s;
    }
  }
  for (unsigned c = gid; c < (unsigned)m; c += total) {
    const int b = con_ptr[c], cnt = con_ptr[c + 1] - b;
    if (cnt > AO_SHORT) continue;
    double v[AO_SHORT];
#pragma unroll
    for (int u = 0; u < AO_SHORT; ++u)
      v[u] = (u < cnt) ? triple_value(b + u, t_row, t_col, a, U, ldu, k) : 0.0;
#pragma unroll
    for (int o = AO_SHORT / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int u = 0; u < o; ++u)
        if (u + o < cnt) v[u] += v[u + o];
    }
    out[c] = v[0];
  }
}

int apply_A_operator(int m, const int* con_ptr, const int* t_row, const int* t_col,
                     const double* a, const double* U, int ldu, int k, double* out,
                     cudaStream_t stream) {
  if (m <= 0) return 0;
  const int threads = 256;
  long long need = ((long long)m * 32 + threads - 1) / threads;       // a warp per constraint
  int blocks = (int)(need < 152 * 8 ? need : 152 * 8);
  A_operator_kernel<<<blocks, threads, 0, stream>>>(m, con_ptr, t_row, t_col, a, U, ldu, k, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("apply_A_operator: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

// out[i, q] = sum_{t with row i} a_t z[c_t] U[j_t, q], summed as A_operator_kernel
// sums: 32 accumulators, then pairwise.  Rows of at most AO_SHORT triples (one in
// MaxCut) take one thread for all columns, longer ones (the QAP's hold about 900,
// the lifted row several thousand) one warp per column, because a warp gets one
// FP64 instruction per 60 cycles; eight triples' loads in flight per lane.
__global__ void __launch_bounds__(256) A_adjoint_kernel(
    int n, const int* __restrict__ row_ptr, const int* __restrict__ r_con,
    const int* __restrict__ r_col, const double* __restrict__ r_a, const double* __restrict__ z,
    const double* __restrict__ U, int ldu, int k, double* __restrict__ out, int ldo) {
  const int lane = threadIdx.x & 31;
  const int total = gridDim.x * blockDim.x, warps = total >> 5;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x, wid = gid >> 5;
  const long long tasks = (long long)n * k;        // (row, column), column fastest
  for (long long w0 = wid; w0 < tasks; w0 += 32ll * warps) {
    const long long w = w0 + (long long)lane * warps;
    int b = 0, e = 0;
    if (w < tasks) { b = row_ptr[w / k]; e = row_ptr[w / k + 1]; }
    unsigned todo = __ballot_sync(0xffffffffu, e - b > AO_SHORT);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const long long ws = w0 + (long long)src * warps;
      const int i = (int)(ws / k), q = (int)(ws - (long long)i * k);
      const unsigned tb = __shfl_sync(0xffffffffu, b, src), te = __shfl_sync(0xffffffffu, e, src);
      const double* Uq = U + (size_t)q * ldu;
      double s = 0.0;
      for (unsigned t = tb + lane; t < te; t += 256) {
        double av[8], zv[8], uv[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const unsigned th = min(t + 32 * h, te - 1);
          av[h] = r_a[th];
          zv[h] = z[r_con[th]];
          uv[h] = Uq[r_col[th]];
        }
#pragma unroll
        for (int h = 0; h < 8; ++h)
          if (t + 32 * h < te) s += av[h] * zv[h] * uv[h];
      }
      s = warp_sum(s);
      if (lane == 0) out[(size_t)q * ldo + i] = s;
    }
  }
  for (unsigned i = gid; i < (unsigned)n; i += total) {
    const int b = row_ptr[i], cnt = row_ptr[i + 1] - b;
    if (cnt > AO_SHORT) continue;
    double az[AO_SHORT];
    int col[AO_SHORT];
#pragma unroll
    for (int u = 0; u < AO_SHORT; ++u) {
      az[u] = 0.0;
      col[u] = 0;
      if (u < cnt) {
        az[u] = r_a[b + u] * z[r_con[b + u]];
        col[u] = r_col[b + u];
      }
    }
    for (int q = 0; q < k; ++q) {
      const double* Uq = U + (size_t)q * ldu;
      double v[AO_SHORT];
#pragma unroll
      for (int u = 0; u < AO_SHORT; ++u) v[u] = (u < cnt) ? fma(az[u], Uq[col[u]], 0.0) : 0.0;
#pragma unroll
      for (int o = AO_SHORT / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int u = 0; u < o; ++u)
          if (u + o < cnt) v[u] += v[u + o];
      }
      out[(size_t)q * ldo + i] = v[0];
    }
  }
}

int apply_A_adjoint(int n, const int* row_ptr, const int* r_con, const int* r_col,
                    const double* r_a, const double* z, const double* U, int ldu, int k,
                    double* out, int ldo, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int threads = 256;
  long long need = ((long long)n * k * 32 + threads - 1) / threads;   // a warp per (row, column)
  if (need < 1) need = 1;
  int blocks = (int)(need < 152 * 8 ? need : 152 * 8);
  A_adjoint_kernel<<<blocks, threads, 0, stream>>>(n, row_ptr, r_con, r_col, r_a, z, U, ldu, k,
                                                   out, ldo);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("apply_A_adjoint: %s", cudaGetErrorString(e)); return -5; }
  return 0;
}

}  // namespace usbs
