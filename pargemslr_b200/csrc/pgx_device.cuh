// Device-side building blocks of the GeMSLR-FGMRES solve phase (sm_100a).
//
// Every kernel takes a Skip descriptor: up to three device flags (the
// "cycle finished" / "solve finished" words of the enclosing FGMRES solves).
// A kernel whose flags are set returns at once, so a whole restart cycle can
// be enqueued (or captured in a CUDA graph) ahead of time and the iterations
// after convergence cost one launch each and no memory traffic.
#pragma once

#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pgx_complex.cuh"

namespace pgx {

using ::__shfl_xor_sync;  // the real forms beside the complex overload

constexpr int kWarp = 32;
constexpr int KMAX = 128;          // largest Krylov dimension a handle accepts
constexpr int kMaxLanes = 16;      // right-hand sides one slot advances together
constexpr int kTsThreads = 512;    // block size of the tall-skinny kernels
constexpr int kTsMaxBlocks = 296;  // 2 blocks per SM on a 148-SM B200
constexpr int kSpinLimit = 1 << 21;  // default bound of the waits in the sync-free triangular solves

// status bits written by kernels into the handle's error word
constexpr int kErrTimeout = 1;  // a dependency wait of a cross-subdomain triangular solve gave up
constexpr int kErrIndex = 2;    // an index check failed
constexpr int kErrStage = 4;    // a staging wait of the per-subdomain triangular solve gave up

struct Skip {
  const int* f0;
  const int* f1;
  const int* f2;
  __device__ __forceinline__ bool on() const {
    return (f0 && *(const volatile int*)f0) || (f1 && *(const volatile int*)f1) ||
           (f2 && *(const volatile int*)f2);
  }
};

// Skip flags of R solves advancing together: a kernel shared by them returns
// only when every one of them is skipped.
template <int R>
struct SkipR {
  Skip s[R];
  __device__ __forceinline__ bool on() const {
#pragma unroll
    for (int r = 0; r < R; r++)
      if (!s[r].on()) return false;
    return true;
  }
};

// ---------------------------------------------------------------- FGMRES
// Device-resident state of one flexible GMRES solve (FlexGmresClass::Solve,
// ParGeMSLR SRC/solvers/fgmres.hpp:263-558).  H is column-major (KMAX+1) x KMAX.
// S is the solver's scalar: double, or cf64 for a complex solve (Hessenberg,
// rotations and right-hand side of the least-squares problem complex; norms,
// tolerances and the lazy column scales real).  The header up to sc has the
// same layout for both.
template <typename S>
struct FgmresDevT {
  int done;        // solve finished (converged, max iterations or breakdown)
  int cycle_done;  // current restart cycle finished
  int breakdown;   // Givens breakdown: the reference skips the x update
  int converged;
  int iter;        // iterations so far (FlexGmresClass::_iter)
  int i;           // columns built in the current cycle
  int kdim;
  int maxits;
  double tolr;     // absolute threshold on the Givens residual estimate
  double tol;
  double normb;
  double normr;    // Givens residual estimate (reference: normr)
  double normr0;   // ||r0|| at the start of the solve (first entry of the residual history)
  double eps;      // numeric_limits<RealDataType>::epsilon() of the solver
  int absolute;
  int pad;
  double sc[KMAX + 1];     // V(:,c) = Vstored(:,c) * sc[c] (lazy normalisation)
  double hist[KMAX];       // Givens estimate after each column of the current cycle (0 at a breakdown)
  S hcol[KMAX + 1];   // column of H being built
  S coefA[KMAX + 1];  // first Gram-Schmidt coefficients
  S coefB[KMAX + 1];  // re-orthogonalisation coefficients
  S c[KMAX], s[KMAX], rs[KMAX + 1], y[KMAX];
  S H[(KMAX + 1) * KMAX];
};
using FgmresDev = FgmresDevT<double>;

template <typename T>
__device__ __forceinline__ T ldg(const T* p) { return __ldg(p); }
template <>
__device__ __forceinline__ cf32 ldg<cf32>(const cf32* p) {
  const float2 v = __ldg((const float2*)p);
  return cf32(v.x, v.y);
}
template <>
__device__ __forceinline__ cf64 ldg<cf64>(const cf64* p) {
  const double2 v = __ldg((const double2*)p);
  return cf64(v.x, v.y);
}
template <typename T>
__device__ __forceinline__ T ldcg(const T* p) { return __ldcg(p); }
template <>
__device__ __forceinline__ cf32 ldcg<cf32>(const cf32* p) {
  const float2 v = __ldcg((const float2*)p);
  return cf32(v.x, v.y);
}
template <>
__device__ __forceinline__ cf64 ldcg<cf64>(const cf64* p) {
  const double2 v = __ldcg((const double2*)p);
  return cf64(v.x, v.y);
}

template <typename T>
__device__ __forceinline__ T group_reduce(T v, int S, int lane) {
  // sum over this lane's aligned group of S lanes; only that group's lanes
  // take part, so other groups of the warp may be elsewhere (spinning)
  const unsigned mask = S == 32 ? 0xffffffffu : (((1u << S) - 1u) << (lane & ~(S - 1)));
  for (int off = S >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(mask, v, off);
  return v;
}

// Products and sums whose rounding is spelled out, so that a single-lane
// kernel and its multi-lane form cannot be contracted differently: a slot's
// results do not depend on its lane count.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ void mac(float& acc, float v, float w) { acc = fmaf(v, w, acc); }
__device__ __forceinline__ void mac(double& acc, double v, double w) { acc = fma(v, w, acc); }
template <typename R>
__device__ __forceinline__ cplx<R> mul_rn(const cplx<R>& a, const cplx<R>& b) {
  cplx<R> t(mul_rn(a.x, b.x), mul_rn(a.x, b.y));
  t.x = fma(-a.y, b.y, t.x);
  t.y = fma(a.y, b.x, t.y);
  return t;
}
// The product is formed first and added with one rounding at the sum's size.
// Two multiply-adds into the sum round twice there: in a CPU model of a lower
// pass, 67 / 201 entries a row, the error was 1.1 / 1.2 times this one's.
template <typename R>
__device__ __forceinline__ void mac(cplx<R>& acc, const cplx<R>& v, const cplx<R>& w) {
  const cplx<R> t = mul_rn(v, w);
  acc.x += t.x;
  acc.y += t.y;
}
__device__ __forceinline__ cf64 mul_rn(const cf64& a, double s) { return cf64(__dmul_rn(a.x, s), __dmul_rn(a.y, s)); }
__device__ __forceinline__ double abs2_rn(double v) { return __dmul_rn(v, v); }
__device__ __forceinline__ double abs2_rn(const cf64& v) { return fma(v.x, v.x, __dmul_rn(v.y, v.y)); }

// lane l's value for the whole warp
__device__ __forceinline__ double bcast(double v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ cf64 bcast(const cf64& v, int l) {
  return cf64(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}

template <typename T>
__device__ __forceinline__ T warp_reduce(T v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// ------------------------------------------------------------ CSR SpMV
// y = alpha * (A1 x1) + alpha2 * (A2 x2) + beta * b, S lanes per row.
// A2 may be absent (rp2 == nullptr); b may be absent or alias y.
// Follows CsrMatrixPMatVecHostTemplate (ParGeMSLR SRC/matrices/matrixops.cpp:5139)
// for one matrix; the two-matrix form fuses the Schur operator
// C x - E (B^-1 F x) of GemslrClass::SchurMatVec (gemslr.cpp:3799-3960).
// Each lane issues the loads of its first kSpmvUnroll column indices, then
// of the x entries they name, before it multiplies: the gathers of x are in
// flight together.  A lane sums its entries in increasing order either way.
constexpr int kSpmvUnroll = 4;

template <typename TA, typename TX, typename TC, int S>
__device__ __forceinline__ TC row_dot(int k1, int k2, int lane, const int* __restrict__ cj, const TA* __restrict__ va,
                                      const TX* __restrict__ x, int xcols, bool& bad) {
  int c[kSpmvUnroll];
  TA v[kSpmvUnroll];
#pragma unroll
  for (int u = 0; u < kSpmvUnroll; u++) {
    const int k = k1 + lane + u * S;
    c[u] = k < k2 ? __ldg(&cj[k]) : -1;
    v[u] = k < k2 ? ldg(&va[k]) : TA(0);
    if (k < k2 && (unsigned)c[u] >= (unsigned)xcols) {
      bad = true;  // a column outside x: the entry is skipped
      c[u] = -1;
    }
  }
  TX xv[kSpmvUnroll];
#pragma unroll
  for (int u = 0; u < kSpmvUnroll; u++) xv[u] = c[u] >= 0 ? x[c[u]] : TX(0);
  TC acc = 0;
#pragma unroll
  for (int u = 0; u < kSpmvUnroll; u++)
    if (c[u] >= 0) mac(acc, (TC)v[u], (TC)xv[u]);
  for (int k = k1 + lane + kSpmvUnroll * S; k < k2; k += S) {
    const int cc = __ldg(&cj[k]);
    if ((unsigned)cc < (unsigned)xcols)
      mac(acc, (TC)ldg(&va[k]), (TC)x[cc]);
    else
      bad = true;
  }
  return acc;
}

// The same dot product with 128-bit loads: the row's entries [k1, k2) lie in
// the aligned 4-entry blocks k1/4 .. (k2+3)/4 - 1; the S lanes take the
// blocks in turn, each loading a block's column indices as one int4 and its
// values as one float4 or two double2, and mask the entries outside the row.
// Needs cj and va 16-byte aligned and padded to a whole last block (the
// library's own uploads are).  A lane sums its entries in increasing order.
template <typename TA>
__device__ __forceinline__ void load_block4(const TA* __restrict__ p, TA* v);
template <>
__device__ __forceinline__ void load_block4<float>(const float* __restrict__ p, float* v) {
  const float4 a = __ldg((const float4*)p);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
}
template <>
__device__ __forceinline__ void load_block4<double>(const double* __restrict__ p, double* v) {
  const double2 a = __ldg((const double2*)p), b = __ldg((const double2*)p + 1);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}

template <>
__device__ __forceinline__ void load_block4<cf32>(const cf32* __restrict__ p, cf32* v) {
  const float4 a = __ldg((const float4*)p), b = __ldg((const float4*)p + 1);
  v[0] = cf32(a.x, a.y);
  v[1] = cf32(a.z, a.w);
  v[2] = cf32(b.x, b.y);
  v[3] = cf32(b.z, b.w);
}
template <>
__device__ __forceinline__ void load_block4<cf64>(const cf64* __restrict__ p, cf64* v) {
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const double2 a = __ldg((const double2*)p + u);
    v[u] = cf64(a.x, a.y);
  }
}

template <typename TA, typename TX, typename TC, int S>
__device__ __forceinline__ TC row_dot_vec(int k1, int k2, int lane, const int* __restrict__ cj,
                                          const TA* __restrict__ va, const TX* __restrict__ x, int xcols, bool& bad) {
  TC acc = 0;
  const int b1 = (k2 + 3) >> 2;
  for (int bb = (k1 >> 2) + lane; bb < b1; bb += S) {
    const int kb = bb << 2;
    const int4 c4 = __ldg((const int4*)cj + bb);
    TA v[4];
    load_block4<TA>(va + kb, v);
    const int c[4] = {c4.x, c4.y, c4.z, c4.w};
    bool in[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      in[u] = kb + u >= k1 && kb + u < k2;
      if (in[u] && (unsigned)c[u] >= (unsigned)xcols) {
        bad = true;  // a column outside x: the entry is skipped
        in[u] = false;
      }
    }
    TX xv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) xv[u] = in[u] ? x[c[u]] : TX(0);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (in[u]) mac(acc, (TC)v[u], (TC)xv[u]);
  }
  return acc;
}

template <typename TA, typename TX, typename TY, typename TC, int S, bool VEC>
__device__ __forceinline__ void spmv_rows(
    int nrows, const int* __restrict__ rp1, const int* __restrict__ cj1, const TA* __restrict__ va1,
    const TX* __restrict__ x1, int xcols1, TC alpha, const int* __restrict__ rp2, const int* __restrict__ cj2,
    const TA* __restrict__ va2, const TX* __restrict__ x2, int xcols2, TC alpha2, const TY* b, TC beta, TY* y,
    const double* __restrict__ xscale, int* err) {
  const int lane = threadIdx.x & (S - 1);
  const int wlane = threadIdx.x & 31;
  const int groups_per_block = blockDim.x / S;
  const TC xs = xscale ? (TC)(*xscale) : (TC)1;
  bool bad = false;
  for (int row = blockIdx.x * groups_per_block + threadIdx.x / S; row < nrows;
       row += gridDim.x * groups_per_block) {
    const int k1 = __ldg(&rp1[row]), k2 = __ldg(&rp1[row + 1]);
    TC acc = VEC ? row_dot_vec<TA, TX, TC, S>(k1, k2, lane, cj1, va1, x1, xcols1, bad)
                 : row_dot<TA, TX, TC, S>(k1, k2, lane, cj1, va1, x1, xcols1, bad);
    acc = group_reduce(acc, S, wlane);
    TC acc2 = 0;
    if (rp2) {
      const int q1 = __ldg(&rp2[row]), q2 = __ldg(&rp2[row + 1]);
      acc2 = VEC ? row_dot_vec<TA, TX, TC, S>(q1, q2, lane, cj2, va2, x2, xcols2, bad)
                 : row_dot<TA, TX, TC, S>(q1, q2, lane, cj2, va2, x2, xcols2, bad);
      acc2 = group_reduce(acc2, S, wlane);
    }
    if (lane == 0) {
      TC v = mul_rn(alpha, mul_rn(acc, xs));
      if (rp2) mac(v, alpha2, acc2);
      if (b) mac(v, beta, (TC)b[row]);
      y[row] = (TY)v;
    }
  }
  if (bad && err) atomicOr(err, kErrIndex);
}

template <typename TA, typename TX, typename TY, typename TC, int S, bool VEC>
__global__ void __launch_bounds__(256) spmv_kernel(
    int nrows, const int* __restrict__ rp1, const int* __restrict__ cj1, const TA* __restrict__ va1,
    const TX* __restrict__ x1, int xcols1, TC alpha, const int* __restrict__ rp2, const int* __restrict__ cj2,
    const TA* __restrict__ va2, const TX* __restrict__ x2, int xcols2, TC alpha2, const TY* b, TC beta, TY* y,
    const double* __restrict__ xscale, int* err, Skip skip) {
  if (skip.on()) return;
  spmv_rows<TA, TX, TY, TC, S, VEC>(nrows, rp1, cj1, va1, x1, xcols1, alpha, rp2, cj2, va2, x2, xcols2, alpha2, b, beta,
                                    y, xscale, err);
}

// ------------------------------------------------- the variant of a matrix
// whose arrays are on the device (pgx_csr_spmv_device).  spmv_plan_kernel
// gathers what the rule of the host's spmv_plan asks of the row lengths, in
// one pass over the row pointer: how many rows fit each batch size, the
// longest row, and the nonzeros in rows longer than four batches; the last
// block to finish applies the rule.  All sums are of integers, so the plan
// is the host's.  spmv_planned_kernel then takes S from device memory, and
// leaves a matrix planned for the merge path alone.
// Bound by launches at small sizes and the row pointer's bytes at large ones.
// On a B200, a whole pgx_csr_spmv_device call (plan, product, wait): 33 us at
// 65,536 rows of a 5-point stencil and 83 us at 2,097,152 of a 7-point one;
// with the row pointer copied to the host and planned there 196 us and 6.3 ms.
constexpr int kPlanSizes = 5;  // S = 2, 4, 8, 16, 32
struct SpmvPlanDev {
  unsigned long long heavy[kPlanSizes];  // nonzeros of rows longer than 4 batches of S = 2 << k lanes
  unsigned fits[kPlanSizes];             // rows of at most one batch
  unsigned longest, blocks;              // the longest row; blocks that are done
  int S, merge;
};
__global__ void __launch_bounds__(512) spmv_plan_kernel(int nrows, long long nnz, const int* __restrict__ rp,
                                                        SpmvPlanDev* __restrict__ plan) {
  __shared__ unsigned long long s_heavy[kPlanSizes];
  __shared__ unsigned s_fits[kPlanSizes], s_longest;
  if (threadIdx.x < kPlanSizes) {
    s_heavy[threadIdx.x] = 0;
    s_fits[threadIdx.x] = 0;
  }
  if (threadIdx.x == 0) s_longest = 0;
  __syncthreads();
  unsigned long long heavy[kPlanSizes] = {};
  unsigned fits[kPlanSizes] = {}, longest = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
    const int len = __ldg(&rp[r + 1]) - __ldg(&rp[r]);
    longest = max(longest, (unsigned)max(len, 0));
#pragma unroll
    for (int k = 0; k < kPlanSizes; k++) {
      const int batch = (2 << k) * kSpmvUnroll;
      fits[k] += len <= batch;
      if (len > 4 * batch) heavy[k] += (unsigned)len;
    }
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
#pragma unroll
  for (int k = 0; k < kPlanSizes; k++) {
    fits[k] = __reduce_add_sync(0xffffffffu, fits[k]);
    heavy[k] = warp_reduce(heavy[k]);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_longest, longest);
#pragma unroll
    for (int k = 0; k < kPlanSizes; k++) {
      atomicAdd(&s_fits[k], fits[k]);
      if (heavy[k]) atomicAdd(&s_heavy[k], heavy[k]);
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  atomicMax(&plan->longest, s_longest);
  for (int k = 0; k < kPlanSizes; k++) {
    atomicAdd(&plan->fits[k], s_fits[k]);
    if (s_heavy[k]) atomicAdd(&plan->heavy[k], s_heavy[k]);
  }
  __threadfence();
  if (atomicAdd(&plan->blocks, 1u) != gridDim.x - 1) return;
  __threadfence();
  // the rows below and at the 90th percentile; k: the smallest size whose batch holds them
  const unsigned want = (unsigned)min((long long)nrows, max(1ll, (long long)ceil(0.9 * nrows)));
  int k = 0;
  while (k < kPlanSizes - 1 && atomicAdd(&plan->fits[k], 0u) < want) k++;
  const unsigned batch = (2u << k) * kSpmvUnroll;
  plan->S = 2 << k;
  plan->merge = atomicMax(&plan->longest, 0u) > 16 * batch && (long long)atomicAdd(&plan->heavy[k], 0ull) * 10 > nnz;
}

template <bool VEC>
__global__ void __launch_bounds__(256) spmv_planned_kernel(const SpmvPlanDev* __restrict__ plan, int forced, int nrows,
                                                           const int* __restrict__ rp, const int* __restrict__ cj,
                                                           const double* __restrict__ va, const double* __restrict__ x,
                                                           int xcols, double alpha, const double* b, double beta,
                                                           double* y) {
  if (plan->merge && !forced) return;
#define PGX_ROWS(SS)                                                                                                   \
  spmv_rows<double, double, double, double, SS, VEC>(nrows, rp, cj, va, x, xcols, alpha, nullptr, nullptr, nullptr,    \
                                                     nullptr, 0, 0.0, b, beta, y, nullptr, nullptr)
  switch (plan->S) {
    case 2: PGX_ROWS(2); break;
    case 4: PGX_ROWS(4); break;
    case 8: PGX_ROWS(8); break;
    case 16: PGX_ROWS(16); break;
    default: PGX_ROWS(32); break;
  }
#undef PGX_ROWS
}

// ---------------------------------------------------- merge-path CSR SpMV
// For matrices whose row lengths are skewed (a few very long rows among
// short ones), the row-per-group kernel leaves most lanes idle on the short
// rows and serialises the long ones.  The merge-path SpMV (Merrill and
// Garland, "Merge-based parallel sparse matrix-vector multiplication", SC16)
// gives every thread the same number of merge items, where the items are
// the n row ends and the nnz nonzeros taken in merge order (a nonzero k of
// row r comes before the end of row r).  A thread finds its start on the
// merge path by a binary search on its diagonal, then consumes its items:
// rows that end in its range are written at once; the partial sum of the
// row it stops inside is its carry, added by merge_spmv_fixup_kernel.
// y = alpha * A x + beta * b (b may be absent or alias y).
constexpr int kMergeItems = 16;  // merge items per thread

__device__ __forceinline__ void merge_path_search(int diag, const int* __restrict__ rp, int nrows, int nnz, int* row,
                                                  int* k) {
  // the number of row ends among the first `diag` merge items: the largest i
  // with rp[i] (the end of row i-1) <= diag - i
  int lo = max(diag - nnz, 0), hi = min(diag, nrows);
  while (lo < hi) {
    const int pivot = (lo + hi) >> 1;
    if (__ldg(&rp[pivot + 1]) <= diag - pivot - 1)
      lo = pivot + 1;
    else
      hi = pivot;
  }
  *row = min(lo, nrows);
  *k = diag - *row;
}

template <typename TA, typename TX, typename TY, typename TC>
__global__ void __launch_bounds__(256) merge_spmv_kernel(
    int nrows, int nnz, const int* __restrict__ rp, const int* __restrict__ cj, const TA* __restrict__ va,
    const TX* __restrict__ x, TC alpha, const TY* b, TC beta, TY* y, int* __restrict__ carry_row,
    TC* __restrict__ carry_val, Skip skip) {
  if (skip.on()) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)nrows + nnz;
  const long long d0 = (long long)t * kMergeItems;
  if (d0 >= total) return;
  const int d1 = (int)min(d0 + kMergeItems, total);
  int r, k, r1, k1;
  merge_path_search((int)d0, rp, nrows, nnz, &r, &k);
  merge_path_search(d1, rp, nrows, nnz, &r1, &k1);
  TC acc = 0;
  int rend = r < nrows ? __ldg(&rp[r + 1]) : nnz;
  while (r < r1 || k < k1) {
    if (r < nrows && k < rend && k < k1) {
      acc += (TC)ldg(&va[k]) * (TC)x[__ldg(&cj[k])];
      k++;
    } else {
      // row r ends inside this range: its sum here plus the carries of the
      // threads before it that stopped inside the row
      TC v = alpha * acc;
      if (b) v += beta * (TC)b[r];
      y[r] = (TY)v;
      acc = 0;
      r++;
      rend = r < nrows ? __ldg(&rp[r + 1]) : nnz;
    }
  }
  carry_row[t] = r < nrows ? r : -1;
  carry_val[t] = acc;
}

// y[row] += alpha * (carries of that row, in thread order): one thread per
// run of equal rows, so the sum is deterministic
template <typename TY, typename TC>
__global__ void merge_spmv_fixup_kernel(int nthreads, const int* __restrict__ carry_row,
                                        const TC* __restrict__ carry_val, TC alpha, TY* y, Skip skip) {
  if (skip.on()) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nthreads; t += gridDim.x * blockDim.x) {
    const int row = carry_row[t];
    if (row < 0 || (t > 0 && carry_row[t - 1] == row)) continue;
    TC s = 0;
    for (int u = t; u < nthreads && carry_row[u] == row; u++) s += carry_val[u];
    y[row] = (TY)((TC)y[row] + alpha * s);
  }
}

// ----------------------------------------------- sync-free triangular solve
// One pass of the ILU solve of IluClass::SolveHost (ParGeMSLR
// SRC/preconditioners/ilu.cpp:3677-3790) over a whole level (all subdomains
// of the level concatenated block-diagonally):
//   lower:  y_r = rhs_r - sum_j L_rj y_j               (unit diagonal)
//   upper:  x_r = (y_r - sum_j U_rj x_j) * dinv_r     (dinv = inverse diagonal)
// Rows are stored in level-set order (IluClass::BuildLevels rule,
// ilu.cpp:832-1062), each level padded to whole groups of G = 32/S rows, so a
// group never holds two rows of which one depends on the other.
//
// Readiness is carried by the value itself: entries not yet computed hold a
// signalling-NaN sentinel that arithmetic never produces.  A row publishes
// its result with one relaxed store; a consumer polls the entry with relaxed
// loads until the sentinel is gone - one L2 round trip per dependency and no
// fences.  The lower pass writes y and sets x to the sentinel; the upper pass
// consumes y, writes x and puts the sentinel back into y, so each pass leaves
// the buffers ready for the next one.
//
// The grid is persistent and sized to the level width (few pollers, little
// L2 pressure).  Warps claim groups from a 64-bit ticket counter in schedule
// order; a row only waits on rows of earlier levels, whose groups were
// claimed earlier by warps that are running, so the waits always end.  The
// last warp to leave resets the counter (ticket[0]) and the exit count
// (ticket[1]) for the next launch, whatever the grid size.  Waits are
// bounded by spin_limit polls (kSpinLimit unless the handle sets another);
// on expiry the kernel records kErrTimeout and finishes.
template <typename T>
struct Sentinel;
template <>
struct Sentinel<double> {
  static __device__ __forceinline__ double value() { return __longlong_as_double(0xFFF4DEADBEEF0001LL); }
  static __device__ __forceinline__ bool is(double v) { return __double_as_longlong(v) == 0xFFF4DEADBEEF0001LL; }
  static __device__ __forceinline__ double load(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
  }
};
template <>
struct Sentinel<float> {
  static __device__ __forceinline__ float value() { return __int_as_float((int)0xFFA0BEEFu); }
  static __device__ __forceinline__ bool is(float v) { return __float_as_int(v) == (int)0xFFA0BEEFu; }
  static __device__ __forceinline__ float load(const float* p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(float* p, float v) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
  }
};

// Complex values: the sentinel sits in the real part.  A complex64 value is
// published with one 8-byte store.  A complex128 value spans two 8-byte
// words: the imaginary part is stored first and the real part after it with
// release semantics, and a reader loads the real part with acquire semantics
// before the imaginary part, so a reader that sees a final real part also
// sees the imaginary part that belongs to it.
template <>
struct Sentinel<cf32> {
  static __device__ __forceinline__ cf32 value() { return cf32(Sentinel<float>::value(), 0.f); }
  static __device__ __forceinline__ bool is(const cf32& v) { return Sentinel<float>::is(v.x); }
  static __device__ __forceinline__ cf32 load(const cf32* p) {
    unsigned long long u;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
    return cf32(__int_as_float((int)(u & 0xffffffffull)), __int_as_float((int)(u >> 32)));
  }
  static __device__ __forceinline__ void store(cf32* p, const cf32& v) {
    const unsigned long long u =
        (unsigned long long)(unsigned)__float_as_int(v.x) | ((unsigned long long)(unsigned)__float_as_int(v.y) << 32);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
  }
};
template <>
struct Sentinel<cf64> {
  static __device__ __forceinline__ cf64 value() { return cf64(Sentinel<double>::value(), 0.0); }
  static __device__ __forceinline__ bool is(const cf64& v) { return Sentinel<double>::is(v.x); }
  static __device__ __forceinline__ cf64 load(const cf64* p) {
    double re, im;
    asm volatile("ld.acquire.gpu.global.f64 %0, [%1];" : "=d"(re) : "l"(&p->x) : "memory");
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(im) : "l"(&p->y) : "memory");
    return cf64(re, im);
  }
  static __device__ __forceinline__ void store(cf64* p, const cf64& v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(&p->y), "d"(v.y) : "memory");
    asm volatile("st.release.gpu.global.f64 [%0], %1;" ::"l"(&p->x), "d"(v.x) : "memory");
  }
};
// the segmented solve's operand prefetch: a complex128 operand goes through
// the acquire/release pair above
template <typename T>
__device__ __forceinline__ T ldcg_dep(const T* p) { return ldcg(p); }
template <>
__device__ __forceinline__ cf64 ldcg_dep<cf64>(const cf64* p) { return Sentinel<cf64>::load(p); }

template <typename T>
__global__ void sentinel_fill_kernel(int n, T* p) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = Sentinel<T>::value();
}

template <typename T, int S, bool UPPER>
__global__ void __launch_bounds__(256) trsv_kernel(
    int n, int ngroups, const int* __restrict__ ord, const int* __restrict__ rp, const int* __restrict__ cj,
    const T* __restrict__ va, const T* __restrict__ dinv, const T* __restrict__ rhs,
    const double* __restrict__ rhs_scale, T* y, T* x, unsigned long long* ticket, int* err, int spin_limit,
    Skip skip) {
  constexpr int G = kWarp / S;  // rows per warp
  if (skip.on()) return;
  const int lane = threadIdx.x & (kWarp - 1);
  const int sl = lane & (S - 1);
  const double rs = rhs_scale ? *rhs_scale : 1.0;
  T* dep = UPPER ? x : y;  // the vector this pass polls
  while (true) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(&ticket[0], 1ULL);
    t = __shfl_sync(0xffffffffu, t, 0);
    const unsigned long long g = t;
    if (g >= (unsigned long long)ngroups) break;
    const int pos = (int)g * G + lane / S;
    const int r = ord[pos];  // -1 marks padding; uniform over the S-lane group
    if (r >= 0) {
      T acc = 0;
      const int k1 = rp[pos], k2 = rp[pos + 1];
      for (int k = k1 + sl; k < k2; k += S) {
        const int j = cj[k];
        if ((unsigned)j >= (unsigned)n) {
          atomicOr(err, kErrIndex);
          continue;
        }
        T v = Sentinel<T>::load(&dep[j]);
        if (Sentinel<T>::is(v)) {
          int spins = 0;
          do {
            if (++spins > spin_limit || (*(volatile int*)err & kErrTimeout)) {
              atomicOr(err, kErrTimeout);
              v = 0;
              break;
            }
            __nanosleep(20);
            v = Sentinel<T>::load(&dep[j]);
          } while (Sentinel<T>::is(v));
        }
        acc += va[k] * v;
      }
      acc = group_reduce(acc, S, lane);
      if (sl == 0) {
        if (UPPER) {
          const T yr = y[r];
          y[r] = Sentinel<T>::value();
          Sentinel<T>::store(&x[r], (yr - acc) * dinv[r]);
        } else {
          T b = rhs[r];
          if (rhs_scale) b = to<T>(to<typename Sc<T>::acc>(b) * rs);
          x[r] = Sentinel<T>::value();
          Sentinel<T>::store(&y[r], b - acc);
        }
      }
    }
  }
  // the last warp to leave rewinds the counters for the next launch
  if (lane == 0) {
    __threadfence();
    const unsigned long long nw = (unsigned long long)gridDim.x * (blockDim.x / kWarp);
    if (atomicAdd(&ticket[1], 1ULL) == nw - 1) {
      ticket[0] = 0ULL;
      ticket[1] = 0ULL;
      __threadfence();
    }
  }
}

// ------------------------------------- segmented (CTA-local) triangular solve
// Same arithmetic as trsv_kernel, different schedule.  Each subdomain's rows,
// in level-set order, are cut into segments of at most kSegRows rows and
// kSegNnz nonzeros.  A CTA claims a segment (ticket order: by first level,
// then subdomain, so a segment only depends on segments claimed earlier),
// stages the segment's row list, row pointers, column indices and values into
// shared memory with cp.async, then sweeps the segment's levels with one
// __syncthreads per level.  Dependencies inside the segment are read from the
// shared-memory copy of the results (column index encoded as -(slot+1));
// dependencies on earlier segments are polled in global memory through the
// sentinel protocol of trsv_kernel.  Every result is also published to global
// memory for later segments and the next kernel.
constexpr int kSegThreads = 1024;
constexpr int kSegRows = 1024;
constexpr int kSegNnzF64 = 8192;    // staged cj + va + gathered operands: 160 KB (FP64)
constexpr int kSegNnzF32 = 12288;   // 144 KB (FP32)
constexpr int kSegNnzC128 = 4096;   // 192 KB (complex128)

template <typename T>
struct SegCfg {
  static constexpr int nnz = sizeof(T) == 16 ? kSegNnzC128 : sizeof(T) == 8 ? kSegNnzF64 : kSegNnzF32;
  // smem layout: xs[kSegRows] T | sb[kSegRows] T | sd[kSegRows] T | va[nnz] T | ext[nnz] T |
  // cj[nnz] int | ord[kSegRows] int | rp[kSegRows+4] int | lvb[kSegRows+4] int; the host keeps
  // segments within kSegRows-4 rows and nnz-4 nonzeros
  static constexpr size_t bytes =
      sizeof(T) * (size_t)(3 * kSegRows + 2 * nnz) + sizeof(int) * (size_t)(nnz + kSegRows + 2 * (kSegRows + 4));
  static_assert(bytes <= 227 * 1024, "segmented solve exceeds the shared memory of a CTA");
};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// copy `bytes` (multiple of 16, both addresses 16-byte aligned) with cp.async
__device__ __forceinline__ void stage16(void* dst, const void* src, int bytes) {
  for (int o = threadIdx.x * 16; o < bytes; o += blockDim.x * 16) cp_async16((char*)dst + o, (const char*)src + o);
}

template <typename T, int S, bool UPPER>
__global__ void __launch_bounds__(kSegThreads) trsv_seg_kernel(
    int n, int nseg, const int* __restrict__ seg_row0,  // nseg+1: first slot in ord
    const int* __restrict__ seg_rp0,                     // nseg+1: first slot in rp (segment-relative values)
    const int* __restrict__ seg_nnz0,                    // nseg+1: first slot in cj / va
    const int* __restrict__ seg_lv0,                     // nseg+1: first slot in lvb
    const int* __restrict__ seg_nlvb,                    // nseg: number of level boundaries
    const int* __restrict__ ord, const int* __restrict__ rp,  // rp: segment-relative row pointers
    const int* __restrict__ cj, const T* __restrict__ va, const int* __restrict__ lvb,  // lvb: segment-relative
    const T* __restrict__ dinv, const T* __restrict__ rhs, const double* __restrict__ rhs_scale, T* y, T* x,
    unsigned long long* ticket, int* err, int spin_limit, Skip skip) {
  if (skip.on()) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NNZ = SegCfg<T>::nnz;
  T* xs = (T*)smem_raw;
  T* sb = xs + kSegRows;  // rhs (lower) or y (upper) of the segment's rows
  T* sd = sb + kSegRows;  // dinv of the segment's rows (upper)
  T* sva = sd + kSegRows;
  T* sext = sva + NNZ;  // operands from earlier segments, gathered at staging
  int* scj = (int*)(sext + NNZ);
  int* sord = scj + NNZ;
  int* srp = sord + kSegRows;
  int* slvb = srp + kSegRows + 4;
  __shared__ unsigned long long s_t;
  const int tid = threadIdx.x, lane = tid & 31;
  const int sl = lane & (S - 1);
  const int group = tid / S, ngroups = kSegThreads / S;
  const double rs = rhs_scale ? *rhs_scale : 1.0;
  T* dep = UPPER ? x : y;
  while (true) {
    if (tid == 0) s_t = atomicAdd(&ticket[0], 1ULL);
    __syncthreads();
    const unsigned long long g = s_t;
    if (g >= (unsigned long long)nseg) break;
    const int sgi = (int)g;
    // every per-segment block starts 16-byte aligned and has a 16-byte
    // multiple length (padded on the host)
    const int r0 = seg_row0[sgi], r1 = seg_row0[sgi + 1];
    const int p0 = seg_rp0[sgi], p1 = seg_rp0[sgi + 1];
    const int z0 = seg_nnz0[sgi], z1 = seg_nnz0[sgi + 1];
    const int v0 = seg_lv0[sgi];
    const int nlvb = seg_nlvb[sgi];
    stage16(sva, va + z0, (z1 - z0) * (int)sizeof(T));
    stage16(scj, cj + z0, (z1 - z0) * 4);
    stage16(sord, ord + r0, (r1 - r0) * 4);
    stage16(srp, rp + p0, (p1 - p0) * 4);
    stage16(slvb, lvb + v0, (seg_lv0[sgi + 1] - v0) * 4);
    // gather the per-row operands while the copies are in flight (plain
    // loads: independent, so they overlap)
    for (int i = tid; i < r1 - r0; i += blockDim.x) {
      const int r = __ldg(&ord[r0 + i]);
      if (r < 0) continue;
      if (UPPER) {
        sb[i] = ldcg_dep(&y[r]);
        sd[i] = ldg(&dinv[r]);
      } else {
        T bb = ldg(&rhs[r]);
        if (rhs_scale) bb = to<T>(to<typename Sc<T>::acc>(bb) * rs);
        sb[i] = bb;
      }
    }
    cp_async_wait_all();
    __syncthreads();
    // gather every operand owned by an earlier segment in one parallel sweep
    // through L2; most are final already, the rest still read the sentinel
    // and are polled in the sweep below.  Entries are written with single
    // 4/8-byte stores, so a load sees either the sentinel or the final value.
    for (int k = tid; k < z1 - z0; k += blockDim.x) {
      const int c = scj[k];
      if (c >= 0 && c < n) sext[k] = ldcg_dep(&dep[c]);
    }
    // this segment's rows: hand the buffers to the next pass
    for (int i = tid; i < r1 - r0; i += blockDim.x) {
      const int r = sord[i];
      if (r < 0) continue;
      if (UPPER)
        y[r] = Sentinel<T>::value();
      else
        x[r] = Sentinel<T>::value();
    }
    __syncthreads();
    for (int lv = 0; lv + 1 < nlvb; lv++) {
      const int a = slvb[lv], b = slvb[lv + 1];
      for (int i = a + group; i < b; i += ngroups) {
        const int r = sord[i];
        if (r < 0) continue;  // padding slot
        T acc = 0;
        const int k1 = srp[i], k2 = srp[i + 1];
        for (int k = k1 + sl; k < k2; k += S) {
          const int c = scj[k];
          T v;
          if (c < 0) {
            v = xs[-c - 1];
          } else {
            if ((unsigned)c >= (unsigned)n) {
              atomicOr(err, kErrIndex);
              continue;
            }
            v = sext[k];
            if (Sentinel<T>::is(v)) {
              v = Sentinel<T>::load(&dep[c]);
            }
            if (Sentinel<T>::is(v)) {
              int spins = 0;
              do {
                if (++spins > spin_limit || (*(volatile int*)err & kErrTimeout)) {
                  atomicOr(err, kErrTimeout);
                  v = 0;
                  break;
                }
                __nanosleep(20);
                v = Sentinel<T>::load(&dep[c]);
              } while (Sentinel<T>::is(v));
            }
          }
          acc += sva[k] * v;
        }
        acc = group_reduce(acc, S, lane);
        if (sl == 0) {
          T out;
          if (UPPER) {
            out = (sb[i] - acc) * sd[i];
            Sentinel<T>::store(&x[r], out);
          } else {
            out = sb[i] - acc;
            Sentinel<T>::store(&y[r], out);
          }
          xs[i] = out;
        }
      }
      __syncthreads();
    }
    __syncthreads();  // s_t and the staged arrays are reused by the next claim
  }
  // the last CTA to leave rewinds the counters for the next launch
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&ticket[1], 1ULL) == (unsigned long long)gridDim.x - 1) {
      ticket[0] = 0ULL;
      ticket[1] = 0ULL;
      __threadfence();
    }
  }
}

// ------------------------------------------------ building blocks of the
// one-CTA-per-subdomain triangular solve (pgx_flow.cuh)
constexpr long long kMbarWaitCycles = 1ll << 31;  // bound of a wait on a staging barrier: about 1 s

template <typename T, int R>
struct __align__(sizeof(T) * R <= 16 ? sizeof(T) * R : 16) VecR {
  T v[R];
};
template <typename T, int R>
struct PtrR {
  T* p[R];
};

// mbarrier and bulk-copy (TMA, non-tensor) helpers.  The copies read this
// GPU's own global memory only.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// orders this thread's ordinary accesses to shared memory before bulk copies into it
__device__ __forceinline__ void proxy_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false (and kErrStage recorded) if the phase did not
// complete within kMbarWaitCycles SM clocks
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (clock64() - t0 < kMbarWaitCycles)
    if (mbar_try_wait(bar, parity)) return true;
  atomicOr(err, kErrStage);
  return false;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// ------------------------------------------------- tall-skinny kernels
// One kernel family covers every operation on a block of dense columns:
// the Gram-Schmidt passes of the Arnoldi step (PargemslrMgs / PargemslrCgs2,
// ParGeMSLR SRC/matrices/matrixops.cpp:10588-10806), the Woodbury low-rank
// correction W^T x then WH y (GemslrClass::SolveApplyLowRankLevel,
// gemslr.cpp:3681-3722) and the solution update x += Z y (fgmres.hpp:483-490).
//
//   TS_DOT          sums[c] = V(:,c) . w,            w = in * in_scale
//   TS_UPDATE       out = in * in_scale + sign * M coef'
//   TS_UPDATE_DOT   out = w' = (update above); sums[c] = V(:,c) . w'
//   TS_UPDATE_NORM  out = w' = (update above); sums[0] = w' . w'
//   TS_NORM_COPY    sums[0] = w . w; out = w (if out)
// with coef'[c] = coef[c] * msc[c] and msc the lazy column scales of M.
// Columns are column-major with leading dimension ld.  Each block walks
// 512-row tiles; per tile, thread t updates row t, then warp w reduces the
// columns c = w mod 16 over the tile (the tile is re-read from L1/L2, so DRAM
// sees each column once).  Block partials are combined by the last block to
// finish, in a fixed order, so results do not depend on block scheduling;
// that block then runs the epilogue (storing coefficients, or the Givens
// update of the Hessenberg column).
enum TsMode { TS_DOT = 0, TS_UPDATE = 1, TS_UPDATE_DOT = 2, TS_UPDATE_NORM = 3, TS_NORM_COPY = 4 };
enum EpiKind {
  EPI_NONE = 0,
  EPI_STORE = 1,       // dst[c] = sums[c] * vsc[c]
  EPI_CGS_FIRST = 2,   // hcol = coefA = sums * vsc
  EPI_CGS_SECOND = 3,  // coefB = sums * vsc; hcol += coefB
  EPI_GIVENS = 4,      // finish column j: norm, rotations, convergence, back-solve
  EPI_NORMB = 5,       // st->normb = sqrt(sums[0])
  EPI_INIT = 6,        // outer start of solve: normr, tolr, rs[0], sc[0]
  EPI_INIT_INNER = 7,  // inner solve from x0 = 0: normb = normr = ||rhs||
};

// Reductions and coefficients are carried in TsAcc<TW>: double for a real
// solve, cf64 for a complex one (dots conjugate the basis column,
// V(:,c)^H w, as the reference's complex VectorDot does).
template <typename TW>
using TsAcc = typename Sc<TW>::acc;

template <typename TV, typename TM, typename TW>
struct TsArgs {
  using A = TsAcc<TW>;
  int n;
  int ncols;
  const int* ncols_dev;  // if set, the column count is read here (<= KMAX)
  const TV* V;
  long long ldv;
  const double* vsc;
  const TM* M;
  long long ldm;
  const double* msc;
  const A* coef;
  double sign;
  const TW* in;          // null: zero input
  const double* in_scale;
  TW* out;
  A* partial;            // [KMAX+1][gridDim.x]
  unsigned int* counter; // zero between launches
  int epi;
  FgmresDevT<A>* st;
  A* dst;
  int j;
  Skip skip;
};

template <typename S>
__device__ inline void fgmres_givens(FgmresDevT<S>* st, int j, double t) {
  // H(:, j) from the Gram-Schmidt coefficients and ||w||
  // (PargemslrMgs sets H(0..k, k) and H(k+1, k), matrixops.cpp:10728-10806)
  const int ldh = KMAX + 1;
  S* H = st->H + (size_t)j * ldh;
  for (int c = 0; c <= j; c++) H[c] = st->hcol[c];
  H[j + 1] = S(t);
  st->sc[j + 1] = 1.0 / t;
  st->iter += 1;
  st->i = j + 1;
  // apply the previous rotations, then form the new one (fgmres.hpp:430-458;
  // for complex values the rotation is conj(c), s as in the reference)
  for (int k = 1; k <= j; k++) {
    S hii = H[k - 1];
    H[k - 1] = conj(st->c[k - 1]) * hii + st->s[k - 1] * H[k];
    H[k] = -st->s[k - 1] * hii + st->c[k - 1] * H[k];
  }
  S hii = H[j], hii1 = H[j + 1];
  double gam = sqrt(cabs(hii) * cabs(hii) + cabs(hii1) * cabs(hii1));
  if (fabs(gam) < st->eps) {
    // breakdown: the reference jumps past the solution update (fgmres.hpp:440-443)
    // and records no residual for this iteration
    st->hist[j] = 0.0;
    st->breakdown = 1;
    st->i = 0;
    st->cycle_done = 1;
    st->done = 1;
    return;
  }
  st->c[j] = hii / gam;
  st->s[j] = hii1 / gam;
  st->rs[j + 1] = -st->s[j] * st->rs[j];
  st->rs[j] = conj(st->c[j]) * st->rs[j];
  H[j] = conj(st->c[j]) * hii + st->s[j] * hii1;
  st->normr = cabs(st->rs[j + 1]);
  st->hist[j] = st->normr;  // _rel_res_vector[_iter] = normr / normb (fgmres.hpp:450-452)
  const bool conv = st->normr <= st->tolr;
  if (conv) st->converged = 1;
  if (conv || st->i >= st->kdim || st->iter >= st->maxits) {
    st->cycle_done = 1;
    if (conv || st->iter >= st->maxits) st->done = 1;
    // back substitution H y = rs, in place in rs (fgmres.hpp:471-480)
    const int i = st->i;
    S* rs = st->rs;
    rs[i - 1] = rs[i - 1] / st->H[(size_t)(i - 1) * ldh + (i - 1)];
    for (int k = i - 2; k >= 0; k--) {
      for (int jj = k + 1; jj < i; jj++) rs[k] -= st->H[(size_t)jj * ldh + k] * rs[jj];
      rs[k] = rs[k] / st->H[(size_t)k * ldh + k];
    }
  }
}

// The same by a whole block (the last one of a reduction), for the kernel
// whose end is on the critical path of every Krylov step: one thread read the
// state word by word from global memory (ncu, inner steps of a 64^3 solve:
// 12.4 us a launch then, 10.7 us now; of outer steps 17.0 and 14.2 us).
// The column, the rotations and the scalars are read by all threads at once,
// thread 0 rotates in shared memory, and one warp substitutes back with the
// next column of H on its way.  `sh` holds 3 * (KMAX + 1) values.
template <typename S>
__device__ inline void fgmres_givens_block(FgmresDevT<S>* st, int j, double t, S* sh, int* s_back) {
  const int ldh = KMAX + 1, tid = threadIdx.x;
  S *h = sh, *rc = sh + ldh, *rs_ = sh + 2 * ldh;
  for (int c = tid; c <= j; c += blockDim.x) {
    h[c] = st->hcol[c];
    if (c < j) {
      rc[c] = st->c[c];
      rs_[c] = st->s[c];
    }
  }
  if (tid == 0) *s_back = 0;
  __syncthreads();
  if (tid == 0) {
    const S rsj = st->rs[j];
    const double eps = st->eps, tolr = st->tolr;
    const int kdim = st->kdim, maxits = st->maxits, iter = st->iter + 1;
    h[j + 1] = S(t);
    st->sc[j + 1] = 1.0 / t;
    st->iter = iter;
    st->i = j + 1;
    for (int k = 1; k <= j; k++) {
      const S hii = h[k - 1], hk = h[k];
      h[k - 1] = conj(rc[k - 1]) * hii + rs_[k - 1] * hk;
      h[k] = -rs_[k - 1] * hii + rc[k - 1] * hk;
    }
    const S hii = h[j], hii1 = h[j + 1];
    const double gam = sqrt(cabs(hii) * cabs(hii) + cabs(hii1) * cabs(hii1));
    if (fabs(gam) < eps) {
      st->hist[j] = 0.0;
      st->breakdown = 1;
      st->i = 0;
      st->cycle_done = 1;
      st->done = 1;
    } else {
      const S c = hii / gam, s = hii1 / gam;
      st->c[j] = c;
      st->s[j] = s;
      const S next = -s * rsj;
      st->rs[j + 1] = next;
      st->rs[j] = conj(c) * rsj;
      h[j] = conj(c) * hii + s * hii1;
      const double normr = cabs(next);
      st->normr = normr;
      st->hist[j] = normr;
      const bool conv = normr <= tolr;
      if (conv) st->converged = 1;
      if (conv || j + 1 >= kdim || iter >= maxits) {
        st->cycle_done = 1;
        if (conv || iter >= maxits) st->done = 1;
        *s_back = j + 1;
      }
    }
  }
  __syncthreads();
  for (int c = tid; c <= j + 1; c += blockDim.x) st->H[(size_t)j * ldh + c] = h[c];
  const int n = *s_back;
  if (n == 0) return;
  __syncthreads();  // rs and the last column of H are written
  if (tid < 32) {
    constexpr int Q = (KMAX + 31) / 32;
    S r[Q], col[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = tid + 32 * q;
      r[q] = i < n ? st->rs[i] : S(0.0);
      col[q] = i < n ? st->H[(size_t)(n - 1) * ldh + i] : S(0.0);
    }
    for (int k = n - 1; k >= 0; k--) {
      S nxt[Q];
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int i = tid + 32 * q;
        nxt[q] = k > 0 && i < k ? st->H[(size_t)(k - 1) * ldh + i] : S(0.0);
      }
      S rk = S(0.0), d = S(0.0);
#pragma unroll
      for (int q = 0; q < Q; q++)
        if (k / 32 == q) {
          rk = r[q];
          d = col[q];
        }
      const S y = bcast(rk, k & 31) / bcast(d, k & 31);
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int i = tid + 32 * q;
        if (i < k) r[q] -= col[q] * y;
        if (i == k) r[q] = y;
        col[q] = nxt[q];
      }
    }
#pragma unroll
    for (int q = 0; q < Q; q++)
      if (tid + 32 * q < n) st->rs[tid + 32 * q] = r[q];
  }
}

template <typename TV, typename TM, typename TW>
__device__ inline void ts_epilogue(const TsArgs<TV, TM, TW>& a, const TsAcc<TW>* sums) {
  using A = TsAcc<TW>;
  FgmresDevT<A>* st = a.st;
  switch (a.epi) {
    case EPI_NORMB:
      st->normb = sqrt(re(sums[0]));
      if (st->normb < st->eps) {
        st->done = 1;
        st->cycle_done = 1;
        st->normr = 0.0;
        st->i = 0;
      }
      break;
    case EPI_INIT: {
      st->i = 0;
      st->iter = 0;
      st->converged = 0;
      st->breakdown = 0;
      if (st->done) break;  // zero right-hand side
      const double normr = sqrt(re(sums[0]));
      st->normr = normr;
      st->normr0 = normr;
      if (normr < st->eps) {
        st->done = 1;
        st->cycle_done = 1;
        st->converged = 1;
        break;
      }
      st->tolr = st->absolute ? st->tol : st->tol * st->normb;
      st->rs[0] = A(normr);
      st->sc[0] = 1.0 / normr;
      st->cycle_done = 0;
      break;
    }
    case EPI_INIT_INNER: {
      const double normb = sqrt(re(sums[0]));
      st->normb = normb;
      st->normr = normb;
      st->i = 0;
      st->iter = 0;
      st->converged = 0;
      st->breakdown = 0;
      st->done = 0;
      st->cycle_done = 0;
      if (normb < st->eps) {
        st->done = 1;
        st->cycle_done = 1;
        break;
      }
      st->tolr = st->absolute ? st->tol : st->tol * normb;
      st->rs[0] = A(normb);
      st->sc[0] = 1.0 / normb;
      break;
    }
    default:
      break;
  }
}

template <typename TV, typename TM, typename TW, int MODE>
__device__ __forceinline__ void ts_body(const TsArgs<TV, TM, TW>& a) {
  using A = TsAcc<TW>;
  if (a.skip.on()) return;
  __shared__ A scoef[KMAX + 1];
  __shared__ A sacc[KMAX + 1];
  __shared__ double swarp[kTsThreads / 32];
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = kTsThreads / 32;
  const int ncols = a.ncols_dev ? min(*(const volatile int*)a.ncols_dev, KMAX + 1) : a.ncols;
  const bool update = MODE == TS_UPDATE || MODE == TS_UPDATE_DOT || MODE == TS_UPDATE_NORM;
  const bool reduce = MODE != TS_UPDATE;
  const int nred = (MODE == TS_DOT || MODE == TS_UPDATE_DOT) ? ncols : 1;
  if (MODE == TS_UPDATE && ncols == 0 && a.in == a.out) return;  // nothing to add
  const double in_s = a.in_scale ? *a.in_scale : 1.0;
  for (int c = tid; c <= KMAX; c += kTsThreads) {
    scoef[c] = (update && c < ncols) ? a.sign * a.coef[c] * (a.msc ? a.msc[c] : 1.0) : A(0.0);
    sacc[c] = A(0.0);
  }
  if (tid < NW) swarp[tid] = 0.0;
  __syncthreads();
  const int ntiles = (a.n + kTsThreads - 1) / kTsThreads;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * kTsThreads;
    const int row = r0 + tid;
    A wv = A(0.0);
    if (row < a.n) {
      wv = a.in ? mul_rn(to<A>(a.in[row]), in_s) : A(0.0);
      if (update) {
        A acc = A(0.0);
        const TM* m = a.M + row;
        for (int c = 0; c < ncols; c++) mac(acc, to<A>(m[(long long)c * a.ldm]), scoef[c]);
        wv += acc;
      }
      if (MODE != TS_DOT && a.out) a.out[row] = to<TW>(wv);
    }
    if (MODE == TS_UPDATE_NORM || MODE == TS_NORM_COPY) {
      double sq = (row < a.n) ? abs2_rn(wv) : 0.0;
      if (MODE == TS_UPDATE_NORM) {
        // the norm of the stored (rounded) vector, as Norm2 of the reference
        TW stored = to<TW>(wv);
        sq = (row < a.n) ? abs2_rn(to<A>(stored)) : 0.0;
      }
      sq = warp_reduce(sq);
      if (lane == 0) swarp[warp] += sq;  // one writer per slot: deterministic
    }
    if (MODE == TS_DOT || MODE == TS_UPDATE_DOT) {
      __syncthreads();  // out[] of this tile written by the whole block
      const int nrows_tile = min(kTsThreads, a.n - r0);
      for (int c = warp; c < ncols; c += NW) {
        const TV* v = a.V + (long long)c * a.ldv + r0;
        A acc = A(0.0);
        for (int k = lane; k < nrows_tile; k += 32) {
          A w = (MODE == TS_DOT) ? (a.in ? mul_rn(to<A>(a.in[r0 + k]), in_s) : A(0.0)) : to<A>(a.out[r0 + k]);
          mac(acc, conj(to<A>(v[k])), w);
        }
        acc = warp_reduce(acc);
        if (lane == 0) sacc[c] += acc;
      }
      __syncthreads();
    }
  }
  if (!reduce) return;
  __syncthreads();
  if ((MODE == TS_UPDATE_NORM || MODE == TS_NORM_COPY) && tid == 0) {
    double t = 0.0;
    for (int w = 0; w < NW; w++) t += swarp[w];
    sacc[0] = A(t);
  }
  __syncthreads();
  // block partials -> global, column-major by block
  for (int c = tid; c < nred; c += kTsThreads) a.partial[(long long)c * gridDim.x + blockIdx.x] = sacc[c];
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    unsigned int prev = atomicAdd(a.counter, 1u);
    s_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int c = warp; c < nred; c += NW) {
    A acc = A(0.0);
    for (int b = lane; b < (int)gridDim.x; b += 32) acc += ldcg(&a.partial[(long long)c * gridDim.x + b]);
    acc = warp_reduce(acc);
    if (lane == 0) sacc[c] = acc;
  }
  __syncthreads();
  switch (a.epi) {
    case EPI_STORE:
      for (int c = tid; c < nred; c += kTsThreads) a.dst[c] = sacc[c] * (a.vsc ? a.vsc[c] : 1.0);
      break;
    case EPI_CGS_FIRST:
      for (int c = tid; c < nred; c += kTsThreads) {
        const A h = sacc[c] * (a.vsc ? a.vsc[c] : 1.0);
        a.st->hcol[c] = h;
        a.st->coefA[c] = h;
      }
      break;
    case EPI_CGS_SECOND:
      for (int c = tid; c < nred; c += kTsThreads) {
        const A h = sacc[c] * (a.vsc ? a.vsc[c] : 1.0);
        a.st->hcol[c] += h;
        a.st->coefB[c] = h;
      }
      break;
    case EPI_GIVENS:
      // only the kernel that ends a Krylov step carries this code
      if constexpr (MODE == TS_UPDATE_NORM) {
        __shared__ A sgiv[3 * (KMAX + 1)];
        __shared__ int s_back;
        fgmres_givens_block(a.st, a.j, sqrt(re(sacc[0])), sgiv, &s_back);
      }
      break;
    default:
      if (tid == 0) ts_epilogue(a, sacc);
      break;
  }
  if (tid == 0) *a.counter = 0u;
  __threadfence();
}

template <typename TV, typename TM, typename TW, int MODE>
__global__ void __launch_bounds__(kTsThreads) ts_kernel(const __grid_constant__ TsArgs<TV, TM, TW> a) {
  ts_body<TV, TM, TW, MODE>(a);
}

// The kernels of a multi-lane slot: one launch for all lanes, lane
// blockIdx.y with the arguments, grid and sums of its own single launch.
// Most of these kernels work on a few thousand rows and are bound by their
// launch: 16 right-hand sides of a complex 24^3 problem as one block took
// 198 ms with a launch per lane and take 58 ms (B200); 24 at 48^3, four to a
// slot, 131 and 86 ms.
template <typename TV, typename TM, typename TW>
struct TsLanes {
  TsArgs<TV, TM, TW> a[kMaxLanes];
};
template <typename TV, typename TM, typename TW, int MODE>
__global__ void __launch_bounds__(kTsThreads) ts_lanes_kernel(const __grid_constant__ TsLanes<TV, TM, TW> p) {
  ts_body<TV, TM, TW, MODE>(p.a[blockIdx.y]);
}

template <typename TX, typename TY>
struct SpmvLanes {
  const TX *x1[kMaxLanes], *x2[kMaxLanes];
  const TY* b[kMaxLanes];
  TY* y[kMaxLanes];
  int* err[kMaxLanes];
  Skip skip[kMaxLanes];
};
template <typename TA, typename TX, typename TY, typename TC, int S>
__global__ void __launch_bounds__(256) spmv_lanes_kernel(
    int nrows, const int* __restrict__ rp1, const int* __restrict__ cj1, const TA* __restrict__ va1, int xcols1,
    TC alpha, const int* __restrict__ rp2, const int* __restrict__ cj2, const TA* __restrict__ va2, int xcols2,
    TC alpha2, TC beta, const __grid_constant__ SpmvLanes<TX, TY> p) {
  const int r = blockIdx.y;
  if (p.skip[r].on()) return;
  spmv_rows<TA, TX, TY, TC, S, true>(nrows, rp1, cj1, va1, p.x1[r], xcols1, alpha, rp2, cj2, va2, p.x2[r], xcols2,
                                     alpha2, p.b[r], beta, p.y[r], nullptr, p.err[r]);
}

template <typename S>
struct StateLanes {
  FgmresDevT<S>* st[kMaxLanes];
};
template <typename S>
__device__ __forceinline__ void fgmres_cycle_reset(FgmresDevT<S>* st) {
  st->i = 0;
  if (st->done) return;
  st->cycle_done = 0;
  st->rs[0] = S(st->normr);
  st->sc[0] = 1.0 / st->normr;
}
template <typename S>
__global__ void fgmres_cycle_reset_kernel(FgmresDevT<S>* st, Skip skip) {
  if (!skip.on()) fgmres_cycle_reset(st);
}
template <typename S>
__global__ void fgmres_cycle_reset_lanes_kernel(const __grid_constant__ StateLanes<S> p) {
  fgmres_cycle_reset(p.st[threadIdx.x]);
}

// --------------------------------------------------- permutation + convert
// out[i] = (TO)(in[perm[i]] * scale)  (IntVectorClass::GatherPerm, int_vector.cpp:668)
// Each thread handles kPermUnroll entries a block apart: it loads their
// permutation indices, then the values they name, then stores, so the
// dependent loads of several entries are in flight together.
constexpr int kPermUnroll = 4;
template <typename TI, typename TO>
struct PermLanes {
  const TI* in[kMaxLanes];
  const double* scale[kMaxLanes];
  TO* out[kMaxLanes];
  Skip skip[kMaxLanes];
};
template <typename TI, typename TO>
__device__ __forceinline__ void gather_rows(int n, const int* __restrict__ perm, const TI* __restrict__ in,
                                            const double* __restrict__ scale, TO* __restrict__ out) {
  const double s = scale ? *scale : 1.0;
  const int stride = gridDim.x * blockDim.x * kPermUnroll;
  for (int base = blockIdx.x * blockDim.x * kPermUnroll + threadIdx.x; base < n; base += stride) {
    int p[kPermUnroll];
#pragma unroll
    for (int u = 0; u < kPermUnroll; u++) {
      const int i = base + u * blockDim.x;
      p[u] = i < n ? (perm ? __ldg(&perm[i]) : i) : -1;
    }
    TI v[kPermUnroll];
#pragma unroll
    for (int u = 0; u < kPermUnroll; u++) v[u] = p[u] >= 0 ? in[p[u]] : TI(0);
#pragma unroll
    for (int u = 0; u < kPermUnroll; u++) {
      const int i = base + u * blockDim.x;
      if (i < n) out[i] = scale ? to<TO>(to<typename Sc<TI>::acc>(v[u]) * s) : to<TO>(v[u]);
    }
  }
}

template <typename TI, typename TO>
__global__ void __launch_bounds__(256) gather_kernel(int n, const int* __restrict__ perm, const TI* __restrict__ in,
                                                     const double* __restrict__ scale, TO* __restrict__ out,
                                                     Skip skip) {
  if (!skip.on()) gather_rows<TI, TO>(n, perm, in, scale, out);
}
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) gather_lanes_kernel(int n, const int* __restrict__ perm,
                                                           const __grid_constant__ PermLanes<TI, TO> p) {
  const int r = blockIdx.y;
  if (!p.skip[r].on()) gather_rows<TI, TO>(n, perm, p.in[r], p.scale[r], p.out[r]);
}

// y += x  (the solution update of the multiplicative level solve)
template <typename T>
__global__ void __launch_bounds__(256) axpy_kernel(int n, const T* __restrict__ x, T* __restrict__ y, Skip skip) {
  if (skip.on()) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] += x[i];
}

// out[perm[i]] = in[i]  (IntVectorClass::ScatterRperm, int_vector.cpp:629)
template <typename TI, typename TO>
__device__ __forceinline__ void scatter_rows(int n, const int* __restrict__ perm, const TI* __restrict__ in,
                                             TO* __restrict__ out) {
  const int stride = gridDim.x * blockDim.x * kPermUnroll;
  for (int base = blockIdx.x * blockDim.x * kPermUnroll + threadIdx.x; base < n; base += stride) {
    int p[kPermUnroll];
    TI v[kPermUnroll];
#pragma unroll
    for (int u = 0; u < kPermUnroll; u++) {
      const int i = base + u * blockDim.x;
      p[u] = i < n ? (perm ? __ldg(&perm[i]) : i) : -1;
      v[u] = i < n ? in[i] : TI(0);
    }
#pragma unroll
    for (int u = 0; u < kPermUnroll; u++)
      if (p[u] >= 0) out[p[u]] = to<TO>(v[u]);
  }
}

template <typename TI, typename TO>
__global__ void __launch_bounds__(256) scatter_kernel(int n, const int* __restrict__ perm, const TI* __restrict__ in,
                                                      TO* __restrict__ out, Skip skip) {
  if (!skip.on()) scatter_rows<TI, TO>(n, perm, in, out);
}
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) scatter_lanes_kernel(int n, const int* __restrict__ perm,
                                                            const __grid_constant__ PermLanes<TI, TO> p) {
  const int r = blockIdx.y;
  if (!p.skip[r].on()) scatter_rows<TI, TO>(n, perm, p.in[r], p.out[r]);
}

template <typename T>
__global__ void fill_kernel(int n, T v, T* out, Skip skip) {
  if (skip.on()) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = v;
}

}  // namespace pgx
