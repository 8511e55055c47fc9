// FP64 iterative refinement around an FP32 factor (precision form).
//
// Each step computes r = b - A x with the original matrix in FP64, measures the
// backward error eta = ||r||_inf / (||A||_inf ||x||_inf + ||b||_inf) per
// right-hand side and per system (a batch of block-diagonal systems is measured
// system by system, with that system's own norms), solves A d = r with the FP32 factor and updates x += d in FP64.
// A is held as full symmetric CSR in the original ordering; its values are
// gathered from the lower-triangle input on every DistributeMatrix.
#include <type_traits>

#include "kernels.cuh"

namespace spb {
namespace dev {

namespace {

int grid_for(int64_t work, int threads) {
  int64_t g = (work + threads - 1) / threads;
  if (g > 148 * 16) g = 148 * 16;
  return g < 1 ? 1 : (int)g;
}

__global__ void k_gather(double* __restrict__ dst, const double* __restrict__ src, const int64_t* __restrict__ idx,
                         int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[idx[i]];
}

// Non-negative doubles order like their bit patterns, a NaN above infinity: maxima through
// 64-bit integers keep it, where fmax would drop it.
__device__ __forceinline__ double max_nonneg(double a, double b) {
  return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

// Per-system maxima.  Rows are grouped into systems (segments) given by
// rowseg[i] (nullptr: one system); out[seg * 64 + c] = max |v[i + c*ld]| over
// the rows i of that system.  Each CTA takes a contiguous chunk of rows, each
// thread keeps a running maximum while its rows stay in one system, and a warp
// whose lanes end in the same system merges before the atomic.  out zeroed by
// the caller.
constexpr int kChunk = 1024;

__device__ __forceinline__ void flush_segmax(double* out, int seg, double m) {
  const unsigned full = 0xffffffffu;
  const int seg0 = __shfl_sync(full, seg, 0);
  if (__all_sync(full, seg == seg0)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max_nonneg(m, __shfl_xor_sync(full, m, o));
    if ((threadIdx.x & 31) == 0 && seg0 >= 0) atomic_max_nonneg(out + seg0 * 64, m);
  } else if (seg >= 0) {
    atomic_max_nonneg(out + seg * 64, m);
  }
}

__global__ void k_segmax(const double* __restrict__ v, int n, int64_t ld, const int32_t* __restrict__ rowseg,
                         double* __restrict__ out) {
  const int64_t r0 = (int64_t)blockIdx.x * kChunk;
  const int64_t r1 = min((int64_t)n, r0 + kChunk);
  {
    const int c = blockIdx.y;
    int seg = -1;
    double m = 0.0;
    for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
      const int si = rowseg ? rowseg[i] : 0;
      if (si != seg) {
        if (seg >= 0) atomic_max_nonneg(out + seg * 64 + c, m);
        seg = si;
        m = 0.0;
      }
      m = max_nonneg(m, fabs(v[i + c * ld]));
    }
    flush_segmax(out + c, seg, m);
  }
}

// One refinement step's view of the current x: r = b - A x, stored permuted (R[invp[i] + c n],
// the right-hand side of the correction solve), with max |x| and max |r| per system and
// column (xmax, rmax; layout as in k_segmax) taken on the way and Z and the counters cleared
// for the correction's sweeps.  Bound by the reads of A: LPR lanes
// share a row, so that a load of val takes whole sectors, and CB columns share each
// entry of A, so that A is read ceil(nrhs / CB) times.  A block takes a contiguous run of rows
// and keeps its maxima in registers to the end of the run (or of a system).  27-point 36^3, 50
// columns: the warp-per-entry kernel and the two passes for the maxima took 0.73 ms a step.
// Four lanes share a short row, a warp the rows of matrices with more than kWarpRow entries a
// row on average (refined solve of one right-hand side, dense n = 1,000: 297 us with 4 lanes,
// 177 with 32; 42 entries a row: equal).  Rows beyond kLongRow entries are left to the whole
// block at the end (n = 50,000 with one full row: 6.58 ms with 4 lanes on it, 0.38 so).
constexpr int kLongRow = 1024, kLongRows = 64, kWarpRow = 64;
constexpr int kResThreads = 256;
template <int CB, int LPR>
__global__ void __launch_bounds__(kResThreads) k_residual(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                                                          const double* __restrict__ val, const double* __restrict__ x,
                                                          int64_t ldx, const double* __restrict__ b, int64_t ldb,
                                                          double* __restrict__ R, const int32_t* __restrict__ invp0,
                                                          int n, int nrhs, const int32_t* __restrict__ rowseg,
                                                          double* __restrict__ xmax, double* __restrict__ rmax,
                                                          double* __restrict__ Z, int32_t* __restrict__ sync,
                                                          int64_t nsync) {
  constexpr int kOwn = (CB + LPR - 1) / LPR;  // columns whose sums a lane finishes
  __shared__ unsigned long long smax[2][CB];
  __shared__ double part[kResThreads / 32][CB];
  __shared__ int nlong, longs[kLongRows];
  const int c0 = blockIdx.y * CB, nc = min(CB, nrhs - c0), q = threadIdx.x & (LPR - 1);
  for (int64_t i = (blockIdx.y * (int64_t)gridDim.x + blockIdx.x) * kResThreads + threadIdx.x; i < nsync;
       i += (int64_t)gridDim.x * gridDim.y * kResThreads)
    sync[i] = 0;
  if (threadIdx.x < 2 * CB) smax[threadIdx.x / CB][threadIdx.x % CB] = 0;
  if (threadIdx.x == 0) nlong = 0;
  __syncthreads();
  constexpr int kRows = kResThreads / LPR;
  const int64_t chunk = ((n + gridDim.x - 1) / gridDim.x + kRows - 1) / kRows * kRows;
  const int64_t r0 = blockIdx.x * chunk, r1 = min((int64_t)n, r0 + chunk);
  double mr[kOwn], mx[kOwn];
#pragma unroll
  for (int o = 0; o < kOwn; ++o) mr[o] = mx[o] = 0.0;
  int seg = -1;
  for (int64_t base = r0; base < r1; base += kRows) {
    const int64_t i = base + threadIdx.x / LPR;
    bool in = i < r1;
    double s[CB], bv[kOwn], xv[kOwn];
    int64_t pr = 0, p0 = 0, p1 = 0;
#pragma unroll
    for (int c = 0; c < CB; ++c) s[c] = 0.0;
    if (in) {
      p1 = rowptr[i + 1], p0 = rowptr[i] + q;
      if (p1 - p0 + q > kLongRow) {  // to the list, while it has room
        const unsigned group = 0xffffffffu >> (32 - LPR) << (threadIdx.x & 31 & ~(LPR - 1));
        int at = q == 0 ? atomicAdd(&nlong, 1) : 0;
        at = __shfl_sync(group, at, 0, LPR);
        if (at < kLongRows) {
          if (q == 0) longs[at] = (int)i;
          in = false;
        }
      }
    }
    if (in) {  // everything that does not depend on the row's entries first
      pr = invp0[i];
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int c = LPR * o + q;
        bv[o] = c < nc ? b[i + (c0 + c) * ldb] : 0.0;
        xv[o] = c < nc ? x[i + (c0 + c) * ldx] : 0.0;
      }
      for (int64_t p = p0; p < p1; p += 2 * LPR) {  // two of the lane's entries at a time
        const bool two = p + LPR < p1;
        const double v0 = val[p], v1 = two ? val[p + LPR] : 0.0;
        const double* x0 = x + col[p] + c0 * ldx;
        const double* x1 = two ? x + col[p + LPR] + c0 * ldx : x0;
#pragma unroll
        for (int c = 0; c < CB; ++c)
          if (c < nc) s[c] = fma(v1, two ? x1[c * ldx] : 0.0, fma(v0, x0[c * ldx], s[c]));
      }
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < CB; ++c)
#pragma unroll
      for (int o = 1; o < LPR; o *= 2) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
    if (!in) continue;
    if (rowseg && rowseg[i] != seg) {
      if (seg >= 0) {
#pragma unroll
        for (int o = 0; o < kOwn; ++o) {
          const int c = LPR * o + q;
          if (c >= nc) continue;
          atomic_max_nonneg(rmax + seg * 64 + c0 + c, mr[o]);
          atomic_max_nonneg(xmax + seg * 64 + c0 + c, mx[o]);
          mr[o] = mx[o] = 0.0;
        }
      }
      seg = rowseg[i];
    }
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const int c = LPR * o + q;
      if (c >= nc) continue;
      double sum = s[0];
#pragma unroll
      for (int e = 1; e < CB; ++e)
        if (e / LPR == o && c == e) sum = s[e];
      const double r = bv[o] - sum;
      R[pr + (int64_t)(c0 + c) * n] = r;
      Z[i + (int64_t)(c0 + c) * n] = 0.0;
      mr[o] = max_nonneg(mr[o], fabs(r));
      mx[o] = max_nonneg(mx[o], fabs(xv[o]));
    }
  }
  __syncthreads();
  const int listed = min(nlong, kLongRows);
  for (int k = 0; k < listed; ++k) {  // a long row: every thread its share, summed over the block
    const int64_t i = longs[k], p1 = rowptr[i + 1];
    double s[CB];
#pragma unroll
    for (int c = 0; c < CB; ++c) s[c] = 0.0;
#pragma unroll 2
    for (int64_t p = rowptr[i] + threadIdx.x; p < p1; p += kResThreads) {
      const double v = val[p];
      const double* xp = x + col[p] + c0 * ldx;
#pragma unroll
      for (int c = 0; c < CB; ++c)
        if (c < nc) s[c] = fma(v, xp[c * ldx], s[c]);
    }
#pragma unroll
    for (int c = 0; c < CB; ++c) {
#pragma unroll
      for (int o = 1; o < 32; o *= 2) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
      if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][c] = s[c];
    }
    __syncthreads();
    if (threadIdx.x < nc) {
      const int c = threadIdx.x;
      double sum = 0.0;
#pragma unroll
      for (int w = 0; w < kResThreads / 32; ++w) sum += part[w][c];
      const double r = b[i + (c0 + c) * ldb] - sum, xi = fabs(x[i + (c0 + c) * ldx]);
      R[invp0[i] + (int64_t)(c0 + c) * n] = r;
      Z[i + (int64_t)(c0 + c) * n] = 0.0;
      const int sg = rowseg ? rowseg[i] : 0;
      atomic_max_nonneg(rmax + sg * 64 + c0 + c, fabs(r));
      atomic_max_nonneg(xmax + sg * 64 + c0 + c, xi);
    }
    __syncthreads();
  }
  if (rowseg) {
    if (seg >= 0) {
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int c = LPR * o + q;
        if (c >= nc) continue;
        atomic_max_nonneg(rmax + seg * 64 + c0 + c, mr[o]);
        atomic_max_nonneg(xmax + seg * 64 + c0 + c, mx[o]);
      }
    }
    return;
  }
#pragma unroll
  for (int o = 0; o < kOwn; ++o) {
    const int c = LPR * o + q;
    if (c >= nc) continue;
    atomicMax(&smax[0][c], (unsigned long long)__double_as_longlong(mr[o]));
    atomicMax(&smax[1][c], (unsigned long long)__double_as_longlong(mx[o]));
  }
  __syncthreads();
  if (threadIdx.x < nc) {
    atomicMax(reinterpret_cast<unsigned long long*>(rmax + c0 + threadIdx.x), smax[0][threadIdx.x]);
    atomicMax(reinterpret_cast<unsigned long long*>(xmax + c0 + threadIdx.x), smax[1][threadIdx.x]);
  }
}

// anorm[seg] = max over the rows i of the system of sum_j |A_ij|
__global__ void k_rowsum_segmax(const int64_t* __restrict__ rowptr, const double* __restrict__ val, int n,
                                const int32_t* __restrict__ rowseg, double* __restrict__ anorm) {
  const int64_t r0 = (int64_t)blockIdx.x * kChunk;
  const int64_t r1 = min((int64_t)n, r0 + kChunk);
  int seg = -1;
  double m = 0.0;
  for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    const int si = rowseg ? rowseg[i] : 0;
    if (si != seg) {
      if (seg >= 0) atomic_max_nonneg(anorm + seg, m);
      seg = si;
      m = 0.0;
    }
    double s = 0.0;
    for (int64_t p = rowptr[i]; p < rowptr[i + 1]; ++p) s += fabs(val[p]);
    m = max_nonneg(m, s);
  }
  const unsigned full = 0xffffffffu;
  const int seg0 = __shfl_sync(full, seg, 0);
  if (__all_sync(full, seg == seg0)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max_nonneg(m, __shfl_xor_sync(full, m, o));
    if ((threadIdx.x & 31) == 0 && seg0 >= 0) atomic_max_nonneg(anorm + seg0, m);
  } else if (seg >= 0) {
    atomic_max_nonneg(anorm + seg, m);
  }
}

// eta[0] = max over systems and right-hand sides of rmax / (anorm * xmax + bmax), the normwise
// backward error of every system by itself, over those where all four are finite; eta[1] = 1
// when there are others.
__global__ void k_eta(const double* __restrict__ anorm, const double* __restrict__ bmax,
                      const double* __restrict__ xmax, const double* __restrict__ rmax, int nseg, int nrhs,
                      double* __restrict__ eta) {
  double e = 0.0;
  bool bad = false;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nseg * nrhs; k += gridDim.x * blockDim.x) {
    const int seg = k / nrhs, c = k - seg * nrhs;
    const double an = anorm[seg], b = bmax[seg * 64 + c], x = xmax[seg * 64 + c], r = rmax[seg * 64 + c];
    if (!isfinite(an) || !isfinite(b) || !isfinite(x) || !isfinite(r)) {
      bad = true;
      continue;
    }
    const double den = an * x + b;
    e = max_nonneg(e, den > 0.0 ? r / den : (r > 0.0 ? 1e300 : 0.0));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e = max_nonneg(e, __shfl_xor_sync(0xffffffffu, e, o));
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    atomic_max_nonneg(eta, e);
    if (bad) atomic_max_nonneg(eta + 1, 1.0);
  }
}

}  // namespace

void launch_gather(cudaStream_t st, double* dst, const double* src, const int64_t* idx, int64_t n) {
  if (n > 0) k_gather<<<grid_for(n, 256), 256, 0, st>>>(dst, src, idx, n);
}

void launch_residual(cudaStream_t st, const int64_t* rowptr, const int32_t* col, const double* val, const double* x,
                     int64_t ldx, const double* b, int64_t ldb, double* R, const int32_t* invp0, int n, int64_t nnz,
                     int nrhs, const int32_t* rowseg, double* xmax, double* rmax, double* Z, int32_t* sync,
                     int64_t nsync) {
  auto run = [&](auto cb, auto lpr) {
    constexpr int CB = decltype(cb)::value, LPR = decltype(lpr)::value, kRows = kResThreads / LPR;
    const int by = (nrhs + CB - 1) / CB, rows = (n + kRows - 1) / kRows, cap = (148 * 16 + by - 1) / by;
    k_residual<CB, LPR><<<dim3(rows < cap ? rows : cap, by), kResThreads, 0, st>>>(
        rowptr, col, val, x, ldx, b, ldb, R, invp0, n, nrhs, rowseg, xmax, rmax, Z, sync, nsync);
  };
  auto lanes = [&](auto cb) {
    if (nnz > kWarpRow * (int64_t)n) run(cb, std::integral_constant<int, 32>());
    else run(cb, std::integral_constant<int, 4>());
  };
  if (nrhs == 1) lanes(std::integral_constant<int, 1>());
  else if (nrhs <= 4) lanes(std::integral_constant<int, 4>());
  else lanes(std::integral_constant<int, 8>());
}

void launch_segmax(cudaStream_t st, const double* v, int n, int nrhs, int64_t ld, const int32_t* rowseg,
                   double* out) {
  k_segmax<<<dim3((n + kChunk - 1) / kChunk, nrhs), 256, 0, st>>>(v, n, ld, rowseg, out);
}

void launch_rowsum_segmax(cudaStream_t st, const int64_t* rowptr, const double* val, int n, const int32_t* rowseg,
                          double* anorm) {
  k_rowsum_segmax<<<(n + kChunk - 1) / kChunk, 256, 0, st>>>(rowptr, val, n, rowseg, anorm);
}

void launch_eta(cudaStream_t st, const double* anorm, const double* bmax, const double* xmax, const double* rmax,
                int nseg, int nrhs, double* eta) {
  k_eta<<<grid_for((int64_t)nseg * nrhs, 256), 256, 0, st>>>(anorm, bmax, xmax, rmax, nseg, nrhs, eta);
}

}  // namespace dev
}  // namespace spb
