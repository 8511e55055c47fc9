// Device bodies of the panel tasks of the supernodal factorization (sm_100a),
// shared by the per-step kernels (kernels.cu) and the persistent factorization
// kernel (gemm.cu).  Every body works with the whole thread block (any multiple of
// 32 threads for the small panel, 256 for the others) and the shared memory it is given.
//
// Numerics follow symPACK's blockCell_t operations (symPACKMatrix2D.hpp):
//   factorize   1052-1102  Potrf of the diagonal block
//   trsm        1104-1178  L_KI = A_KI * L_II^-T
// on a column-major panel per supernode instead of row-major cells.
// LDL^T (blockCellLDL_t, 2D.hpp:1802-2465): Potrf_LDL of the diagonal block
// (lapack.hpp:206-560, no pivoting, a zero pivot is reported), unit TRSM then
// scaling by 1/D (2D.hpp:2118-2137).
#pragma once
#include <type_traits>
#include "kernels.cuh"

namespace spb {
namespace dev {
namespace ftask {
namespace {

// threadIdx.x, read anew: inside the persistent kernel's task loop the compiler would keep
// every value that a task derives from it in registers across all the other tasks.
__device__ __forceinline__ int thread_id() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

__device__ __forceinline__ void report(Status* st, int code, int s, int col) {
  if (atomicCAS(&st->code, 0, code) == 0) {
    st->supernode = s;
    st->column = col;
  }
}

// Split copy of final FP32 panel rows (TMA-fed tcgen05 tiles): tf32 hi part (round to
// nearest, ties away) and the rounded remainder, row-major, hi block then lo block.
__device__ __forceinline__ void split_store(const FactorArgs& a, const SnMeta& m, int64_t off, int r, int c, float x) {
  uint32_t hi, lo;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
  const int64_t pitch = (m.w + 3) & ~3;
  float* p = a.split + off + (int64_t)r * pitch + c;
  p[0] = __uint_as_float(hi);
  p[(int64_t)m.h * pitch] = __uint_as_float(lo);
}
// A panel task's writes that update tiles read through the async proxy (the split copies by
// TMA, FP64 panels by bulk copies) come before the copies of the tiles that wait for this
// task's counters: executed by the threads that wrote, before the barrier of the release.
__device__ __forceinline__ void async_fence() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

constexpr int kNB = 64;
constexpr int kThreads = 256;  // threads of the POTRF and TRSM kernels

// FP64 tensor-core step, D = A(16x4, row) * B(4x8, col) + D (lane = 4*g + t):
//   a0 = A[g][t], a1 = A[g+8][t], b0 = B[t][g],
//   d0 = D[g][2t], d1 = D[g][2t+1], d2 = D[g+8][2t], d3 = D[g+8][2t+1].
__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Leading dimension of a 64-row block in shared memory: 4 mod 16 doubles, so that the 8 x 4
// fragment reads of a half warp fall on different banks.
constexpr int kDL = kNB + 4;
// scratch slot: factored block (FP64), 1/L_kk, and (LDL^T) 1/D_kk
constexpr size_t kSlot = kDiagSlotDoubles;
static_assert(kSlot >= (size_t)kNB * kNB + 2 * kNB, "slot layout");
constexpr int kPiece = 8;

// One warp factors an 8 x 8 diagonal piece and solves up to 24 rows below it.  Lanes 0 .. 7
// hold the piece's rows (lower triangle; entries above the diagonal are carried along and
// meaningless), lanes 8 .. 31 a row each, 8 entries x.  A column takes the pivot and the
// column's entries from their lanes by shuffles, so that every lane issues the same 28 FMAs:
// a warp issues an FP64 instruction every 8 cycles or so, which is what the chain of pivots
// costs (the piece factored redundantly by every lane, 120 FMAs, took 1.2 us a piece).
// Cholesky: rs = 1 / L_kk, x becomes row L^-T, and lane k keeps the pivot d_k as x[k] for its
// consumer to take sqrt of beside the chain (L_kk = d_k rs would round d_k's root twice over,
// and L_kk^2 twice that: residual of the factor 18 % larger on a 100 x 103 grid); a pivot not
// > 0 is reported (who: this warp reports) and replaced by 1.  LDL^T (Potf2_LDL, lapack.hpp:206-270, lower triangle): d_k =
// A_kk, |d_k| > 0 or reported; rs = 1 / d_k, x becomes the row's entries of L D.  Reported
// pivots: column col + k of supernode s, k < valid.
// kShort: a piece of fewer than 8 columns ends there (valid of them), else its padding is factored too.
template <bool kLdl, bool kShort>
__device__ __forceinline__ void piece_rows(double (&x)[kPiece], double (&rs)[kPiece], bool who, int valid,
                                           Status* status, int s, int col) {
  const int lane = thread_id() & 31;
  double own = x[0];  // lane k: its pivot, kept ahead of the row's other entries
#pragma unroll
  for (int k = 0; k < kPiece; ++k) {
    if (kShort && k >= valid) {
      rs[k] = 1.0;
      continue;
    }
    const double d = __shfl_sync(0xffffffffu, own, k);
    rs[k] = kLdl ? 1.0 / d : rsqrt(d);
    if (kLdl ? !(fabs(d) > 0.0) : !(d > 0.0)) {
      if (who && lane == k && k < valid) report(status, 1, s, col + k);
      rs[k] = 1.0;
      if (lane == k) x[k] = 1.0;
    }
    const double y = x[k] * rs[k];          // the row's entry of L
    const double l = kLdl ? x[k] : y;
    if (k + 1 < kPiece) own = fma(-l, y, x[k + 1]);
#pragma unroll
    for (int j = k + 1; j < kPiece; ++j) x[j] = fma(-l, __shfl_sync(0xffffffffu, y, j), x[j]);
    if constexpr (!kLdl) x[k] = lane == k ? (d > 0.0 ? d : 1.0) : y;
  }
}

// Small panel s factored whole in shared memory, and (panels of at most kFuseRows
// off-diagonal rows, Plan::fuses_update) its external update scattered from there: the
// update's operands are already on the SM and no second task has to wait for the first.
// Right-looking by 8-column pieces (piece_rows), the trailing columns of
// the panel by a warp per column; the update's 16 x 8 tiles on the FP64 tensor pipe, in FP64
// for FP32 panels too, scattered from the accumulators through the relative indices, whose
// column tables are fetched while the panel is loaded.  Bound by latency: global round trips
// and the chain of pivots.  463 x 467 grid: 5.9 us a panel with its update; the panel by
// single columns took 6.1 us and the separate 64 x 64 update task 5.4 us and a dispatch.
// sm: kSmallHeadDoubles doubles (D of LDL^T, column tables), then the panel; cap = doubles of
// shared memory.
template <class T, bool kLdl>
__device__ __forceinline__ void factor_small_task(const FactorArgs& a, int s, const SnMeta& meta, double* sm, int cap) {
  const SnMeta m = meta;
  const int h = m.h, w = m.w, M = h - w;
  double* Dk = sm;
  int64_t* cbase = reinterpret_cast<int64_t*>(sm + kSmallDEntries);
  int64_t* crel = cbase + kFuseRows;
  double* P = sm + kSmallHeadDoubles;
  const int pad = (h + 11) / 16 * 16 + 4;  // 4 mod 16: conflict-free fragment reads
  const int ldp = pad * w + kSmallHeadDoubles <= cap ? pad : h;
  const int tid = thread_id(), nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;
  T* gl = static_cast<T*>(a.L) + m.off;
  const bool fuse = fuses_update(m, a.big_rows);
  const float rh = 1.0f / h;
  for (int base = tid; base < h * w; base += 8 * nthr) {
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int idx = base + q * nthr, c = (int)((idx + 0.5f) * rh), r = idx - c * h;
      v[q] = idx < h * w ? (double)gl[r + (int64_t)c * m.ld] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int idx = base + q * nthr, c = (int)((idx + 0.5f) * rh), r = idx - c * h;
      if (idx < h * w) P[r + c * ldp] = v[q];
    }
  }
  if (fuse)
    for (int c = tid; c < M; c += nthr) {
      const RelGroup g = a.groups[a.row_group[m.lidx + w + c]];
      const SnMeta mt = a.meta[g.t];
      cbase[c] = mt.off + (int64_t)(a.rows[m.lidx + w + c] - mt.fc) * mt.ld;
      crel[c] = g.rel_off - g.j0;
    }
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < w; kb += kPiece) {
    const int pw = min(kPiece, w - kb);  // a narrower last piece is padded with the identity
    // a warp takes the piece's rows and 24 rows below it, then (tall panels) more of those
    const int below = h - kb - pw;  // rows below the piece
    const bool active = warp == 0 || 24 * warp < below;
    double x[kPiece], rs[kPiece];
    int r = lane < kPiece ? kb + lane : kb + pw + 24 * warp + lane - kPiece;
    if (active) {
#pragma unroll
      for (int j = 0; j < kPiece; ++j)
        x[j] = r < h && j < pw && (lane < pw || lane >= kPiece) ? P[r + (kb + j) * ldp] : (lane == j ? 1.0 : 0.0);
      piece_rows<kLdl, true>(x, rs, warp == 0, pw, a.status, s, m.fc + kb);
    }
    __syncthreads();  // every warp has the piece before its rows are overwritten
    if (active) {
      // entries above the diagonal of the piece are written too; nothing reads them
      auto put = [&](const double (&v)[kPiece], int row) {
#pragma unroll
        for (int j = 0; j < kPiece; ++j)
          if (j < pw) P[row + (kb + j) * ldp] = kLdl ? v[j] * rs[j] : v[j];
      };
      if (lane < kPiece ? warp == 0 && lane < pw : r < h) put(x, r);
      if constexpr (kLdl) {
        if (warp == 0) {
#pragma unroll
          for (int j = 0; j < kPiece; ++j)
            if (lane == j && j < pw) {
              Dk[kb + j] = x[j];
              P[kb + j + (kb + j) * ldp] = 1.0;
            }
        }
      }
      for (int r0 = kb + pw + 24 * (warp + nw); r0 < h; r0 += 24 * nw) {
        r = r0 + lane - kPiece;
        const bool in = lane >= kPiece && r < h;
        double y[kPiece];
#pragma unroll
        for (int j = 0; j < kPiece; ++j) y[j] = in && j < pw ? P[r + (kb + j) * ldp] : 0.0;
#pragma unroll
        for (int k = 0; k < kPiece; ++k) {
          const double l = kLdl ? x[k] * rs[k] : x[k];
          if constexpr (!kLdl) y[k] *= rs[k];
#pragma unroll
          for (int j = k + 1; j < kPiece; ++j) y[j] = fma(-y[k], __shfl_sync(0xffffffffu, l, j), y[j]);
        }
        if (in) put(y, r);
      }
    }
    __syncthreads();
    if (kb + kPiece < w) {
      for (int j = kb + kPiece + warp; j < w; j += nw) {
        double y[kPiece];
#pragma unroll
        for (int k = 0; k < kPiece; ++k) y[k] = P[j + (kb + k) * ldp] * (kLdl ? Dk[kb + k] : 1.0);
        for (int i = j + lane; i < h; i += 32) {
          double t0 = P[i + j * ldp], t1 = 0.0;
#pragma unroll
          for (int k = 0; k < kPiece; k += 2) {
            t0 = fma(-P[i + (kb + k) * ldp], y[k], t0);
            t1 = fma(-P[i + (kb + k + 1) * ldp], y[k + 1], t1);
          }
          P[i + j * ldp] = t0 + t1;
        }
      }
      __syncthreads();
    }
  }
  double* gw = kLdl ? a.W + m.off : nullptr;
  for (int idx = tid; idx < h * w; idx += nthr) {
    const int c = (int)((idx + 0.5f) * rh), r = idx - c * h;
    if (kLdl ? r < c : r <= c) continue;
    const double v = P[r + c * ldp];
    gl[r + (int64_t)c * m.ld] = (T)v;
    if constexpr (kLdl) gw[r + (int64_t)c * m.ld] = v * Dk[c];
  }
  if constexpr (!kLdl) {  // the last warp: the diagonal, from the pivots
    if (warp == nw - 1)
      for (int c = lane; c < w; c += 32) gl[c + (int64_t)c * m.ld] = (T)sqrt(P[c + c * ldp]);
  }
  if constexpr (std::is_same<T, double>::value) {
    if (!fuse) async_fence();  // a fused panel has no update tiles
  }
  if constexpr (std::is_same<T, float>::value) {
    const int64_t off = a.split ? a.split_off[s] : -1;
    if (off >= 0) {  // off-diagonal rows, row by row (consecutive threads take consecutive columns)
      for (int idx = tid; idx < M * w; idx += nthr) {
        const int r = w + idx / w, c = idx % w;
        split_store(a, m, off, r, c, (float)P[r + c * ldp]);
      }
      async_fence();
    }
  }
  if (!fuse) return;
  // ancestors -= L_K L_K^T over the lower triangle of the off-diagonal rows: a warp takes
  // 8-column tiles, keeps their fragments and walks the 16-row tiles at and below them
  const int g = lane >> 2, t = lane & 3, ks = (w + 3) >> 2;
  T* L = static_cast<T*>(a.L);
  const double* Po = P + w;
  for (int n = warp; 8 * n < M; n += nw) {
    const int c0 = 8 * n + 2 * t, c1 = c0 + 1, cb = 8 * n + g;
    const int64_t b0 = c0 < M ? cbase[c0] : 0, b1 = c1 < M ? cbase[c1] : 0;
    const int64_t q0 = c0 < M ? crel[c0] + w : 0, q1 = c1 < M ? crel[c1] + w : 0;
    // a row's places in the two columns' targets, fetched one tile ahead
    int pos[4] = {0, 0, 0, 0};
    auto place = [&](int i) {
      const int r0 = 16 * i + g, r1 = r0 + 8;
      if (r0 < M && r0 >= c0) pos[0] = a.rel[q0 + r0];
      if (r0 < M && r0 >= c1) pos[1] = a.rel[q1 + r0];
      if (r1 < M && r1 >= c0) pos[2] = a.rel[q0 + r1];
      if (r1 < M && r1 >= c1) pos[3] = a.rel[q1 + r1];
    };
    place(n / 2);
    for (int i = n / 2; 16 * i < M; ++i) {
      const int r0 = 16 * i + g, r1 = r0 + 8;
      const int p0 = pos[0], p1 = pos[1], p2 = pos[2], p3 = pos[3];
      if (16 * (i + 1) < M) place(i + 1);
      double d[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = 0; k < ks; ++k) {
        const int kk = 4 * k + t;
        const bool in = kk < w;
        double y = in && cb < M ? Po[cb + kk * ldp] : 0.0;
        if (kLdl && in) y *= Dk[kk];
        dmma(d, in && r0 < M ? Po[r0 + kk * ldp] : 0.0, in && r1 < M ? Po[r1 + kk * ldp] : 0.0, y);
      }
      if (r0 < M && r0 >= c0) atomicAdd(L + b0 + p0, (T)(-d[0]));
      if (r0 < M && r0 >= c1) atomicAdd(L + b1 + p1, (T)(-d[1]));
      if (r1 < M && r1 >= c0) atomicAdd(L + b0 + p2, (T)(-d[2]));
      if (r1 < M && r1 >= c1) atomicAdd(L + b1 + p3, (T)(-d[3]));
    }
  }
}

// Shared memory (doubles) of diag_task: the block, 1 / L_kk, D_kk, two pieces' columns of L D.
constexpr int kDiagSmemDoubles = kNB * kDL + 2 * kNB + 2 * kPiece * kDL;

// POTRF (or LDL^T) of one 64-column diagonal block [c0, c0+nb) of a wide panel (one CTA per
// item), right-looking by 8-column pieces.  On the critical path of every wide supernode and
// bound by its dependency chain (8 pieces of 8 pivots), so everything else is kept off it.
// Warps 3-7 hold the block's columns as tensor-core accumulators, 8 columns a tile.  For a
// piece the tile's warp lays its columns in shared memory, warps 0-2 factor it and solve the
// rows below (piece_rows), then every later tile takes the solved columns off with 2 MMA
// steps per 16 rows, the next piece's tile first: the second step from zero and added, five
// roundings of an entry a piece instead of eight (residual of the factor, 27-point 17^3 6.4e-17
// -> 5.9e-17; the scalar version split its sums alike).  The solving warps wait for that tile only;
// finished columns and the pieces' inverses are written out beside the next pieces.
// The scratch slot gets the factored block (FP64) with the inverses of its 8 x 8 diagonal
// pieces transposed into their upper triangles, 1/L_kk (1 for LDL^T, whose TRSM then computes
// W's rows) and 1/D_kk.  11 us a block measured alone, 13 to 18 us beside other tasks; the
// scalar version (the trailing triangle as a chain of shared-memory FMAs) took 19 to 25 us.
// LDL^T: L takes the unit block, W the block times D (its diagonal is D).  A block narrower
// than 64 is padded with the identity.
template <class T, bool kLdl>
__device__ __forceinline__ void diag_task(const FactorArgs& a, const PanelItem& it, const SnMeta& meta,
                                         double* __restrict__ winv, double* sm) {
  double* D = sm;
  double* Rinv = sm + kNB * kDL;  // 1 / L_kk (LDL^T: 1)
  double* Dk = Rinv + kNB;        // LDL^T: D_kk
  double* Wp = Dk + kNB;          // LDL^T: the columns of L D of this piece and the one before, ld kDL
  const SnMeta m = meta;
  T* gl = static_cast<T*>(a.L) + m.off;
  const int nb = it.nb, c0 = it.c0;
  const int64_t ld = m.ld;
  const int tid = thread_id(), lane = tid & 31, warp = tid >> 5;
  constexpr int kPieces = kNB / kPiece;
  double* W = winv ? winv + (size_t)it.slot * kSlot : nullptr;
  // inverse of piece p, lane j its column j, into the upper triangle of the scratch slot's piece
  auto invert = [&](int p) {
    if (!W || lane >= kPiece) return;
    const int kb = kPiece * p;
    double z[kPiece];
#pragma unroll
    for (int i = 0; i < kPiece; ++i) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) v = fma(D[kb + i + (kb + k) * kDL], z[k], v);  // z[k] = 0 for k < lane
      z[i] = i < lane ? 0.0 : i == lane ? Rinv[kb + i] : -v * Rinv[kb + i];
    }
#pragma unroll
    for (int i = 1; i < kPiece; ++i)
      if (i > lane) W[kb + lane + (kb + i) * kNB] = z[i];
  };
  // barriers: 1 the solving warps, 2 they and the next piece's owner, 3 everybody
  if (warp < 3) {
#pragma unroll 1
    for (int p = 0; p < kPieces; ++p) {
      const int kb = p * kPiece;
      asm volatile("bar.sync 2, 128;\n" ::: "memory");
      const int row = lane < kPiece ? kb + lane : kb + 24 * warp + lane;
      const bool active = warp == 0 || kb + 24 * warp + kPiece < kNB;
      double x[kPiece], rs[kPiece];
      if (active) {
#pragma unroll
        for (int j = 0; j < kPiece; ++j) x[j] = row < kNB ? D[row + (kb + j) * kDL] : 0.0;
        piece_rows<kLdl, false>(x, rs, warp == 0, nb - kb, a.status, it.s, m.fc + c0 + kb);
      } else if (warp == 2) {  // no rows left for it: the piece before's inverse
        invert(p - 1);
      }
      asm volatile("bar.sync 1, 96;\n" ::: "memory");  // all have the piece before its rows change
      if (active && (lane < kPiece ? warp == 0 : row < kNB)) {  // the piece's upper entries too; nothing reads them
#pragma unroll
        for (int j = 0; j < kPiece; ++j) {
          if constexpr (kLdl) Wp[(p & 1) * kPiece * kDL + row + j * kDL] = x[j];
          D[row + (kb + j) * kDL] = kLdl ? x[j] * rs[j] : x[j];
        }
      }
      if (warp == 0 && lane < kPiece) {
        double mine = 0.0;
#pragma unroll
        for (int j = 0; j < kPiece; ++j)
          if (lane == j) mine = kLdl ? x[j] : rs[j];
        if constexpr (kLdl) {
          Rinv[kb + lane] = 1.0;
          Dk[kb + lane] = mine;
          D[kb + lane + (kb + lane) * kDL] = 1.0;
        } else {
          Rinv[kb + lane] = mine;
        }
      }
      asm volatile("bar.sync 3, 256;\n" ::: "memory");
    }
    if (warp == 2) invert(kPieces - 1);
  } else {
    const int g = lane >> 2, t = lane & 3;
    const T* gsrc = gl + c0 + (int64_t)c0 * ld;
    // column tile of this warp: 1 .. 5; tiles 6 and 7 (warps 4, 5), which have rows 48 .. 63
    // only; warp 3 lays tile 0 at once
    const int n0 = warp - 2, n1 = warp == 4 ? 7 : warp == 5 ? 6 : kPieces;
    auto entry = [&](int n, int i, int e) {
      const int r = 16 * i + g + 8 * (e >> 1), c = 8 * n + 2 * t + (e & 1);
      return (r < nb && c < nb && r >= c) ? (double)gsrc[r + (int64_t)c * ld] : (r == c ? 1.0 : 0.0);
    };
    double acc[4][4], last[4];  // rows 16 i .. of tile n0, rows 48 .. of tile n1
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = entry(n0, i, e);
#pragma unroll
    for (int e = 0; e < 4; ++e) last[e] = n1 < kPieces ? entry(n1, 3, e) : 0.0;
    auto lay = [&](const double (&v)[4], int n, int i) {  // rows 16 i .. of tile n, part of the next piece
#pragma unroll
      for (int e = 0; e < 4; ++e) D[16 * i + g + 8 * (e >> 1) + (8 * n + 2 * t + (e & 1)) * kDL] = v[e];
    };
    if (warp == 3) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        double v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = entry(0, i, e);
        lay(v, 0, i);
      }
      asm volatile("bar.arrive 2, 128;\n" ::: "memory");
    }
#pragma unroll 1
    for (int p = 0; p < kPieces; ++p) {
      asm volatile("bar.sync 3, 256;\n" ::: "memory");
      const int kb = p * kPiece;
      const double* A = (kLdl ? Wp + (p & 1) * kPiece * kDL : D + kb * kDL) + g + t * kDL;
      if (n0 > p) {
        const double* B = D + 8 * n0 + g + (kb + t) * kDL;
        const double b0 = B[0], b1 = B[4 * kDL];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i >= n0 / 2) {
            const double* v = A + 16 * i;
            double h[4] = {0.0, 0.0, 0.0, 0.0};
            dmma(h, -v[4 * kDL], -v[4 * kDL + 8], b1);
            dmma(acc[i], -v[0], -v[8], b0);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] += h[e];
            if (n0 == p + 1) lay(acc[i], n0, i);
          }
        if (n0 == p + 1) asm volatile("bar.arrive 2, 128;\n" ::: "memory");
      }
      if (n1 < kPieces && n1 > p) {
        const double* B = D + 8 * n1 + g + (kb + t) * kDL;
        const double* v = A + 48;
        double h[4] = {0.0, 0.0, 0.0, 0.0};
        dmma(h, -v[4 * kDL], -v[4 * kDL + 8], B[4 * kDL]);
        dmma(last, -v[0], -v[8], B[0]);
#pragma unroll
        for (int e = 0; e < 4; ++e) last[e] += h[e];
        if (n1 == p + 1) {
          lay(last, n1, 3);
          asm volatile("bar.arrive 2, 128;\n" ::: "memory");
        }
      }
      if (warp >= 6) {  // the finished columns go out while the next piece is factored
        const int r = 32 * (warp - 6) + lane;
        double lrr = 1.0;  // Cholesky: the row's diagonal entry, from its pivot
        if (!kLdl && (r >> 3) == p) lrr = sqrt(D[r + r * kDL]);
#pragma unroll
        for (int j = 0; j < kPiece; ++j) {
          const int c = kb + j;
          if (r < c) continue;
          const double l = !kLdl && r == c ? lrr : D[r + c * kDL];
          if (r < nb && c < nb) {
            gl[(c0 + r) + (int64_t)(c0 + c) * ld] = (T)l;
            if constexpr (kLdl) a.W[m.off + (c0 + r) + (int64_t)(c0 + c) * ld] = l * Dk[c];
          }
          if (W) W[r + c * kNB] = l;
        }
        if (W && (r >> 3) == p) {
          W[kNB * kNB + r] = Rinv[r];
          if constexpr (kLdl) W[kNB * kNB + kNB + r] = 1.0 / Dk[r];
        }
      }
    }
  }
}

// TRSM of one 64-row tile below a factored diagonal block, R <- R L11^-T, by 8-column pieces.
// L11, the inverses of its 8 x 8 diagonal pieces and 1/L_kk come from the scratch slot.  Rows
// do not depend on one another, so a pair of warps takes 16 rows through the whole solve
// without a block barrier: the rows are their tensor-core accumulators (one warp the even
// 8-column tiles, the other the odd ones); a piece's 16 x 8 tile is multiplied by the piece's
// inverse (2 MMA steps) by the warp that has it, and the solved columns are applied to the
// later tiles (2 steps each) by both, through the pair's rows in shared memory.  Bound by that chain; no scalar FP64 instruction is on it, since each would
// queue behind the update tiles that share the SM in the persistent factorization (8 to 9 us
// a tile there; a thread per row substituting took 9.8 us, 12.8 us beside update tiles).
// Shared memory (doubles) of trsm_rows_task.
constexpr int kTrsmSmemDoubles = 2 * kNB * kDL + kNB;

template <class T>
__device__ __forceinline__ void trsm_rows_task(const FactorArgs& a, const PanelItem& it, const SnMeta& meta,
                                              const double* __restrict__ winv, double* sm) {
  double* R = sm;                // R[r + k*kDL]
  double* D = sm + kNB * kDL;    // D[i + j*kDL] = L11[i][j]
  double* Rinv = sm + 2 * kNB * kDL;
  const SnMeta m = meta;
  T* g = static_cast<T*>(a.L) + m.off;
  const int nb = it.nb, c0 = it.c0;
  const int64_t ld = m.ld;
  const int rows = min(kNB, m.h - it.row0);
  const double* W = winv + (size_t)it.slot * kSlot;
  const int tid = thread_id();
  const int lane = tid & 31, warp = tid >> 5, gq = lane >> 2, t = lane & 3, r0 = 16 * (warp & 3), half = warp >> 2;
  double acc[4][4];  // column tiles half, half + 2, ...
  {
    const T* src = g + it.row0 + r0 + gq + (int64_t)(c0 + 8 * half + 2 * t) * ld;
    const bool in0 = r0 + gq < rows, in1 = r0 + gq + 8 < rows;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const bool c = 16 * q + 8 * half + 2 * t + e < nb;
        acc[q][e] = in0 && c ? (double)src[e * ld] : 0.0;
        acc[q][2 + e] = in1 && c ? (double)src[e * ld + 8] : 0.0;
      }
      src += 16 * ld;
    }
    double w[kNB * kNB / kThreads];
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) w[q] = W[tid + q * kThreads];
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) D[(tid & 63) + ((tid >> 6) + 4 * q) * kDL] = w[q];
  }
  if (tid < kNB) Rinv[tid] = W[kNB * kNB + tid];
  __syncthreads();
  if (r0 < rows) {
    double* Rw = R + r0;
    const int np = (nb + kPiece - 1) / kPiece;
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
      const int kb = p * kPiece;
      double* q = Rw + gq + (kb + t) * kDL;  // fragment reads
      const bool owner = (p & 1) == half;    // acc[0] is column tile p
      if (owner) {
        double* o = Rw + gq + (kb + 2 * t) * kDL;  // accumulator places
#pragma unroll
        for (int e = 0; e < 4; ++e) o[8 * (e >> 1) + (e & 1) * kDL] = acc[0][e];
        // inverse fragments: Inv[n = gq][k = t (+ 4)], stored transposed above the diagonal
        const double* iv = D + kb + t + (kb + gq) * kDL;
        const double i0 = t < gq ? iv[0] : t == gq ? Rinv[kb + t] : 0.0;
        const double i1 = t + 4 < gq ? iv[4] : t + 4 == gq ? Rinv[kb + t + 4] : 0.0;
        __syncwarp();
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        dmma(x, q[0], q[8], i0);
        dmma(x, q[4 * kDL], q[4 * kDL + 8], i1);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 4; ++e) o[8 * (e >> 1) + (e & 1) * kDL] = x[e];
#pragma unroll
        for (int n = 1; n < 4; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[n - 1][e] = acc[n][e];
      }
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (warp & 3)) : "memory");
      const double a0 = -q[0], a1 = -q[8], a2 = -q[4 * kDL], a3 = -q[4 * kDL + 8];
      const int first = owner ? 1 : 0;  // tiles p + 1 + first, + 2, ...
      const double* b = D + gq + kb + kPiece + 8 * first + (kb + t) * kDL;
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (p + 1 + first + 2 * n < np) {
          dmma(acc[n], a0, a1, b[16 * n]);
          dmma(acc[n], a2, a3, b[16 * n + 4 * kDL]);
        }
    }
  }
  __syncthreads();
  if (a.ldl) {  // R is W's rows (R L11^-T with unit L11); L's rows are R D^-1
    const double* dinv = W + kNB * kNB + kNB;
    double* gw = a.W + m.off;
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) {
      const int idx = tid + q * kThreads, k = idx / kNB, r = idx - k * kNB;
      if (r < rows && k < nb) {
        const double v = R[r + k * kDL];
        g[(it.row0 + r) + (int64_t)(c0 + k) * ld] = (T)(v * dinv[k]);
        gw[(it.row0 + r) + (int64_t)(c0 + k) * ld] = v;
      }
    }
    async_fence();
    return;
  }
#pragma unroll
  for (int q = 0; q < kNB * kNB / kThreads; ++q) {
    const int idx = tid + q * kThreads, k = idx / kNB, r = idx - k * kNB;
    if (r < rows && k < nb) g[(it.row0 + r) + (int64_t)(c0 + k) * ld] = (T)R[r + k * kDL];
  }
  if constexpr (std::is_same<T, double>::value) {
    async_fence();
  } else {
    const int64_t off = a.split ? a.split_off[it.s] : -1;
    if (off >= 0) {  // the tile's rows, row by row (consecutive threads take consecutive columns)
#pragma unroll
      for (int q = 0; q < kNB * kNB / kThreads; ++q) {
        const int idx = tid + q * kThreads, r = idx / kNB, k = idx - r * kNB;
        if (r < rows && k < nb) split_store(a, m, off, it.row0 + r, c0 + k, (float)R[r + k * kDL]);
      }
      async_fence();
    }
  }
}


}  // namespace
}  // namespace ftask
}  // namespace dev
}  // namespace spb
