// Persistent supernodal triangular solves (sm_100a).
//
// Numerics of symPACK's solve tasks (symPACKMatrix2D.hpp):
//   FUC(J,J): Y_J <- L_JJ^-1 Y_J               (forward_update_contrib, 1519-1527)
//   FUC(K,J): Y_K[rows] -= L_KJ Y_J            (1589-1592)
//   BUC(J,I): X_I -= L_JI^T X_J[rows]           (back_update_contrib, 1741-1744)
//   BUC(I,I): X_I <- L_II^-T X_I                (_tri_solve, 1659-1721)
// The reference's FUC/BUC task graph (5167-5251, 5728-6322) becomes one
// persistent launch per sweep: CTAs take tasks from an atomic counter in a
// topological order (every dependency of a task was handed out earlier, so a
// waiting CTA only ever waits on CTAs that are already running) and
// synchronise through counters in global memory.  Every wait is bounded; on
// expiry the kernel records SPB timeout status and all CTAs leave.
//
// A supernode wider than one 64-column block is split into super-blocks of sb
// blocks.  The diagonal triangle of a super-block is applied through its
// inverse (k_sb_inverse, once per factorization), so the sb dependent block
// solves of a substitution become sb independent row-block products: the chain
// of a wide supernode has two steps per super-block (its DI products, then the
// updates of the next super-block) instead of one per 64 columns.  The diagonal
// block of a one-block supernode is applied through its inverse too
// (k_diag_inverse), in FP64 with one correction by its residual (solve_block), without which
// the residual would grow with the block's condition.  The forward sweep reads the permuted right-hand sides Y
// (accumulating the descendants' contributions there) and writes its solution
// to Z; the backward sweep accumulates into Z and writes the final solution X.
//
// Every task is a product of a stored operand with a few right-hand-side columns.
// The sweeps are bound by the chain of dependent tasks, each a few global round
// trips, so a task does everything that needs no right-hand side before it waits:
// one 64-byte record (SolveRec) says where everything is, the operand is loaded
// straight into registers in the layout of the FP64 tensor-core fragments
// (mma.sync m16n8k4: 32 entries per thread cover a 64 x 128 tile pair), and after
// the wait only the right-hand sides pass through shared memory.  The products run
// on the FP64 tensor pipe for one right-hand side too: an 8-column group costs no
// more issue slots than scalar FMAs with their shared-memory reads would.
// FP32 factors are widened as they enter a product.  60^3 Laplacian, FP64: 1 right-hand side
// 2.16 -> 1.22 ms, 16 right-hand sides 4.85 -> 2.16 ms against tasks that staged their tiles
// in shared memory and multiplied with scalar FMAs (0.34 ms by the bytes of both sweeps).
#include <type_traits>

#include "kernels.cuh"

namespace spb {
namespace dev {

namespace {

constexpr int kT = 64;         // rows / columns per tile
constexpr int kPld = 65;       // padded leading dimension of a staged 64 x 64 tile (inverse kernels)
constexpr int kThreads = 256;
// Leading dimensions (doubles) of the operands staged in shared memory: 4 mod 16, so that
// the fragment reads (8 rows or columns a leading dimension apart x 4 consecutive) of a
// half warp fall on 16 different banks.
constexpr int kInvLd = 68;     // inverse of a one-block supernode's diagonal block
constexpr int kXLd = 260;      // right-hand-side rows of one pass (at most 256)
constexpr int kZLd = 68;       // solved rows of a one-block supernode
constexpr int kRowCap = 512;   // staged row indices

// NG groups of 8 right-hand sides (1 or 2).
template <int NG>
struct SolveSmem {
  double inv[kT * kInvLd];
  double x[kXLd * 8 * NG];
  double part[8 * 16 * 8 * NG];  // G: partial sums of the 8 warps
  double z[8 * 20 * 8 * NG];     // solved rows: 64 of a block (ld kZLd) or 16 per warp (ld kWzLd)
  double ldiag[kT];              // diagonal of a one-block supernode's diagonal block
  int rows[kRowCap];
};
// Three CTAs per SM where the fragments of a pair of tiles leave room in 80 registers (FP32, one
// group); FP64 fragments spill there (60^3, 1 right-hand side: 1.22 -> 1.69 ms).
template <class T, int NG>
constexpr int solve_min_blocks() { return NG == 1 && sizeof(T) == 4 ? 3 : 2; }

__device__ __forceinline__ void report_status(Status* st, int code, int s, int col) {
  if (atomicCAS(&st->code, 0, code) == 0) {
    st->supernode = s;
    st->column = col;
  }
}

__device__ __forceinline__ int ld_acquire(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Counter increment with release semantics: after a barrier, a thread's release
// publishes the whole block's earlier writes to any thread that acquires the counter.
__device__ __forceinline__ void red_release(int32_t* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int status_code(const Status* st) { return *(volatile const int32_t*)&st->code; }

// One thread: wait until *flag >= target.  False on timeout (recorded) or if another CTA
// has already recorded a failure.
__device__ __forceinline__ bool poll_geq(const int32_t* flag, int target, Status* st, int s, long long limit) {
  if (ld_acquire(flag) >= target) return true;
  for (long long it = 0; it < limit; ++it) {
    if (it >= 256) __nanosleep(128);  // short waits poll back to back (each poll is an L2 round trip)
    if (ld_acquire(flag) >= target) return true;
    if (status_code(st) != 0) return false;
  }
  report_status(st, 3, s, target);
  return false;
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// The gathered side's rows, from a record's count of kUnit entries.
template <int kUnit>
__device__ __forceinline__ const int32_t* row_list(const PSolveArgs& a, int32_t at) {
  return a.rows + (int64_t)at * kUnit;
}

// Task timeline for analysis (of the first group of right-hand sides; trace may be null).
__device__ __forceinline__ void trace_mark(unsigned long long* trace, const SolveRec& r, int slot) {
  if (trace) trace[4 * (size_t)((unsigned)r.kind >> 3) + slot] = now_ns();
}
__device__ __forceinline__ void trace_start(unsigned long long* trace, const SolveRec& r) {
  trace_mark(trace, r, 0);
  if (trace) trace[4 * (size_t)((unsigned)r.kind >> 3) + 3] = ((unsigned long long)r.s << 8) | (unsigned)(r.kind & 7);
}

// D = A(16x4, row) * B(4x8, col) + D, FP64.  Fragment ownership (lane = 4*g + t):
//   a0 = A[g][t], a1 = A[g+8][t], b0 = B[t][g],
//   d0 = D[g][2t], d1 = D[g][2t+1], d2 = D[g+8][2t], d3 = D[g+8][2t+1].
__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// A 16 x 64 operand slab of one warp in fragment layout: element (m, k) lies at
// p[m * sm + k * sk]; rows < mv and inner indices < kv are valid, the rest is zero.
template <class T>
struct Frag {
  T a0[16], a1[16];
  __device__ __forceinline__ void load(const T* p, int64_t sm, int64_t sk, int mv, int kv) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const T* q = p + g * sm + t * sk;
    const bool v0 = g < mv, v1 = g + 8 < mv;
    const int64_t s8 = 8 * sm, s4 = 4 * sk;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const bool kk = 4 * i + t < kv;
      a0[i] = v0 && kk ? __ldg(q) : T(0);
      a1[i] = v1 && kk ? __ldg(q + s8) : T(0);
      q += s4;
    }
  }
};

// acc += A(16 x 64 slab) * B, B[k][c] = b[k + c * ldb] of NG groups of 8 columns.
template <class T, int NG>
__device__ __forceinline__ void slab_mma(double (&acc)[NG][4], const Frag<T>& f, const double* b, int ldb) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double* q = b + t + g * ldb;
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int n = 0; n < NG; ++n) dmma(acc[n], (double)f.a0[i], (double)f.a1[i], q[4 * i + n * 8 * ldb]);
}

// Rows of nc right-hand-side columns into b (ld ldb): row r < kr comes from X row
// (rows ? rows[r] : x0 + r) when r < k and is zero otherwise.  kr: 64, 128 or 256.
__device__ __forceinline__ void stage_x(double* b, int ldb, const double* X, int64_t ldx, int x0, const int* rows,
                                        int k, int kr, int nc) {
  const int r = threadIdx.x & (kr - 1);
  const int row = r < k ? (rows ? rows[r] : x0 + r) : 0;
  for (int c = threadIdx.x / kr; c < nc; c += kThreads / kr) {
    const double v = r < k ? __ldcg(X + row + c * ldx) : 0.0;
    b[r + c * ldb] = v;
  }
}

// out(row, c) += sign * acc for the tile rows below mv and columns below nc (atomic, fire
// and forget): tile row r goes to out row (rows ? rows[r] : y0 + r).
template <int NG>
__device__ __forceinline__ void scatter(double* out, int64_t ldx, int y0, const int* rows, const double (&acc)[NG][4],
                                        int mv, int nc, double sign) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = g + 8 * h;
    if (r >= mv) continue;
    double* o = out + (rows ? rows[r] : y0 + r);
#pragma unroll
    for (int n = 0; n < NG; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = n * 8 + 2 * t + e;
        if (c < nc) atomicAdd(o + c * ldx, sign * acc[n][2 * h + e]);
      }
  }
}

template <int NG>
__device__ __forceinline__ void clear(double (&acc)[NG][4]) {
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.0;
}

// FP64 factors: the product with a diagonal block's inverse is corrected once by its residual
// (z += Inv (y - L z)), which brings it to the accuracy of a substitution.  The product alone
// leaves a residual that grows with the block's condition: dense 24 x 24 blocks of condition
// 1e12, residual against |L||L^T||x|: 1.9e-16 alone, 2.0e-17 corrected, 1.2e-17 by
// substitution.  FP32 factors need none: their own rounding is 1e9 times that, and refinement
// recomputes the residual.  Costs two more products and barriers a task: 60^3 Laplacian 1.20 ->
// 1.22 ms, 16 right-hand sides 2.09 -> 2.16, 27-point 17^3 0.168 -> 0.182.
template <class T>
constexpr bool kCorrect = std::is_same<T, double>::value;

// Inverse of a one-block supernode's diagonal block L (w x w lower triangle, ld w) into
// the lower triangle of s, zero outside, up to the fragment sizes the products read.  When
// corrected, L's strict lower triangle goes to the upper one, transposed, and its diagonal to
// ldiag.
template <class T>
__device__ __forceinline__ void stage_inverse(double* s, double* ldiag, const double* inv, const T* L, int64_t ld, int w) {
  const int wr = (w + 15) & ~15, r = threadIdx.x & 63;
  if (r >= wr) return;
  for (int c0 = threadIdx.x >> 6; c0 < wr; c0 += 16) {  // four columns' loads in flight
    double v[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + 4 * q;
      const bool in = r < w && c < w && r >= c;
      v[q] = in ? __ldg(inv + r + c * w) : 0.0;
      if constexpr (kCorrect<T>) l[q] = in ? (double)__ldg(L + r + c * ld) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + 4 * q;
      if (kCorrect<T> ? r < c : c >= wr) continue;
      s[r + c * kInvLd] = v[q];
      if constexpr (kCorrect<T>) {
        if (r > c) s[c + r * kInvLd] = l[q];
        else ldiag[r] = l[q];
      }
    }
  }
}

// d + d2 += Op B for rows 16 im .. of the staged triangle, B[k][c] = b[k] of this lane's column:
// Op = Inv or L (kL), transposed with kTrans.  Entries on the other side of the diagonal belong
// to the other operand (kMask) or are zero.
template <bool kTrans, bool kL, bool kMask>
__device__ __forceinline__ void tri_mma(double (&d)[4], double (&d2)[4], const double* s, const double* ldiag,
                                        const double* b, int im, int ks) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, row = im * 16 + g;
  constexpr bool kDown = kTrans != kL;  // the inner index runs down a column of s
  const double* p = kDown ? s + t + row * kInvLd : s + row + t * kInvLd;
  constexpr int s1 = kDown ? 8 * kInvLd : 8, sk = kDown ? 4 : 4 * kInvLd;
  int i = kTrans ? 4 * im + 4 : 0;
  const int e = kTrans ? ks : min(ks, 4 * im);
  for (; i + 1 < e; i += 2) {
    dmma(d, p[i * sk], p[i * sk + s1], b[4 * i]);
    dmma(d2, p[(i + 1) * sk], p[(i + 1) * sk + s1], b[4 * i + 4]);
  }
  if (i < e) dmma(d, p[i * sk], p[i * sk + s1], b[4 * i]);
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // the 16 x 16 tile on the diagonal
    i = 4 * im + q;
    if (i >= ks) break;
    double a0 = p[i * sk], a1 = p[i * sk + s1];
    if (kMask) {
      const int k = 4 * q + t;  // against local rows g, g + 8
      if (kL) {
        const double l = ldiag[4 * i + t];
        if (k == g) a0 = l;
        if (k == g + 8) a1 = l;
      }
      if (kTrans ? k < g : k > g) a0 = 0.0;
      if (kTrans ? k < g + 8 : k > g + 8) a1 = 0.0;
    }
    if (q & 1) dmma(d2, a0, a1, b[4 * i]);
    else dmma(d, a0, a1, b[4 * i]);
  }
}

// z = L^-1 y (kTrans false) or L^-T y for the w rows of a one-block supernode, nc columns, by
// the whole block: y in shared memory (ld ldy, zero from row w on; overwritten when corrected),
// result to global (out, first row) and to zs (ld kZLd, zero from row w on).  A warp has at
// most one 16 x 8 tile.  Ends without a barrier.
template <class T, int NG, bool kTrans>
__device__ __forceinline__ void solve_block(double* out, int64_t ldx, double* zs, const double* inv,
                                            const double* ldiag, double* y, int ldy, int w, int nc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int mt = (w + 15) >> 4, ks = (w + 3) >> 2;
  static_assert(kT / 16 * NG <= kThreads / 32, "a tile per warp");
  const int im = warp / NG, in = warp % NG;
  const bool mine = warp < mt * NG && in * 8 < nc;
  const int row = im * 16 + g, col = in * 8 + 2 * t;  // accumulators: rows row, row + 8 x columns col, col + 1
  double d[4] = {0.0, 0.0, 0.0, 0.0}, d2[4] = {0.0, 0.0, 0.0, 0.0};
  if (mine) {
    tri_mma<kTrans, false, kCorrect<T>>(d, d2, inv, nullptr, y + t + (in * 8 + g) * ldy, im, ks);
#pragma unroll
    for (int e = 0; e < 4; ++e) d[e] += d2[e];
  }
  if constexpr (kCorrect<T>) {
    double r[4], r2[4] = {0.0, 0.0, 0.0, 0.0};
    if (mine) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        zs[row + 8 * (e >> 1) + (col + (e & 1)) * kZLd] = d[e];
        r[e] = -y[row + 8 * (e >> 1) + (col + (e & 1)) * ldy];
      }
    }
    __syncthreads();
    if (mine) {
      tri_mma<kTrans, true, true>(r, r2, inv, ldiag, zs + t + (in * 8 + g) * kZLd, im, ks);  // L z - y
#pragma unroll
      for (int e = 0; e < 4; ++e) y[row + 8 * (e >> 1) + (col + (e & 1)) * ldy] = -(r[e] + r2[e]);
    }
    __syncthreads();
    if (mine) {
#pragma unroll
      for (int e = 0; e < 4; ++e) r[e] = r2[e] = 0.0;
      tri_mma<kTrans, false, true>(r, r2, inv, nullptr, y + t + (in * 8 + g) * ldy, im, ks);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[e] += r[e] + r2[e];
    }
  }
  if (!mine) return;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int r = row + 8 * (e >> 1), c = col + (e & 1);
    if (r < w && c < nc) out[r + c * ldx] = d[e];
    zs[r + c * kZLd] = d[e];  // rows from w on: zero rows of the inverse
  }
}

// Forward sweep of one column of a tiny leaf supernode (w <= kTinyMaxW columns, no arrivals
// to wait for) by one thread: Z_0 <- L_00^-1 Y_0 by substitution (multiplying by the pivots'
// reciprocals), then Y[ancestor rows] -= L_u0 Z_0 with atomic additions.
template <class T>
__device__ __forceinline__ void tiny_forward(const PSolveArgs& a, const TinyRec& m, int64_t xo) {
  const T* P = static_cast<const T*>(a.L) + m.off;
  const int32_t* rl = a.rows + m.lidx;
  const int w = m.w, h = m.h;
  const int64_t ld = m.ld;
  double y[kTinyMaxW];
#pragma unroll
  for (int j = 0; j < kTinyMaxW; ++j) {
    y[j] = 0.0;
    if (j < w) {
      double t = __ldcg(a.X + m.fc + j + xo);
#pragma unroll
      for (int k = 0; k < j; ++k) t = fma(-(double)P[j + k * ld], y[k], t);
      y[j] = t * (1.0 / (double)P[j + j * ld]);
      a.Z[m.fc + j + xo] = y[j];
    }
  }
  for (int r = w; r < h; ++r) {
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < kTinyMaxW; ++j)
      if (j < w) t = fma((double)P[r + j * ld], y[j], t);
    // leaves of one warp that all hang on the same row add there once (50,000 leaves on one row,
    // 16 right-hand sides: 290 -> 92 us; grids unchanged)
    double* out = a.X + rl[r] + xo;
    const unsigned on = __activemask();
    int same = 0;
    __match_all_sync(on, (unsigned long long)out, &same);
    if (same && on == 0xffffffffu) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if ((threadIdx.x & 31) == 0) atomicAdd(out, -t);
    } else {
      atomicAdd(out, -t);
    }
  }
}

// Backward sweep of one column of a tiny leaf supernode by one thread, its parent done:
// Z_0 -= L_u0^T X[ancestor rows], then X_0 <- L_00^-T Z_0 by substitution.
template <class T>
__device__ __forceinline__ void tiny_backward(const PSolveArgs& a, const TinyRec& m, int64_t xo) {
  const T* P = static_cast<const T*>(a.L) + m.off;
  const int32_t* rl = a.rows + m.lidx;
  const int w = m.w, h = m.h;
  const int64_t ld = m.ld;
  double z[kTinyMaxW];
#pragma unroll
  for (int j = 0; j < kTinyMaxW; ++j) z[j] = j < w ? a.Z[m.fc + j + xo] : 0.0;
  for (int r = w; r < h; ++r) {
    const double xr = __ldcg(a.X + rl[r] + xo);
#pragma unroll
    for (int j = 0; j < kTinyMaxW; ++j)
      if (j < w) z[j] = fma(-(double)P[r + j * ld], xr, z[j]);
  }
#pragma unroll
  for (int j = kTinyMaxW - 1; j >= 0; --j) {
    if (j >= w) continue;
    double t = z[j];
#pragma unroll
    for (int k = j + 1; k < kTinyMaxW; ++k)
      if (k < w) t = fma(-(double)P[k + j * ld], z[k], t);
    z[j] = t * (1.0 / (double)P[j + j * ld]);
    a.X[m.fc + j + xo] = z[j];
  }
}

// Tiny leaf supernodes of one sweep, one thread per leaf and column (leaves fastest).
template <class T, bool kFwd>
__global__ void __launch_bounds__(128) k_solve_tiny(PSolveArgs a) {
  const int st = status_code(a.status);  // in flight beside the first record
  const int64_t total = (int64_t)a.ntiny * a.nrhs;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i / a.ntiny), j = (int)(i - (int64_t)c * a.ntiny);
    const TinyRec m = a.tiny[j];
    if (st != 0) return;
    unsigned long long* tr = a.trace && c == 0 && j % kTinyBatch == 0 ? a.trace + 4 * (a.tiny_task0 + j / kTinyBatch) : nullptr;
    if (tr) {
      tr[0] = tr[1] = now_ns();
      tr[3] = ((unsigned long long)m.s << 8) | 6;
    }
    if (kFwd) tiny_forward<T>(a, m, c * a.ldx);
    else tiny_backward<T>(a, m, c * a.ldx);
    if (tr) tr[2] = now_ns();
  }
}

// ---- small one-block supernodes, one per warp ---------------------------------------------
// w <= 16 columns: the inverse and four 16-row tiles of the off-diagonal part (backward: 64
// of its rows) are the warp's fragments, the right-hand sides are loaded straight into
// fragments too, and only the solved rows pass through the warp's 16 x 8 NG shared tile zs.
// No block barrier.  False when the wait gave up.
constexpr int kWzLd = 20;

template <class T>
__device__ __forceinline__ void frag_rows(Frag<T>& f, const T* A, int ld, int row0, int mrows, int w) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = row0 + (i >> 2) * 16 + g, col = 4 * (i & 3) + t;
    const T* q = A + row + (int64_t)col * ld;
    f.a0[i] = row < mrows && col < w ? __ldg(q) : T(0);
    f.a1[i] = row + 8 < mrows && col < w ? __ldg(q + 8) : T(0);
  }
}

// d += (4 fragment steps, zero from inner index w on) * zs
template <int NG>
__device__ __forceinline__ void small_mma(double (&d)[NG][4], const double (&v0)[4], const double (&v1)[4],
                                          const double* zs, int w) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (4 * i >= w) break;
#pragma unroll
    for (int n = 0; n < NG; ++n) dmma(d[n], v0[i], v1[i], zs[4 * i + t + (n * 8 + g) * kWzLd]);
  }
}

// FP64: the diagonal block's lower triangle into the warp's Ls (16 x 16, ld kWzLd), for the
// correction by the residual.
__device__ __forceinline__ void stage_small(double* Ls, const double* L, int64_t ld, int w) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = 2 * q + (lane >> 4), r = lane & 15;
    Ls[r + c * kWzLd] = r < w && c <= r ? __ldg(L + r + c * ld) : 0.0;
  }
}

// d <- d + Inv (y - L d), Inv in the fragments v0, v1, L in Ls (kTrans: both transposed), y the
// 16 x 8 NG tile ys (overwritten); zs: the warp's other tile.
template <int NG, bool kTrans>
__device__ __forceinline__ void correct_small(double (&d)[NG][4], const double (&v0)[4], const double (&v1)[4],
                                              const double* Ls, double* zs, double* ys, int w) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double r[NG][4];
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int o = g + 8 * (e >> 1) + (n * 8 + 2 * t + (e & 1)) * kWzLd;
      zs[o] = d[n][e];
      r[n][e] = -ys[o];
    }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // L d - y
    if (4 * i >= w) break;
    const int k = 4 * i + t;
    const double l0 = kTrans ? Ls[k + g * kWzLd] : Ls[g + k * kWzLd];
    const double l1 = kTrans ? Ls[k + (g + 8) * kWzLd] : Ls[g + 8 + k * kWzLd];
#pragma unroll
    for (int n = 0; n < NG; ++n) dmma(r[n], l0, l1, zs[k + (n * 8 + g) * kWzLd]);
  }
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) ys[g + 8 * (e >> 1) + (n * 8 + 2 * t + (e & 1)) * kWzLd] = -r[n][e];
  __syncwarp();
  clear<NG>(r);
  small_mma<NG>(r, v0, v1, ys, w);
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) d[n][e] += r[n][e];
}

template <class T, int NG, int kUnit>
__device__ bool warp_forward(const PSolveArgs& a, const SolveRec& r, double* zs, double* ys, double* Ls, double* X, double* Z, int32_t* sync,
                             int nc, Frag<T>& f, unsigned long long* trace) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = r.m;
  const T* A = static_cast<const T*>(a.L) + r.a + w;
  const double* inv = a.Inv1 + r.inv;
  double v0[4], v1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = 4 * i + t;
    v0[i] = g < w && k < w ? __ldg(inv + g + k * w) : 0.0;
    v1[i] = g + 8 < w && k < w ? __ldg(inv + g + 8 + k * w) : 0.0;
  }
  frag_rows<T>(f, A, r.ld, 0, r.k, w);
  if constexpr (kCorrect<T>) stage_small(Ls, A - w, r.ld, w);
  int tgt = 0, cnt = 0;  // this lane's arrival
  if (lane < r.ng) {
    const RelGroup gr = a.groups[r.g0 + lane];
    const int lo = gr.j0 - w, hi = (lane + 1 < r.ng ? a.groups[r.g0 + lane + 1].j0 - w : r.k) - 1;
    tgt = gr.t;
    cnt = (hi >> 6) - (lo >> 6) + 1;
  }
  const int32_t* rows = row_list<kUnit>(a, r.y0);
  bool ok = true;
  if (lane == 0) ok = poll_geq(sync + r.wait, a.expected[r.s], a.status, r.s, a.spin_limit);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // orders the warp's reads after lane 0's acquire
  if (!ok) return false;
  if (trace) trace_mark(trace, r, 1);
  double d[NG][4];
  clear<NG>(d);
  {
    double y[4][NG];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int n = 0; n < NG; ++n)
        y[i][n] = 4 * i + t < w && n * 8 + g < nc ? __ldcg(X + r.x0 + 4 * i + t + (n * 8 + g) * a.ldx) : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        if constexpr (kCorrect<T>) ys[4 * i + t + (n * 8 + g) * kWzLd] = y[i][n];
        dmma(d[n], v0[i], v1[i], y[i][n]);
      }
  }
  if constexpr (kCorrect<T>) {
    __syncwarp();
    correct_small<NG, false>(d, v0, v1, Ls, zs, ys, w);
  }
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = g + 8 * (e >> 1), c = n * 8 + 2 * t + (e & 1);
      zs[row + c * kWzLd] = d[n][e];
      if (row < w && c < nc) Z[r.x0 + row + c * a.ldx] = d[n][e];
    }
  __syncwarp();
  for (int row0 = 0; row0 < r.k; row0 += 64) {
    if (row0 > 0) frag_rows<T>(f, A, r.ld, row0, r.k, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (row0 + 16 * j >= r.k) break;
      const double x0[4] = {(double)f.a0[4 * j], (double)f.a0[4 * j + 1], (double)f.a0[4 * j + 2], (double)f.a0[4 * j + 3]};
      const double x1[4] = {(double)f.a1[4 * j], (double)f.a1[4 * j + 1], (double)f.a1[4 * j + 2], (double)f.a1[4 * j + 3]};
      clear<NG>(d);
      small_mma<NG>(d, x0, x1, zs, w);
      scatter<NG>(X, a.ldx, 0, rows + row0 + 16 * j, d, r.k - row0 - 16 * j, nc, -1.0);
    }
  }
  __syncwarp();
  if (lane < r.ng) red_release(sync + 2 + tgt, cnt);
  for (int q = lane + 32; q < r.ng; q += 32) {
    const RelGroup gr = a.groups[r.g0 + q];
    const int lo = gr.j0 - w, hi = (q + 1 < r.ng ? a.groups[r.g0 + q + 1].j0 - w : r.k) - 1;
    red_release(sync + 2 + gr.t, (hi >> 6) - (lo >> 6) + 1);
  }
  return true;
}

template <class T, int NG, int kUnit>
__device__ bool warp_backward(const PSolveArgs& a, const SolveRec& r, double* zs, double* ys, double* Ls, double* X,
                              const double* Z, int32_t* sync, int nc, Frag<T>& f, unsigned long long* trace) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = r.m;
  const T* A = static_cast<const T*>(a.L) + r.a + w;
  const double* inv = a.Inv1 + r.inv;
  double v0[4], v1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = 4 * i + t;
    v0[i] = g < w && k < w ? __ldg(inv + k + g * w) : 0.0;
    v1[i] = g + 8 < w && k < w ? __ldg(inv + k + (g + 8) * w) : 0.0;
  }
  f.load(A, r.ld, 1, w, min(64, r.k));
  if constexpr (kCorrect<T>) stage_small(Ls, A - w, r.ld, w);
  const int32_t* rows = row_list<kUnit>(a, r.y0);
  int idx[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) idx[i] = 4 * i + t < r.k ? rows[4 * i + t] : -1;
  bool ok = true;
  if (lane == 0 && r.wait >= 0) ok = poll_geq(sync + r.wait, r.target, a.status, r.s, a.spin_limit);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // orders the warp's reads after lane 0's acquire
  if (!ok) return false;
  if (trace) trace_mark(trace, r, 1);
  double d[NG][4];
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = g + 8 * (e >> 1), c = n * 8 + 2 * t + (e & 1);
      d[n][e] = row < w && c < nc ? -__ldcg(Z + r.x0 + row + c * a.ldx) : 0.0;  // d = L^T x - z
    }
  for (int row0 = 0; row0 < r.k; row0 += 64) {
    if (row0 > 0) {
      f.load(A + row0, r.ld, 1, w, min(64, r.k - row0));
#pragma unroll
      for (int i = 0; i < 16; ++i) idx[i] = row0 + 4 * i + t < r.k ? rows[row0 + 4 * i + t] : -1;
    }
#pragma unroll
    for (int i0 = 0; i0 < 16; i0 += 8) {
      if (row0 + 4 * i0 >= r.k) break;
      double x[8][NG];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int n = 0; n < NG; ++n)
          x[i][n] = idx[i0 + i] >= 0 && n * 8 + g < nc ? __ldcg(X + idx[i0 + i] + (n * 8 + g) * a.ldx) : 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int n = 0; n < NG; ++n) dmma(d[n], (double)f.a0[i0 + i], (double)f.a1[i0 + i], x[i][n]);
    }
  }
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) zs[g + 8 * (e >> 1) + (n * 8 + 2 * t + (e & 1)) * kWzLd] = -d[n][e];
  __syncwarp();
  clear<NG>(d);
  small_mma<NG>(d, v0, v1, zs, w);
  if constexpr (kCorrect<T>) correct_small<NG, true>(d, v0, v1, Ls, ys, zs, w);
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = g + 8 * (e >> 1), c = n * 8 + 2 * t + (e & 1);
      if (row < w && c < nc) X[r.x0 + row + c * a.ldx] = d[n][e];
    }
  __syncwarp();
  if (lane == 0) red_release(sync + r.sig, 1);
  return true;
}

// One persistent sweep.  Per task: the record, the operand's loads, the wait, then the
// staged right-hand sides and the product.  A ticket is one task for one group of kSolveGroup
// right-hand sides: the groups are independent solves with counters of their own whose
// chains run side by side, and share the operand's tiles in L2.  The next ticket is drawn
// while the last results are on their way.  kUnit: Plan::row_unit (a kernel of its own, since
// the multiplication costs the forward sweep registers: 27-point 17^3, one right-hand side, 182 ->
// 187 us).
template <class T, int NG, bool kFwd, int kUnit>
__global__ void __launch_bounds__(kThreads, solve_min_blocks<T, NG>()) k_solve(PSolveArgs a) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  SolveSmem<NG>& sm = *reinterpret_cast<SolveSmem<NG>*>(sm_raw);
  __shared__ int sh_task[2], sh_ok;  // the ticket of a turn is drawn into the other slot during the turn before
  const int tid = threadIdx.x, warp = tid >> 5;
  constexpr int NC = 8 * NG;
  const int ngrp = (a.nrhs + kSolveGroup - 1) / kSolveGroup, ntickets = a.ntasks * ngrp;
  Frag<T> f;
  if (tid == 0) sh_task[0] = status_code(a.status) != 0 ? ntickets : atomicAdd(a.counter, 1);
  __syncthreads();
  for (int turn = 0;; turn ^= 1) {
    const int ticket = sh_task[turn];
    if (ticket >= ntickets) return;
    const int tk = ticket / ngrp, grp = ticket - tk * ngrp;
    const SolveRec r = a.recs[tk];
    int32_t* sync = a.sync + grp * a.sync_stride;
    double* X = a.X + (int64_t)grp * kSolveGroup * a.ldx;
    double* Z = a.Z + (int64_t)grp * kSolveGroup * a.ldx;
    const int nc = min(kSolveGroup, a.nrhs - grp * kSolveGroup);
    const int kind = r.kind & 7;
    unsigned long long* trace = grp == 0 && tid == 0 && kind != 7 ? a.trace : nullptr;
    if (trace) trace_start(trace, r);
    const T* L = static_cast<const T*>(a.L);
    int tgt = 0, cnt = 1;  // this thread's arrival (O, F)
    if (kFwd && tid < r.ng) {
      const RelGroup gr = a.groups[r.g0 + tid];
      tgt = gr.t;
      if (kind != 2) {  // F: one arrival per 64-row tile and target, as the plan counts them
        const int lo = gr.j0 - r.m, hi = (tid + 1 < r.ng ? a.groups[r.g0 + tid + 1].j0 - r.m : r.k) - 1;
        cnt = (hi >> 6) - (lo >> 6) + 1;
      }
    }

    // ---- before the wait: the operand --------------------------------------------------
    const bool one_block = kind == 4 || kind == 0;
    int wm = warp & 3, wk = warp >> 2;  // row tile and inner half of this warp
    // F / G: shapes of the off-diagonal part
    int sh = 0, mtl = 1, ksp = 1, sc = 0;
    if (kind == 7) {
      bool ok = true;
      if (warp < r.m) {
        const SolveRec q = a.subs[r.x0 + warp];
        double* zs = sm.z + warp * kWzLd * 8 * NG;
        double* ys = sm.x + warp * kXLd * NG;           // a second tile and the diagonal block
        double* Ls = sm.inv + warp * (kT * kInvLd / 8);
        static_assert(kXLd * NG >= kWzLd * 8 * NG && kT * kInvLd / 8 >= 16 * kWzLd, "a warp's tiles");
        unsigned long long* wtrace = grp == 0 && (tid & 31) == 0 ? a.trace : nullptr;
        if (wtrace) trace_start(wtrace, q);
        if (kFwd) ok = warp_forward<T, NG, kUnit>(a, q, zs, ys, Ls, X, Z, sync, nc, f, wtrace);
        else ok = warp_backward<T, NG, kUnit>(a, q, zs, ys, Ls, X, Z, sync, nc, f, wtrace);
        if (wtrace) trace_mark(wtrace, q, 2);
      }
      if (tid == 0) sh_task[turn ^ 1] = atomicAdd(a.counter, 1);
      if (!__syncthreads_and(ok)) return;
      continue;
    } else if (one_block) {
      stage_inverse<T>(sm.inv, sm.ldiag, a.Inv1 + r.inv, L + r.a, r.ld, r.m);
      for (int i = tid; i < min(r.k, kRowCap); i += kThreads) sm.rows[i] = row_list<kUnit>(a, r.y0)[i];
      const T* A = L + r.a + r.m;  // first off-diagonal row
      if (kFwd) {
        // m-tiles of 16 off-diagonal rows dealt to the warps; a warp's 16 fragment steps hold
        // 4, 2 or 1 of them (w <= 16, 32, 64)
        sh = r.m <= 16 ? 2 : r.m <= 32 ? 3 : 4;
        sc = 128 << (4 - sh);  // rows per chunk
        const int lane = tid & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int row = ((i >> sh) * 8 + warp) * 16 + g, col = 4 * (i & ((1 << sh) - 1)) + t;
          const T* q = A + row + (int64_t)col * r.ld;
          f.a0[i] = row < r.k && col < r.m ? __ldg(q) : T(0);
          f.a1[i] = row + 8 < r.k && col < r.m ? __ldg(q + 8) : T(0);
        }
      } else {
        // 16-column tiles x splits of the off-diagonal rows over the 8 warps
        mtl = r.m <= 16 ? 1 : r.m <= 32 ? 2 : 4;
        ksp = 8 / mtl;
        sc = mtl <= 2 ? 256 : 128;
        wm = warp & (mtl - 1);
        wk = warp / mtl;
        const int rw = sc / ksp;  // rows of a warp: 32 or 64
        f.load(A + (int64_t)wm * 16 * r.ld + wk * rw, r.ld, 1, r.m - wm * 16, min(rw, r.k - wk * rw));
      }
    } else if (!kFwd && kind == 3) {  // W: one 16-column tile per warp
      wm = warp;
      wk = 0;
      for (int i = tid; i < r.k; i += kThreads) sm.rows[i] = row_list<kUnit>(a, r.x0)[i];
      f.load(L + r.a + (int64_t)warp * 16 * r.ld, r.ld, 1, r.m - warp * 16, r.k);
    } else if (!kFwd && kind == 5) {  // DI: this warp's tile of the inverse, transposed
      const int R = r.g0 + wk;
      f.load(static_cast<const T*>(a.Inv) + r.a + ((int64_t)R * (R + 1) / 2 + r.ng) * (kT * kT) + wm * 16 * kT, kT, 1,
             r.m - wm * 16, min(kT, r.k - wk * kT));
    } else if (!kFwd) {  // V
      f.load(L + r.a + (int64_t)wm * 16 * r.ld + wk * kT, r.ld, 1, r.m - wm * 16, min(kT, r.k - wk * kT));
    } else {  // DI, U, O
      if (kind == 2)
        for (int i = tid; i < r.m; i += kThreads) sm.rows[i] = row_list<kUnit>(a, r.y0)[i];
      const T* A = kind == 5 ? static_cast<const T*>(a.Inv) + r.a : L + r.a;
      f.load(A + wm * 16 + (int64_t)wk * kT * r.ld, 1, r.ld, r.m - wm * 16, min(kT, r.k - wk * kT));
    }

    // ---- the wait ----------------------------------------------------------------------
    if (tid == 0) {
      bool ok = true;
      if (kFwd && (one_block || kind == 5)) ok = poll_geq(sync + 2 + r.s, a.expected[r.s], a.status, r.s, a.spin_limit);
      if (ok && r.wait >= 0 && !(kFwd && one_block)) ok = poll_geq(sync + r.wait, r.target, a.status, r.s, a.spin_limit);
      sh_ok = ok;
    }
    __syncthreads();
    if (!sh_ok) return;
    if (trace) trace_mark(trace, r, 1);

    // ---- the product -------------------------------------------------------------------
    if (one_block) {
      const int w = r.m;
      const T* A = L + r.a + w;
      const int nch = (r.k + sc - 1) / sc;
      {
        if (kFwd) {
          // F, D: Z_0 <- L_00^-1 Y_0, then every off-diagonal row's Y[ancestor row] -= L_u0 Z_0
          stage_x(sm.x, kXLd, X, a.ldx, r.x0, nullptr, w, kT, nc);
          __syncthreads();
          solve_block<T, NG, false>(Z + r.x0, a.ldx, sm.z, sm.inv, sm.ldiag, sm.x, kXLd, w, nc);
          __syncthreads();
          const int lane = tid & 31, g = lane >> 2, t = lane & 3;
          for (int ch = 0; ch < nch; ++ch) {
            const int rb = ch * sc;
            if (ch > 0) {  // this chunk's fragments
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const int row = rb + ((i >> sh) * 8 + warp) * 16 + g, col = 4 * (i & ((1 << sh) - 1)) + t;
                const T* q = A + row + (int64_t)col * r.ld;
                f.a0[i] = row < r.k && col < w ? __ldg(q) : T(0);
                f.a1[i] = row + 8 < r.k && col < w ? __ldg(q + 8) : T(0);
              }
            }
            double acc[NG][4];
            clear<NG>(acc);
            const double* b = sm.z + t + g * kZLd;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {  // quarters of the fragment steps; a tile ends after 1, 2 or 4
              const int kb = 16 * (q4 & ((1 << (sh - 2)) - 1));
              if (kb < w) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                  for (int n = 0; n < NG; ++n)
                    dmma(acc[n], (double)f.a0[4 * q4 + i], (double)f.a1[4 * q4 + i], b[kb + 4 * i + n * 8 * kZLd]);
              }
              if (((q4 + 1) & ((1 << (sh - 2)) - 1)) == 0) {
                const int row0 = rb + ((4 * q4 >> sh) * 8 + warp) * 16;
                if (row0 < r.k) {
                  if (row0 + 16 <= kRowCap) scatter<NG>(X, a.ldx, 0, sm.rows + row0, acc, r.k - row0, nc, -1.0);
                  else scatter<NG>(X, a.ldx, 0, row_list<kUnit>(a, r.y0) + row0, acc, r.k - row0, nc, -1.0);
                }
                clear<NG>(acc);
              }
            }
          }
        } else {
          // G, B: Z_0 -= L_u0^T X[ancestor rows], then X_0 <- L_00^-T Z_0
          double zv[2 * NG];
          const int zi = tid & 63, zc = tid >> 6;
#pragma unroll
          for (int q = 0; q < 2 * NG; ++q) zv[q] = zi < w && zc + 4 * q < nc ? __ldcg(Z + r.x0 + zi + (zc + 4 * q) * a.ldx) : 0.0;
          double acc[NG][4];
          clear<NG>(acc);
          const int rw = sc / ksp;
          for (int ch = 0; ch < nch; ++ch) {
            const int rb = ch * sc, kc = min(sc, r.k - rb);
            if (ch > 0) __syncthreads();
            stage_x(sm.x, kXLd, X, a.ldx, 0, rb + sc <= kRowCap ? sm.rows + rb : row_list<kUnit>(a, r.y0) + rb, kc, sc, nc);
            if (ch > 0)
              f.load(A + (int64_t)wm * 16 * r.ld + rb + wk * rw, r.ld, 1, w - wm * 16, min(rw, kc - wk * rw));
            __syncthreads();
            if (wk * rw < kc) {
              const int lane = tid & 31, g = lane >> 2, t = lane & 3;
              const double* b = sm.x + wk * rw + t + g * kXLd;
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (i < 8 || rw > 32)
#pragma unroll
                  for (int n = 0; n < NG; ++n) dmma(acc[n], (double)f.a0[i], (double)f.a1[i], b[4 * i + n * 8 * kXLd]);
            }
          }
          {
            const int lane = tid & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
            for (int n = 0; n < NG; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e)
                sm.part[((warp * NC) + n * 8 + 2 * t + (e & 1)) * 16 + g + 8 * (e >> 1)] = acc[n][e];
          }
          __syncthreads();
#pragma unroll
          for (int q = 0; q < 2 * NG; ++q) {
            const int c = zc + 4 * q;
            if (c < nc) {
              double v = zv[q];
              if (zi < w && nch > 0)
                for (int k = 0; k < ksp; ++k) v -= sm.part[(((k * mtl + (zi >> 4)) * NC) + c) * 16 + (zi & 15)];
              sm.z[zi + c * kZLd] = v;
            }
          }
          __syncthreads();
          solve_block<T, NG, true>(X + r.x0, a.ldx, sm.x, sm.inv, sm.ldiag, sm.z, kZLd, w, nc);
        }
      }
    } else {
      // wide supernodes: one operand of up to tpt tiles, two at a time
      const bool W = !kFwd && kind == 3;
      const int nch = ((W ? r.m : r.k) + 127) / 128;
      // forward: DI reads Y into Z, U and O read Z into Y; backward: DI reads Z into X, V and W read X into Z
      const bool to_z = kFwd == (kind == 5);
      const double sign = kind == 5 ? 1.0 : -1.0;
      {
        const double* src = to_z ? X : Z;
        double* dst = to_z ? Z : X;
        double acc[NG][4];
        clear<NG>(acc);
        for (int ch = 0; ch < nch; ++ch) {
          if (ch > 0 && !W) __syncthreads();
          if (W) {
            if (ch == 0) stage_x(sm.x, kXLd, src, a.ldx, 0, sm.rows, r.k, kT, nc);
          } else {
            stage_x(sm.x, kXLd, src, a.ldx, r.x0 + ch * 128, nullptr, r.k - ch * 128, 128, nc);
          }
          if (ch > 0) {  // further tiles of the task
            const int kv = min(kT, r.k - ch * 128 - wk * kT);
            if (W) {
              f.load(L + r.a + (int64_t)(ch * 128 + warp * 16) * r.ld, r.ld, 1, r.m - ch * 128 - warp * 16, r.k);
            } else if (!kFwd && kind == 5) {
              const int R = r.g0 + 2 * ch + wk;
              f.load(static_cast<const T*>(a.Inv) + r.a + ((int64_t)R * (R + 1) / 2 + r.ng) * (kT * kT) + wm * 16 * kT,
                     kT, 1, r.m - wm * 16, kv);
            } else if (!kFwd) {
              f.load(L + r.a + (int64_t)wm * 16 * r.ld + ch * 128 + wk * kT, r.ld, 1, r.m - wm * 16, kv);
            } else {
              const T* A = kind == 5 ? static_cast<const T*>(a.Inv) + r.a : L + r.a;
              f.load(A + wm * 16 + (int64_t)(ch * 128 + wk * kT) * r.ld, 1, r.ld, r.m - wm * 16, kv);
            }
          }
          if (!W || ch == 0) __syncthreads();
          const int mv = W ? r.m - ch * 128 - wm * 16 : r.m - wm * 16;
          if (mv > 0 && (W || ch * 128 + wk * kT < r.k)) slab_mma<T, NG>(acc, f, sm.x + wk * kT, kXLd);
          if (W) {
            if (mv > 0) scatter<NG>(dst, a.ldx, r.y0 + ch * 128 + wm * 16, nullptr, acc, mv, nc, sign);
            clear<NG>(acc);
          }
        }
        const int mv = r.m - wm * 16;
        if (!W && mv > 0) {
          if (kFwd && kind == 2) scatter<NG>(dst, a.ldx, 0, sm.rows + wm * 16, acc, mv, nc, sign);
          else scatter<NG>(dst, a.ldx, r.y0 + wm * 16, nullptr, acc, mv, nc, sign);
        }
      }
    }

    // ---- next ticket, signals ------------------------------------------------------------
    if (tid == 0) {
      const int stop = status_code(a.status);
      const int nx = atomicAdd(a.counter, 1);
      sh_task[turn ^ 1] = stop != 0 ? ntickets : nx;
    }
    __syncthreads();
    if (r.sig >= 0 && tid == 0) red_release(sync + r.sig, 1);
    if (kFwd && (kind == 2 || one_block)) {
      if (tid < r.ng) red_release(sync + 2 + tgt, cnt);
      for (int g = tid + kThreads; g < r.ng; g += kThreads) {  // F with more targets than threads
        const RelGroup gr = a.groups[r.g0 + g];
        const int lo = gr.j0 - r.m, hi = (g + 1 < r.ng ? a.groups[r.g0 + g + 1].j0 - r.m : r.k) - 1;
        red_release(sync + 2 + gr.t, (hi >> 6) - (lo >> 6) + 1);
      }
    }
    if (trace) trace_mark(trace, r, 2);
  }
}

// ---- diagonal super-block inverses ---------------------------------------------------
// Super-blocks of more than kStripBlocks blocks, whose strips do not fit in shared memory.
// One CTA per (super-block p, column block j): the tiles Inv(i, j), i = j .. nb - 1, of
// Inv_p = L_pp^-1 by block substitution down column j:
//   Inv(j, j) = L_jj^-1,   Inv(i, j) = -L_ii^-1 sum_{k=j}^{i-1} L_ik Inv(k, j),
// in FP64 (the panel widened), stored in the arena's type.  The tiles of column j above
// tile i are this CTA's own earlier writes, read back through L2.
constexpr int kInvThreads = 256;
constexpr size_t kInvSmem = (size_t)3 * kT * kPld * sizeof(double);  // two CTAs per SM

// C (64 x 64, ld kPld) = A * B or += A * B (both 64 x 64, ld kPld); thread (ty, tx)
// owns C[ty + 16 ii][tx + 16 jj].
template <bool kAccumulate>
__device__ __forceinline__ void gemm64(double* C, const double* A, const double* B, double scale) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double c[4][4] = {};
  for (int k = 0; k < kT; ++k) {
    double av[4], bv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) av[i] = A[ty + 16 * i + k * kPld];
#pragma unroll
    for (int j = 0; j < 4; ++j) bv[j] = B[k + (tx + 16 * j) * kPld];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) c[i][j] = fma(av[i], bv[j], c[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double& d = C[ty + 16 * i + (tx + 16 * j) * kPld];
      d = kAccumulate ? d + scale * c[i][j] : scale * c[i][j];
    }
}

// Ti = inverse of the b x b lower triangle of Ls (both ld kPld; zero outside b x b).
// Four threads per column c: x_i = (delta_ic - sum_{k<i} L_ik x_k) / L_ii down the column.
__device__ __forceinline__ void tri_inverse64(double* Ti, const double* Ls, int b) {
  const int c = threadIdx.x >> 2, part = threadIdx.x & 3;
  for (int i = 0; i < kT; ++i) {
    double s = 0.0;
    if (i < b && c < b && i > c)
      for (int k = c + part; k < i; k += 4) s = fma(Ls[i + k * kPld], Ti[k + c * kPld], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (part == 0) {
      double x = 0.0;
      if (i < b && c < b && i >= c) x = (i == c ? 1.0 : -s) / Ls[i + i * kPld];
      Ti[i + c * kPld] = x;
    }
    __syncwarp();
  }
}

template <class T>
__global__ void __launch_bounds__(kInvThreads, 2) k_sb_inverse(const T* __restrict__ L, T* __restrict__ Inv,
                                                               const SnMeta* __restrict__ meta,
                                                               const InvItem* __restrict__ items, int sb) {
  extern __shared__ __align__(16) double smi[];
  double* Ls = smi;               // L(i, k), then L(i, i), then the output tile
  double* Ti = Ls + kT * kPld;    // Inv(k, j) while accumulating, then L(i, i)^-1
  double* Acc = Ti + kT * kPld;
  const InvItem it = items[blockIdx.x];
  const SnMeta m = meta[it.s];
  const int nblk = (m.w + kT - 1) / kT, b0 = it.p * sb, nb = min(sb, nblk - b0), j = it.j;
  const int64_t full = (int64_t)sb * (sb + 1) / 2;
  T* base = Inv + m.ioff + (int64_t)it.p * full * (kT * kT);
  const T* P = L + m.off;
  const int64_t ld = m.ld;
  auto tile_ptr = [&](int r, int q) { return base + ((int64_t)r * (r + 1) / 2 + q) * (kT * kT); };
  auto stage_L = [&](double* dst, int r0, int rb, int c0, int cb) {
    for (int idx = threadIdx.x; idx < kT * kT; idx += kInvThreads) {
      const int k = idx >> 6, r = idx & 63;
      dst[r + k * kPld] = (r < rb && k < cb) ? (double)P[r0 + r + (int64_t)(c0 + k) * ld] : 0.0;
    }
  };
  for (int i = j; i < nb; ++i) {
    const int ci = (b0 + i) * kT, bi = min(kT, m.w - ci);
    if (i > j) {  // Acc = sum_{k=j}^{i-1} L_ik Inv(k, j)
      for (int k = j; k < i; ++k) {
        const int ck = (b0 + k) * kT, bk = min(kT, m.w - ck);
        stage_L(Ls, ci, bi, ck, bk);
        const T* src = tile_ptr(k, j);
        for (int idx = threadIdx.x; idx < kT * kT; idx += kInvThreads) {
          const int kk = idx >> 6, r = idx & 63;
          Ti[r + kk * kPld] = (double)__ldcg(src + idx);
        }
        __syncthreads();
        if (k == j) gemm64<false>(Acc, Ls, Ti, 1.0);
        else gemm64<true>(Acc, Ls, Ti, 1.0);
        __syncthreads();
      }
    }
    stage_L(Ls, ci, bi, ci, bi);
    __syncthreads();
    tri_inverse64(Ti, Ls, bi);
    __syncthreads();
    const double* out = Ti;
    if (i > j) {  // Inv(i, j) = -L_ii^-1 Acc
      gemm64<false>(Ls, Ti, Acc, -1.0);
      __syncthreads();
      out = Ls;
    }
    T* dst = tile_ptr(i, j);
    for (int idx = threadIdx.x; idx < kT * kT; idx += kInvThreads) {
      const int kk = idx >> 6, r = idx & 63;
      dst[idx] = (T)out[r + kk * kPld];
    }
    __syncthreads();
  }
}

// ---- super-blocks of at most kStripBlocks blocks: strips of 16 columns ------------------
// A CTA takes 16 columns of column block j of Inv_p and carries them, transposed (16 rows),
// through the block rows i = j .. nb - 1 in shared memory:
//   R_i = (E_i - sum_{k=j}^{i-1} R_k L_ik^T) L_ii^-T.
// The sums run on the FP64 tensor pipe, warp v taking rows 8v .. of block i, its fragments of
// L_ik loaded straight from the panel one tile ahead; the triangular solve is one warp's, by
// 8-column pieces as the panel TRSM's.  Bound by that chain, 28 tile products and 8 solves for
// the first column of a full super-block; four strips share a column block so that a product
// takes a quarter of the time, and all CTAs of a launch are independent.  The one-CTA-per-
// column kernel above (products with scalar FMAs, every tile re-read through L2, a 64-step
// inverse per tile) took 0.58 ms on the 60^3 Laplacian and about 0.45 ms on any matrix with
// one full super-block.
constexpr int kStripBlocks = 16;
constexpr int kXs = 16;  // X[k][m] at k * 16 + (m ^ 4 (k & 3)): conflict-free fragment reads
__host__ __device__ constexpr size_t strip_smem(int nb) {
  return ((size_t)nb * kT * kXs + kT * 68 + kT) * sizeof(double);
}
__device__ __forceinline__ int xs(int k, int m) { return k * kXs + (m ^ (4 * (k & 3))); }

// One warp: R <- R D^-T for a strip R of 16 rows x 64 (element (m, k) at xs(k, m)), D lower
// triangular with leading dimension ld and reciprocal diagonal Rinv, by 8-column pieces.
__device__ __forceinline__ void strip_solve(double* R, const double* D, const double* Rinv, int kLd) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double v[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) v[n][e] = R[xs(8 * n + 2 * t + (e & 1), g + 8 * (e >> 1))];
  const int mm = lane & 15;
#pragma unroll 1
  for (int p = 0; p < 8; ++p) {  // v[n] holds column tile p + n
    const int kb = 8 * p;
    if (p > 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) R[xs(kb + 2 * t + (e & 1), g + 8 * (e >> 1))] = v[0][e];
      __syncwarp();
    }
    double x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = R[xs(kb + q, mm)];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      x[q] *= Rinv[kb + q];
#pragma unroll
      for (int k = q + 1; k < 8; ++k) x[k] = fma(-x[q], D[kb + k + (kb + q) * kLd], x[k]);
      if (q & 1) asm volatile("" ::: "memory");
    }
    __syncwarp();
    if (lane < 16) {
#pragma unroll
      for (int q = 0; q < 8; ++q) R[xs(kb + q, mm)] = x[q];
    }
    __syncwarp();
    const double a0 = -R[xs(kb + t, g)], a1 = -R[xs(kb + t, g + 8)];
    const double a2 = -R[xs(kb + 4 + t, g)], a3 = -R[xs(kb + 4 + t, g + 8)];
    const double* b = D + g + kb + 8 + (kb + t) * kLd;
#pragma unroll
    for (int n = 1; n < 8; ++n) {
      if (p + n < 8) {
        dmma(v[n], a0, a1, b[8 * (n - 1)]);
        dmma(v[n], a2, a3, b[8 * (n - 1) + 4 * kLd]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[n - 1][e] = v[n][e];
    }
  }
}

template <class T>
__global__ void __launch_bounds__(256, 2) k_sb_inverse_strips(const T* __restrict__ L, T* __restrict__ Inv,
                                                              const SnMeta* __restrict__ meta,
                                                              const InvItem* __restrict__ items, int sb) {
  constexpr int kLd = 68;
  extern __shared__ __align__(16) double smx[];
  const InvItem it = items[blockIdx.x >> 2];
  const int col0 = (blockIdx.x & 3) * 16;
  const SnMeta m = meta[it.s];
  const int nblk = (m.w + kT - 1) / kT, b0 = it.p * sb, nb = min(sb, nblk - b0), j = it.j;
  double* D = smx;
  double* Rinv = D + kT * kLd;
  double* X = Rinv + kT;
  T* base = Inv + m.ioff + (int64_t)it.p * ((int64_t)sb * (sb + 1) / 2) * (kT * kT);
  const T* P = L + m.off;
  const int64_t ld = m.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (int i = j; i < nb; ++i) {
    const int ci = (b0 + i) * kT, bi = min(kT, m.w - ci);
    // L_ii, identity beyond bi
    T dv[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = tid + q * 256, c = idx >> 6, r = idx & 63;
      dv[q] = r < bi && c <= r ? P[ci + r + (int64_t)(ci + c) * ld] : T(r == c ? 1 : 0);
    }
    const T* row = P + ci + 8 * warp + g + (int64_t)(b0 + j) * kT * ld;
    const bool ok = 8 * warp + g < bi;
    double acc[2][4] = {};
    T f[16];
    auto load = [&](int k) {
#pragma unroll
      for (int q = 0; q < 16; ++q) f[q] = ok ? row[(int64_t)((k - j) * kT + 4 * q + t) * ld] : T(0);
    };
    if (i > j) load(j);
    for (int k = j; k < i; ++k) {
      double b[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) b[q] = (double)f[q];
      if (k + 1 < i) load(k + 1);
      const int k0 = (k - j) * kT;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int kk = k0 + 4 * q + t;
        dmma(acc[q & 1], X[xs(kk, g)], X[xs(kk, g + 8)], b[q]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = 8 * warp + 2 * t + (e & 1), mm = g + 8 * (e >> 1);
      X[xs((i - j) * kT + n, mm)] = (i == j && n < bi && n == col0 + mm ? 1.0 : 0.0) - acc[0][e] - acc[1][e];
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int idx = tid + q * 256, c = idx >> 6, r = idx & 63;
      D[r + c * kLd] = (double)dv[q];
      if (r == c) Rinv[r] = 1.0 / (double)dv[q];
    }
    __syncthreads();
    if (warp == 0) {
      strip_solve(X + (i - j) * kT * kXs, D, Rinv, kLd);  // whole 4-row groups: local rows count alike in xs()
    }
    __syncthreads();
    T* dst = base + ((int64_t)i * (i + 1) / 2 + j) * (kT * kT) + col0 * kT;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + q * 256, r = idx & 63, mm = idx >> 6;
      dst[r + mm * kT] = (T)X[xs((i - j) * kT + r, mm)];
    }
  }
}

// ---- inverses of one-block supernodes' diagonal blocks ------------------------------------
// At most 32 columns: one warp per block, lane c substitutes down column c with the column in
// registers, x_i = (delta_ic - sum_{k<i} L_ik x_k) / L_ii, rows of L broadcast from shared
// memory, four sums at a time against the latency of a chain of FMAs.  (Columns in shared
// memory, two reads per FMA: 113 us on the 463 x 467 grid.)
constexpr int kDiagWarps = 4;
template <class T>
__global__ void __launch_bounds__(32 * kDiagWarps) k_diag_inverse(const T* __restrict__ L, double* __restrict__ Inv,
                                                                  const Inv1Item* __restrict__ items, int count) {
  constexpr int kW = kInv1Narrow, kLd = kW + 2;
  __shared__ __align__(16) double sh[kDiagWarps][kW * kLd];
  __shared__ double shr[kDiagWarps][kW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * kDiagWarps + warp;
  if (i0 >= count) return;
  const Inv1Item it = items[i0];
  const int w = it.w;
  double* A = sh[warp];   // row i at i * kLd
  for (int k = 0; k < w; ++k)
    if (lane < w && lane >= k) A[lane * kLd + k] = (double)L[it.a + lane + (int64_t)k * it.ld];
  if (lane < w) shr[warp][lane] = 1.0 / A[lane * kLd + lane];
  __syncwarp();
  double x[kW];
#pragma unroll
  for (int i = 0; i < kW; ++i) {
    x[i] = 0.0;
    if (i < w) {
      double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k + 1 < i; k += 2) {
        const double2 l = *reinterpret_cast<const double2*>(A + i * kLd + k);
        s[k & 2] = fma(l.x, x[k], s[k & 2]);
        s[(k & 2) + 1] = fma(l.y, x[k + 1], s[(k & 2) + 1]);
      }
      if (i & 1) s[0] = fma(A[i * kLd + i - 1], x[i - 1], s[0]);
      // x_k = 0 for k < c, so columns right of row i stay zero
      x[i] = i < lane ? 0.0 : ((i == lane ? 1.0 : 0.0) - ((s[0] + s[1]) + (s[2] + s[3]))) * shr[warp][i];
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kW; ++i)
    if (lane < w && i < w) A[i * kLd + lane] = x[i];
  __syncwarp();
  for (int k = 0; k < w; ++k)
    if (lane < w) Inv[it.inv + (int64_t)k * w + lane] = A[lane * kLd + k];
}

// Wider blocks: a warp per strip of 16 columns, solved as a strip of a super-block is.
template <class T>
__global__ void __launch_bounds__(128) k_diag_inverse_wide(const T* __restrict__ L, double* __restrict__ Inv,
                                                           const Inv1Item* __restrict__ items) {
  constexpr int kLd = 68;
  __shared__ __align__(16) double D[kT * kLd];
  __shared__ double Rinv[kT];
  extern __shared__ __align__(16) double smw[];  // a strip per warp
  const Inv1Item it = items[blockIdx.x];
  const int w = it.w, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, col0 = 16 * warp;
  for (int idx = threadIdx.x; idx < kT * kT; idx += 128) {
    const int c = idx >> 6, r = idx & 63;
    const double v = r < w && c <= r ? (double)L[it.a + r + (int64_t)c * it.ld] : (r == c ? 1.0 : 0.0);
    D[r + c * kLd] = v;
    if (r == c) Rinv[r] = 1.0 / v;
  }
  double* X = smw + warp * kT * kXs;
  for (int idx = lane; idx < kT * 16; idx += 32) {
    const int k = idx >> 4, m = idx & 15;
    X[xs(k, m)] = k < w && k == col0 + m ? 1.0 : 0.0;
  }
  __syncthreads();
  if (col0 >= w) return;
  strip_solve(X, D, Rinv, kLd);
  __syncwarp();
  for (int m = 0; m < 16 && col0 + m < w; ++m)
    for (int r = lane; r < w; r += 32) Inv[it.inv + r + (int64_t)(col0 + m) * w] = X[xs(r, m)];
}

int g_solve_grid[2][2] = {};  // resident CTAs of the sweeps: [FP32][NG - 1]

template <class T, int NG>
void init_sweeps(int fp32, int sms) {
  int per = 0;
  for (auto f : {k_solve<T, NG, true, 1>, k_solve<T, NG, false, 1>, k_solve<T, NG, true, kRowUnit>, k_solve<T, NG, false, kRowUnit>})
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SolveSmem<NG>));
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_solve<T, NG, true, 1>, kThreads, sizeof(SolveSmem<NG>));
  g_solve_grid[fp32][NG - 1] = sms * (per > 0 ? per : 1);
}

template <class T, int NG>
void run_sweep(cudaStream_t st, const PSolveArgs& a, bool forward) {
  const int64_t tickets = (int64_t)a.ntasks * ((a.nrhs + kSolveGroup - 1) / kSolveGroup);
  const int cap = g_solve_grid[std::is_same<T, float>::value][NG - 1], grid = cap < tickets ? cap : (int)tickets;
  const int64_t pairs = (int64_t)a.ntiny * a.nrhs;
  const int tiny = pairs > 148 * 16 * 128 ? 148 * 16 : (int)((pairs + 127) / 128);
  if (forward) {
    if (tiny > 0) k_solve_tiny<T, true><<<tiny, 128, 0, st>>>(a);
    if (grid > 0)
      (a.row_unit == 1 ? k_solve<T, NG, true, 1> : k_solve<T, NG, true, kRowUnit>)<<<grid, kThreads, sizeof(SolveSmem<NG>), st>>>(a);
  } else {
    if (grid > 0)
      (a.row_unit == 1 ? k_solve<T, NG, false, 1> : k_solve<T, NG, false, kRowUnit>)<<<grid, kThreads, sizeof(SolveSmem<NG>), st>>>(a);
    if (tiny > 0) k_solve_tiny<T, false><<<tiny, 128, 0, st>>>(a);
  }
}

}  // namespace

void init_solve_attributes() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  init_sweeps<double, 1>(0, sms);
  init_sweeps<double, 2>(0, sms);
  init_sweeps<float, 1>(1, sms);
  init_sweeps<float, 2>(1, sms);
  cudaFuncSetAttribute(k_diag_inverse_wide<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kT * kXs * (int)sizeof(double));
  cudaFuncSetAttribute(k_diag_inverse_wide<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kT * kXs * (int)sizeof(double));
  cudaFuncSetAttribute(k_sb_inverse_strips<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strip_smem(kStripBlocks));
  cudaFuncSetAttribute(k_sb_inverse_strips<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strip_smem(kStripBlocks));
  cudaFuncSetAttribute(k_sb_inverse<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInvSmem);
  cudaFuncSetAttribute(k_sb_inverse<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInvSmem);
}

void launch_sb_inverse(cudaStream_t st, const void* L, void* Inv, bool fp32, const SnMeta* meta,
                       const InvItem* items, int count, int sb) {
  if (count <= 0) return;
  if (sb <= kStripBlocks) {
    if (fp32)
      k_sb_inverse_strips<float><<<4 * count, 256, strip_smem(sb), st>>>(static_cast<const float*>(L),
                                                                         static_cast<float*>(Inv), meta, items, sb);
    else
      k_sb_inverse_strips<double><<<4 * count, 256, strip_smem(sb), st>>>(static_cast<const double*>(L),
                                                                          static_cast<double*>(Inv), meta, items, sb);
    return;
  }
  if (fp32)
    k_sb_inverse<float><<<count, kInvThreads, kInvSmem, st>>>(static_cast<const float*>(L), static_cast<float*>(Inv),
                                                              meta, items, sb);
  else
    k_sb_inverse<double><<<count, kInvThreads, kInvSmem, st>>>(static_cast<const double*>(L),
                                                               static_cast<double*>(Inv), meta, items, sb);
}

void launch_diag_inverse(cudaStream_t st, const void* L, double* Inv, bool fp32, const Inv1Item* items, int narrow,
                         int count) {
  auto run = [&](auto* l) {
    using T = typename std::remove_const<typename std::remove_pointer<decltype(l)>::type>::type;
    if (narrow > 0)
      k_diag_inverse<T><<<(narrow + kDiagWarps - 1) / kDiagWarps, 32 * kDiagWarps, 0, st>>>(l, Inv, items, narrow);
    if (count > narrow)
      k_diag_inverse_wide<T><<<count - narrow, 128, 4 * kT * kXs * sizeof(double), st>>>(l, Inv, items + narrow);
  };
  if (fp32) run(static_cast<const float*>(L));
  else run(static_cast<const double*>(L));
}

void launch_solve_persistent(cudaStream_t st, const PSolveArgs& a, bool forward) {
  if (a.ntasks + a.ntiny <= 0 || a.spin_limit <= 0) return;
  if (a.fp32) {
    if (a.nrhs <= 8) run_sweep<float, 1>(st, a, forward);
    else run_sweep<float, 2>(st, a, forward);
  } else {
    if (a.nrhs <= 8) run_sweep<double, 1>(st, a, forward);
    else run_sweep<double, 2>(st, a, forward);
  }
}

}  // namespace dev
}  // namespace spb
