// hqr_tilekernel.cu -- the reference's per-tile kernels (tile_kernel.h:28-230,
// bodies tile_kernel.c:19-716) with their own conventions, on the GPU.
//
// The column loops (dgeqr2, dtsqr2) run on one CTA with the panel in shared
// memory (the factorization's loop, hqr_tile_fp64.cuh, with this file's
// reflector convention); the T factors and the applications, whose columns are
// independent, spread them over the SMs.  One panel step of a tile driver
// (dgeqrt, dlarft, dlarfb, dtsqrt, dlarft, dssrfb) at order 128, block 32:
// 1.40 ms; 12.4 ms with every kernel on one CTA and its operands in global
// memory.  Host pointers are staged through a device scratch
// pool for the call (copied in, and back out for every array the function may
// write); device and managed pointers are used in place.  The calls are
// synchronous, like the reference's.  Conventions (which differ from the
// LAPACK-style factorization path):
//   * reflector (tile_kernel.c:138-218): beta = +sqrt(alpha^2 + ||x||^2),
//     y_head = alpha - beta, t = 2 / (y_head^2 + ||x||^2), v = x / y_head,
//     tau = t * y_head^2; no guard for a zero column;
//   * T lower triangular: T(i,i) = tau_i, T(i,0:i) = -tau_i (T(0:i,0:i)^T
//     (Y^T y_i)(0:i)) (tile_kernel.c:220-262), T's strict upper part read as
//     stored;
//   * application (tile_kernel.c:264-363): W = Y^T A (Y lower, its stored
//     diagonal used), W = T W, A -= Y W.
// The reference's quirks are kept and listed at each function.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "hqr_common.cuh"
#include "hqr_internal.h"
#include "hqr_tile_fp64.cuh"
#include "tile_kernel.h"

namespace hqr {
namespace tk {

// ---------------------------------------------------------------------------
// Device kernels
// ---------------------------------------------------------------------------

// The reflector of this file's kernels: beta = +sqrt(a^2 + ss), head = a -
// beta, v = x / head, tau = t head^2 with t = 2 / (head^2 + ss); no guard (x = 0
// and a > 0 divides by zero, as the reference does).  The loop works with t and
// head (in tau[c] and scal[c]) on x as it is: where x is so small that head is
// zero, v is infinite but t, and with it R and the other columns, is not.  The
// reference changes a column by (t x) d, element by element, which leaves rounding
// errors of a column that is a multiple of x; as one factor t d can be exactly
// that multiple, and the zero column left divides by zero in its own step.  Such
// factors are taken in the reference's order (the loop's update), the others
// whole: tile_step_128 1.40 ms, 1.49 with all of them in that order.
struct TileLarfg {
  static constexpr bool kSplitFactor = true;
  __device__ static bool scalars(double a, double ss, double& t, double& head, double& beta) {
    beta = sqrt(ss + a * a);
    head = a - beta;
    t = 2.0 / (head * head + ss);
    return true;
  }
  __device__ static bool moves(double) { return true; }
  __device__ static void update(double& d, double r, double t, double head, double& s, double& f) {
    d = fma(head, r, d);
    s = t * head * d;
    f = t * d;
  }
};

// Doubles of shared memory of k_panel beyond its row x col panel.
constexpr int kPanelExtra = 2 * kMaxW + kMaxW / 2 + kMaxW * kMaxW;
constexpr size_t kPanelSmem = 220 * 1024;
// k_panel's copy of a panel for its application: its row x col columns, then
// kMaxW t and kMaxW heads.
constexpr size_t kPanelCopy = kPanelSmem / 8 + 2 * kMaxW;
// The widest panel (at most kMaxW columns) of `row` rows that fits (0: none).
int panel_cols(int row) {
  const long fit = ((long)kPanelSmem / 8 - kPanelExtra) / (row > 0 ? row : 1);
  return (int)(fit > kMaxW ? kMaxW : fit);
}

// The column loop on a panel of at most kMaxW columns, one CTA.  TS:
// tile_sub_dtsqr2 on [A1 (upper col x col); A2], A2 becomes V.  !TS:
// tile_sub_dgeqr2 on A2 (row x col) alone, V also to Y (ld lda, unit
// diagonal); a square panel has no last reflector (TAU(col-1) is left as it
// is and Y(col-1, col-1) = 0).  X (or null): kPanelCopy doubles that receive the
// reflectors as [head; x] (ld row; !TS: head on the diagonal), t and head, from
// which H = I - t [head; x] [head; x]^T needs no division by head.  The loop's
// FP64 work (4 row col^2 flops on one SM) and its chain of col norms bound it.
template <bool TS>
__global__ void __launch_bounds__(kThreads) k_panel(int row, int col, double* A1, int lda1, double* A2, int lda2,
                                                    double* TAU, double* Y, double* X) {
  extern __shared__ double sm[];
  double* sA = sm;
  double* tau = sA + (size_t)row * col;
  double* scal = tau + kMaxW;
  int* wide = reinterpret_cast<int*>(scal + kMaxW);
  double* sR = scal + kMaxW + kMaxW / 2;
  for (int e = threadIdx.x; e < row * col; e += kThreads) sA[e] = A2[e % row + (size_t)(e / row) * lda2];
  if (TS)
    for (int e = threadIdx.x; e < col * col; e += kThreads)
      sR[e] = (e % col <= e / col) ? A1[e % col + (size_t)(e / col) * lda1] : 0.0;
  __syncthreads();
  const int nref = (!TS && row == col) ? col - 1 : col;
  if (TS)
    panel_qr<true, TileLarfg, false>(sR, col, sA, row, row, col, nref, tau, scal, wide, nullptr, nullptr);
  else
    panel_qr<false, TileLarfg, false>(sA, row, sA, row, row, col, nref, tau, scal, wide, nullptr, nullptr);
  if (X) {
    for (int e = threadIdx.x; e < row * col; e += kThreads) X[e] = !TS && e % row == e / row ? scal[e / row] : sA[e];
    for (int c = threadIdx.x; c < col; c += kThreads) {
      X[(size_t)row * col + c] = tau[c];
      X[(size_t)row * col + kMaxW + c] = scal[c];
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < nref; c += kThreads) {
    const double head = scal[c];
    TAU[c] = tau[c] * head * head;
    scal[c] = 1.0 / head;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < row * col; e += kThreads) {
    const int r = e % row, c = e / row;
    double v = sA[e];
    if (c < nref && (TS || r > c)) v *= scal[c];
    A2[r + (size_t)c * lda2] = v;
    if (!TS && r >= c) Y[r + (size_t)c * lda2] = c >= nref ? 0.0 : (r == c ? 1.0 : v);
  }
  if (TS)
    for (int e = threadIdx.x; e < col * col; e += kThreads)
      if (e % col <= e / col) A1[e % col + (size_t)(e / col) * lda1] = sR[e];
}

// out[c] = sum_{r < n} x[r] * (base + c*ld)[r] for c < nc: one warp per column.
__device__ void col_dots(const double* x, const double* base, int ld, int n, int nc, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < nc; c += kWarps) {
    const double* y = base + (size_t)c * ld;
    double s = 0.0;
    for (int r = lane; r < n; r += 32) s = fma(x[r], y[r], s);
    s = warp_sum(s);
    if (lane == 0) out[c] = s;
  }
}

// tile_sub_dgeqr2 (tile_kernel.c:138-218).  Quirks: no zero-norm guard; with
// row == col, TAU[col-1] is left unwritten and Y(col-1,col-1) is set to 0.
// Dynamic shared memory: col doubles.
__global__ void __launch_bounds__(kThreads) k_sub_dgeqr2(int row, int col, double* A, int lda, double* TAU,
                                                          double* Y) {
  extern __shared__ double yA[];
  __shared__ double sc[3];
  const int tid = threadIdx.x;
  int i;
  for (i = 0; i < col - 1; i++) {
    double* aii = A + i + (size_t)lda * i;
    col_dots(aii + 1, aii + 1, lda, row - i - 1, col - i, yA);
    __syncthreads();
    if (tid == 0) {
      const double a_head = aii[0], norm_1 = yA[0];
      const double norm = norm_1 + a_head * a_head;
      const double b = sqrt(norm);
      const double y_head = a_head - b;
      aii[0] = y_head;
      sc[0] = b;
      sc[1] = y_head;
      sc[2] = 2.0 / (y_head * y_head + norm_1);
    }
    __syncthreads();
    const double b = sc[0], y_head = sc[1], t = sc[2];
    for (int c = tid; c < col - i - 1; c += kThreads) yA[1 + c] += y_head * A[i + (size_t)lda * (i + 1 + c)];
    __syncthreads();
    const int nr = row - i, nc = col - i - 1;
    for (int e = tid; e < nr * nc; e += kThreads) {
      const int r = e % nr, c = e / nr;
      A[i + r + (size_t)lda * (i + 1 + c)] += -t * aii[r] * yA[1 + c];
    }
    __syncthreads();
    const double inv = 1.0 / y_head;
    for (int r = tid; r < row - i - 1; r += kThreads) {
      const double v = aii[1 + r] * inv;
      aii[1 + r] = v;
      Y[i + (size_t)lda * i + 1 + r] = v;
    }
    if (tid == 0) {
      aii[0] = b;
      Y[i + (size_t)lda * i] = 1.0;
      TAU[i] = t * y_head * y_head;
    }
    __syncthreads();
  }
  if (col <= 0) return;
  i = col - 1;
  if (row > col) {
    double* aii = A + i + (size_t)lda * i;
    col_dots(aii + 1, aii + 1, lda, row - i - 1, 1, yA);
    __syncthreads();
    if (tid == 0) {
      const double a_head = aii[0], norm_1 = yA[0];
      const double norm = norm_1 + a_head * a_head;
      const double b = sqrt(norm);
      const double y_head = a_head - b;
      aii[0] = b;
      sc[1] = y_head;
      sc[2] = 2.0 / (y_head * y_head + norm_1);
    }
    __syncthreads();
    const double y_head = sc[1], t = sc[2];
    const double inv = 1.0 / y_head;
    for (int r = tid; r < row - i - 1; r += kThreads) {
      const double v = aii[1 + r] * inv;
      aii[1 + r] = v;
      Y[i + (size_t)lda * i + 1 + r] = v;
    }
    if (tid == 0) {
      Y[i + (size_t)lda * i] = 1.0;
      TAU[i] = t * y_head * y_head;
    }
  } else if (row == col && tid == 0) {
    Y[i + (size_t)lda * i] = 0.0;
  }
}

// tile_sub_dtsqr2 (tile_kernel.c:654-716): QR of [A1 (upper col x col); A2
// (row x col)], A2 becomes V.  Dynamic shared memory: col doubles.
__global__ void __launch_bounds__(kThreads) k_sub_dtsqr2(int row, int col, double* A1, int lda1, double* A2,
                                                          int lda2, double* TAU) {
  extern __shared__ double dv[];
  __shared__ double sc[3];
  const int tid = threadIdx.x;
  int i;
  for (i = 0; i < col - 1; i++) {
    double* v = A2 + (size_t)i * lda2;
    col_dots(v, v, lda2, row, col - i, dv);
    __syncthreads();
    if (tid == 0) {
      const double a_head = A1[i + (size_t)i * lda1], norm_1 = dv[0];
      const double norm = norm_1 + a_head * a_head;
      const double b = sqrt(norm);
      const double y_head = a_head - b;
      sc[0] = b;
      sc[1] = y_head;
      sc[2] = 2.0 / (y_head * y_head + norm_1);
    }
    __syncthreads();
    const double b = sc[0], y_head = sc[1], t = sc[2];
    for (int c = tid; c < col - i - 1; c += kThreads) {
      double* a1 = A1 + i + (size_t)(i + 1 + c) * lda1;
      const double d = dv[1 + c] + y_head * a1[0];
      dv[1 + c] = d;
      a1[0] += -t * y_head * d;
    }
    __syncthreads();
    const int nc = col - i - 1;
    for (int e = tid; e < row * nc; e += kThreads) {
      const int r = e % row, c = e / row;
      A2[r + (size_t)(i + 1 + c) * lda2] += -t * v[r] * dv[1 + c];
    }
    __syncthreads();
    const double inv = 1.0 / y_head;
    for (int r = tid; r < row; r += kThreads) v[r] *= inv;
    if (tid == 0) {
      A1[i + (size_t)i * lda1] = b;
      TAU[i] = t * y_head * y_head;
    }
    __syncthreads();
  }
  if (col <= 0) return;
  i = col - 1;
  double* v = A2 + (size_t)i * lda2;
  col_dots(v, v, lda2, row, 1, dv);
  __syncthreads();
  if (tid == 0) {
    const double a_head = A1[i + (size_t)i * lda1], norm_1 = dv[0];
    const double norm = norm_1 + a_head * a_head;
    const double b = sqrt(norm);
    const double y_head = a_head - b;
    A1[i + (size_t)i * lda1] = b;
    sc[1] = y_head;
    sc[2] = 2.0 / (y_head * y_head + norm_1);
  }
  __syncthreads();
  const double y_head = sc[1], t = sc[2];
  const double inv = 1.0 / y_head;
  for (int r = tid; r < row; r += kThreads) v[r] *= inv;
  if (tid == 0) TAU[i] = t * y_head * y_head;
}

// G(i, c) = Y(:, i)^T Y(:, c), c < i, to G[i col + c]: block i, four columns c
// of a warp at a time.  lower: Y is unit lower (what is stored above its
// diagonal is not read).
__global__ void __launch_bounds__(kThreads) k_gram(int row, int col, const double* __restrict__ Y, int lda,
                                                   double* __restrict__ G, int lower) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x;
  const double* yi = Y + (size_t)i * lda;
  for (int c0 = 4 * warp; c0 < i; c0 += 4 * kWarps) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r = (lower ? i : 0) + lane; r < row; r += 32) {
      const double x = yi[r];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (c0 + q < i) s[q] = fma(x, Y[r + (size_t)(c0 + q) * lda], s[q]);
    }
    warp_sums_fixed(s);
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (c0 + q < i && lane == q) G[(size_t)i * col + c0 + q] = s[q];
  }
}

// tile_sub_dlarft (tile_kernel.c:220-262): lower T (ld ldt) from G and TAU:
// T(i, r) = -tau_i sum_{c < i} T(c, r) G(i, c) for r < i.  Column r depends on
// its own elements only: one warp per column, its elements t in shared memory
// (col doubles a warp), four rows i at a time: the dots with the t known
// before them together, then the four in turn.  zero_upper: T's strict upper
// part counts as zero instead of as stored; transposed: T(i, r) is stored at
// (r, i).
__global__ void __launch_bounds__(kThreads) k_larft_cols(int col, const double* __restrict__ G,
                                                         const double* __restrict__ TAU, double* T, int ldt,
                                                         int zero_upper, int transposed) {
  extern __shared__ double sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * (blockDim.x >> 5) + warp;
  if (r >= col) return;
  double* t = sm + (size_t)warp * col;
  for (int c = lane; c < col; c += 32)
    t[c] = c == r ? TAU[r] : (c < r && !zero_upper ? T[c + (size_t)r * ldt] : 0.0);
  __syncwarp();
  for (int i0 = (r + 1) & ~3; i0 < col; i0 += 4) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c = lane; c < i0; c += 32) {
      const double tc = t[c];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (i0 + q < col) s[q] = fma(tc, G[(size_t)(i0 + q) * col + c], s[q]);
    }
    warp_sums_fixed(s);
    double v[4];   // t(i0 + q)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = i0 + q;
      if (i >= col) break;
#pragma unroll
      for (int p = 0; p < q; p++) s[q] = fma(v[p], G[(size_t)i * col + i0 + p], s[q]);
      v[q] = i > r ? -TAU[i] * s[q] : t[i];
      if (i > r && lane == 0) t[i] = v[q];
    }
    __syncwarp();
  }
  for (int c = r + lane; c < col; c += 32) T[transposed ? r + (size_t)c * ldt : c + (size_t)r * ldt] = t[c];
}

// tile_dlarft (tile_kernel.c:368-437) with 2 <= block < col: couples the
// existing diagonal blocks, reading T and Y row-major as the reference does
// (Trm(a,b) = T[a*ldt + b]).  G: col x ldg scratch, T1: col x block scratch.
__global__ void __launch_bounds__(kThreads) k_dlarft_block(int row, int col, int block, const double* Y,
                                                            int lda, double* T, int ldt, double* G, int ldg,
                                                            double* T1) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int p = warp; p < col * col; p += kWarps) {
    const int a = p / col, b = p % col;
    const double* ya = Y + (size_t)a * lda;
    const double* yb = Y + (size_t)b * lda;
    double s = 0.0;
    for (int r = lane; r < row; r += 32) s = fma(ya[r], yb[r], s);
    s = warp_sum(s);
    if (lane == 0) G[(size_t)a * ldg + b] = s;
  }
  __syncthreads();
  for (int i = block; i < col - block; i += block) {
    for (int e = tid; e < i * block; e += kThreads) {
      const int a = e / block, b = e % block;
      double s = 0.0;
      for (int q = 0; q < i; q++) s = fma(T[(size_t)a * ldt + q], G[(size_t)q * ldg + i + b], s);
      T1[(size_t)a * block + b] = s;
    }
    __syncthreads();
    for (int e = tid; e < i * block; e += kThreads) {
      const int a = e / block, b = e % block;
      double s = 0.0;
      for (int q = 0; q < block; q++) s = fma(T1[(size_t)a * block + q], T[(size_t)(i + q) * ldt + i + b], s);
      T[(size_t)a * ldt + i + b] = -s;
    }
    __syncthreads();
  }
  for (int i = (col / block) * block; i < col; i++) {
    const double alpha = -T[i + (size_t)i * ldt];
    for (int a = tid; a < i; a += kThreads) {
      double s = 0.0;
      for (int q = 0; q < i; q++) s = fma(T[(size_t)a * ldt + q], G[(size_t)q * ldg + i], s);
      T[(size_t)a * ldt + i] = alpha * s;
    }
    __syncthreads();
  }
}

// One column of W = Y^T a: out[r] = [first[r] (head[r] first[r]) +] sum_{q >=
// (lower ? r : 0)} Y(q, r) a(q), r < Y_col, by the CTA: a warp takes four r at a time.
__device__ void column_yta(int row, int Y_col, const double* Y, int ldy, const double* a, const double* first,
                           double* out, bool lower, const double* head = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r0 = 4 * warp; r0 < Y_col; r0 += 4 * kWarps) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = (lower ? r0 : 0) + lane; q < row; q += 32) {
      const double x = a[q];
#pragma unroll
      for (int p = 0; p < 4; p++)
        if (r0 + p < Y_col && (!lower || q >= r0 + p)) s[p] = fma(x, Y[q + (size_t)(r0 + p) * ldy], s[p]);
    }
    warp_sums_fixed(s);
#pragma unroll
    for (int p = 0; p < 4; p++)
      if (r0 + p < Y_col && lane == p) {
        const double top = first ? first[r0 + p] : 0.0;
        out[r0 + p] = (head ? head[r0 + p] * top : top) + s[p];
      }
  }
  __syncthreads();
}

// One column of a product with n terms: f(r, k) x[k] summed over k < terms(r),
// by the CTA, rows r < rows; done(r, sum).  Up to kThreads / 32 splits of the
// sum where there are few rows.  part: kThreads shared doubles.
template <class F, class N, class Done>
__device__ void column_product(int rows, N terms, F f, Done done, double* part) {
  int P = (rows + 31) & ~31;
  if (P > kThreads) P = kThreads;
  const int S = kThreads / P, r1 = threadIdx.x % P, s = threadIdx.x / P;
  for (int rb = 0; rb < rows; rb += P) {
    const int r = rb + r1;
    double v = 0.0;
    if (r < rows && s < S) {
      const int n = terms(r);
#pragma unroll 4
      for (int k = s; k < n; k += S) v = f(r, k, v);
    }
    part[threadIdx.x] = v;
    __syncthreads();
    if (s == 0 && r < rows) {
      for (int q = 1; q < S; q++) v += part[q * P + r1];
      done(r, v);
    }
    __syncthreads();
  }
}

// W = T w (T lower as stored; transT: the transpose of T's lower part).
__device__ void column_tw(int n, const double* T, int ldt, int transT, const double* w, double* out, double* part) {
  if (transT)   // T(q, r), q >= r
    column_product(n, [=](int r) { return n - r; },
                   [=](int r, int k, double v) { return fma(T[r + k + (size_t)r * ldt], w[r + k], v); },
                   [=](int r, double v) { out[r] = v; }, part);
  else
    column_product(n, [=](int r) { return r + 1; },
                   [=](int r, int k, double v) { return fma(T[r + (size_t)k * ldt], w[k], v); },
                   [=](int r, double v) { out[r] = v; }, part);
}

// tile_sub_dlarfb (tile_kernel.c:264-311): A (row x A_col) <- A - Y T' (Y^T A)
// with Y lower (row x row, stored diagonal) for the product and Y's first
// Y_col columns as stored for the update (lower: not above the diagonal); T' =
// T (lower) or, with transT, the transpose of T's lower part
// (tile_return_dlarfb, tile_kernel.c:501-601).  The columns of A are
// independent: each block takes columns blockIdx.x, + gridDim.x, ....  D, D2:
// Y_col x A_col global scratch.
__global__ void __launch_bounds__(kThreads) k_sub_dlarfb(int row, int Y_col, int A_col, const double* Y,
                                                          int ldy, const double* T, int ldt, double* A, int lda,
                                                          double* D, double* D2, int transT, int lower) {
  __shared__ double part[kThreads];
  for (int c = blockIdx.x; c < A_col; c += gridDim.x) {
    double* a = A + (size_t)c * lda;
    double* d = D + (size_t)c * Y_col;
    double* d2 = D2 + (size_t)c * Y_col;
    column_yta(row, Y_col, Y, ldy, a, nullptr, d, true);
    column_tw(Y_col, T, ldt, transT, d, d2, part);
    column_product(row, [=](int q) { return lower && q + 1 < Y_col ? q + 1 : Y_col; },
                   [=](int q, int r, double v) { return fma(Y[q + (size_t)r * ldy], d2[r], v); },
                   [=](int q, double v) { a[q] -= v; }, part);
  }
}

// tile_sub_dssrfb (tile_kernel.c:313-363) and its pieces.
//   part 0: the whole update; 1: tile_dssrfb_head (A1 update, D kept in U,
//   ld over_row); 2: tile_dssrfb_tail (A2 -= Y D from U).
// Quirk kept: rows Y_col..over_row-1 of A1 are zeroed (A1 -= its own copy).
// transT: T read transposed (tile_return_dssrfb).  head (or null, for 1): what
// Y has above A2's rows, one number a column (over_row = Y_col).  D: over_row x
// A_col, D2: Y_col x A_col global scratch.  Columns as in k_sub_dlarfb.
__global__ void __launch_bounds__(kThreads) k_sub_dssrfb(int over_row, int under_row, int Y_col, int A_col,
                                                          const double* Y, int ldy, const double* T, int ldt,
                                                          double* A1, int lda1, double* A2, int lda2, double* D,
                                                          double* D2, double* U, int part, int transT,
                                                          const double* head) {
  __shared__ double sums[kThreads];
  for (int c = blockIdx.x; c < A_col; c += gridDim.x) {
    double* a1 = A1 + (size_t)c * lda1;
    double* a2 = A2 + (size_t)c * lda2;
    const double* w = U + (size_t)c * over_row;
    if (part != 2) {
      double* d = D + (size_t)c * over_row;
      double* d2 = D2 + (size_t)c * Y_col;
      column_yta(under_row, min(Y_col, over_row), Y, ldy, a2, a1, d, false, head);
      column_tw(Y_col, T, ldt, transT, d, d2, sums);
      for (int r = threadIdx.x; r < over_row; r += kThreads) {
        const double v = r < Y_col ? d2[r] : a1[r];
        a1[r] -= head ? head[r] * v : v;
        if (part == 1) U[r + (size_t)c * over_row] = v;
      }
      if (part == 1) continue;
      __syncthreads();
      w = d2;
    }
    column_product(under_row, [=](int) { return Y_col; },
                   [=](int q, int r, double v) { return fma(Y[q + (size_t)r * ldy], w[r], v); },
                   [=](int q, double v) { a2[q] -= v; }, sums);
  }
}

// ---------------------------------------------------------------------------
// Host side: staging of host arrays, scratch, launches
// ---------------------------------------------------------------------------
std::mutex g_mu;                 // one tile call at a time (shared scratch)
double* g_scratch = nullptr;     // device scratch pool (grow-only)
size_t g_scratch_cap = 0;
cudaStream_t g_stream = nullptr;

// Elements spanned by a column-major rows x cols block with leading dimension ld.
size_t extent(int ld, int rows, int cols) {
  if (rows <= 0 || cols <= 0) return 0;
  return (size_t)(cols - 1) * (size_t)ld + (size_t)rows;
}

bool device_accessible(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();   // an unregistered host pointer: clear the error
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// The arrays of one call: device views of every argument, staged if needed.
class Call {
 public:
  explicit Call(const char* fn) : fn_(fn), lock_(g_mu) {}
  ~Call() { finish(); }
  // Register an array of n doubles; `out`: the function may write it.
  double* arg(const double* p, size_t n, bool out) {
    if (rc_ != HQR_OK || !p || n == 0) return const_cast<double*>(p);
    if (device_accessible(p)) return const_cast<double*>(p);
    if (nargs_ == kMaxArgs) {
      rc_ = HQR_ERR_INVALID;
      return nullptr;
    }
    Arg& a = args_[nargs_++];
    a.host = const_cast<double*>(p);
    a.n = n;
    a.out = out;
    a.off = used_;
    used_ += (n + 31) & ~size_t(31);
    return nullptr;   // resolved by bind()
  }
  // Scratch of n doubles (valid after bind()).
  size_t scratch(size_t n) {
    const size_t off = used_;
    used_ += (n + 31) & ~size_t(31);
    return off;
  }
  // Allocate the pool, copy the staged inputs in; returns the pool base.
  double* bind() {
    if (rc_ != HQR_OK) return nullptr;
    if (!g_stream && cudaStreamCreateWithFlags(&g_stream, cudaStreamNonBlocking) != cudaSuccess) {
      rc_ = record_cuda_error(cudaGetLastError(), fn_);
      return nullptr;
    }
    if (g_scratch_cap < used_) {
      if (g_scratch) cudaFree(g_scratch);
      g_scratch = nullptr;
      g_scratch_cap = 0;
      if (cudaMalloc(&g_scratch, used_ * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        rc_ = HQR_ERR_NOMEM;
        return nullptr;
      }
      g_scratch_cap = used_;
    }
    for (int i = 0; i < nargs_; i++) {
      const Arg& a = args_[i];
      if (cudaMemcpyAsync(g_scratch + a.off, a.host, a.n * sizeof(double), cudaMemcpyHostToDevice,
                          g_stream) != cudaSuccess) {
        rc_ = record_cuda_error(cudaGetLastError(), fn_);
        return nullptr;
      }
    }
    bound_ = true;
    return g_scratch;
  }
  // Device view of a registered array.
  double* view(const double* p, double* registered) const {
    if (registered || !p) return registered;
    for (int i = 0; i < nargs_; i++)
      if (args_[i].host == p) return g_scratch + args_[i].off;
    return nullptr;
  }
  cudaStream_t stream() const { return g_stream; }
  bool ok() const { return rc_ == HQR_OK; }
  void launched() {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess && rc_ == HQR_OK) rc_ = record_cuda_error(e, fn_);
  }

 private:
  struct Arg {
    double* host;
    size_t n, off;
    bool out;
  };
  static constexpr int kMaxArgs = 8;
  void finish() {
    if (bound_ && rc_ == HQR_OK) {
      for (int i = 0; i < nargs_; i++) {
        const Arg& a = args_[i];
        if (!a.out) continue;
        if (cudaMemcpyAsync(a.host, g_scratch + a.off, a.n * sizeof(double), cudaMemcpyDeviceToHost,
                            g_stream) != cudaSuccess) {
          rc_ = record_cuda_error(cudaGetLastError(), fn_);
          break;
        }
      }
    }
    if (bound_) {
      const cudaError_t e = cudaStreamSynchronize(g_stream);
      if (e != cudaSuccess && rc_ == HQR_OK) rc_ = record_cuda_error(e, fn_);
    }
    report_error(fn_, rc_);
  }
  const char* fn_;
  std::lock_guard<std::mutex> lock_;
  Arg args_[kMaxArgs];
  int nargs_ = 0;
  size_t used_ = 0;
  bool bound_ = false;
  int rc_ = HQR_OK;
};

// Launch helpers on device pointers (all sizes already validated).
template <class Kernel>
void opt_in(Kernel k, size_t smem) {
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
int column_blocks(int cols) { return cols < 2 * dag_sm_count() ? cols : 2 * dag_sm_count(); }

// G: col x col scratch.
void sub_dlarft(cudaStream_t s, int row, int col, const double* Y, int lda, const double* TAU, double* T, int ldt,
                double* G, bool lower = false, bool zero_upper = false, bool transposed = false) {
  k_gram<<<col, kThreads, 0, s>>>(row, col, Y, lda, G, lower ? 1 : 0);
  int warps = kWarps;   // t of a block's columns in 48 KiB where that allows it
  while (warps > 1 && (size_t)warps * col * sizeof(double) > 48 * 1024) warps /= 2;
  const size_t smem = (size_t)warps * col * sizeof(double);
  opt_in(k_larft_cols, smem);
  k_larft_cols<<<(col + warps - 1) / warps, warps * 32, smem, s>>>(col, G, TAU, T, ldt, zero_upper ? 1 : 0,
                                                                   transposed ? 1 : 0);
}
void sub_dlarfb(cudaStream_t s, int row, int Y_col, int A_col, const double* Y, int ldy, const double* T, int ldt,
                double* A, int lda, double* D, double* D2, int transT, bool lower = false) {
  k_sub_dlarfb<<<column_blocks(A_col), kThreads, 0, s>>>(row, Y_col, A_col, Y, ldy, T, ldt, A, lda, D, D2, transT,
                                                         lower ? 1 : 0);
}
void sub_dssrfb(cudaStream_t s, int over_row, int under_row, int Y_col, int A_col, const double* Y, int ldy,
                const double* T, int ldt, double* A1, int lda1, double* A2, int lda2, double* D, double* D2,
                double* U, int part, int transT, const double* head = nullptr) {
  k_sub_dssrfb<<<column_blocks(A_col), kThreads, 0, s>>>(over_row, under_row, Y_col, A_col, Y, ldy, T, ldt, A1, lda1,
                                                        A2, lda2, D, D2, U, part, transT, head);
}
// Scratch of the panels wider than one column loop: T and G of a loop's
// columns, D, D2 of their application to the rest, and their copy.
struct PanelScratch {
  double *T, *G, *D, *D2, *X;
  PanelScratch(double* base, int col) : T(base), G(T + kMaxW * kMaxW), D(G + kMaxW * kMaxW), D2(D + (size_t)kMaxW * col),
                                        X(D2 + (size_t)kMaxW * col) {}
  static size_t size(int col) { return 2 * (size_t)kMaxW * kMaxW + 2 * (size_t)kMaxW * col + kPanelCopy; }
};

// tile_sub_dgeqr2: panels of at most kMaxW columns in shared memory, each
// applied to the columns right of it; taller ones than fit go column by
// column through global memory (k_sub_dgeqr2).
void sub_dgeqr2(cudaStream_t s, int row, int col, double* A, int lda, double* TAU, double* Y, double* work) {
  const PanelScratch w(work, col);
  const int cw = panel_cols(row);
  if (cw < 1) {
    k_sub_dgeqr2<<<1, kThreads, (size_t)col * sizeof(double), s>>>(row, col, A, lda, TAU, Y);
    return;
  }
  opt_in(k_panel<false>, kPanelSmem);
  for (int j = 0; j < col; j += cw) {
    const int jb = col - j < cw ? col - j : cw, rows = row - j, rest = col - j - jb;
    double* Aj = A + j + (size_t)j * lda;
    double* Yj = Y + j + (size_t)j * lda;
    k_panel<false><<<1, kThreads, ((size_t)rows * jb + kPanelExtra) * sizeof(double), s>>>(
        rows, jb, nullptr, 0, Aj, lda, TAU + j, Yj, rest > 0 ? w.X : nullptr);
    if (rest == 0) break;
    sub_dlarft(s, rows, jb, w.X, rows, w.X + (size_t)rows * jb, w.T, kMaxW, w.G, true, true);
    sub_dlarfb(s, rows, jb, rest, w.X, rows, w.T, kMaxW, Aj + (size_t)jb * lda, lda, w.D, w.D2, 0, true);
  }
}
// tile_sub_dtsqr2, in the same way.
void sub_dtsqr2(cudaStream_t s, int row, int col, double* A1, int lda1, double* A2, int lda2, double* TAU,
                double* work) {
  const PanelScratch w(work, col);
  const int cw = panel_cols(row);
  if (cw < 1) {
    k_sub_dtsqr2<<<1, kThreads, (size_t)col * sizeof(double), s>>>(row, col, A1, lda1, A2, lda2, TAU);
    return;
  }
  opt_in(k_panel<true>, kPanelSmem);
  for (int j = 0; j < col; j += cw) {
    const int jb = col - j < cw ? col - j : cw, rest = col - j - jb;
    double* A1j = A1 + j + (size_t)j * lda1;
    double* A2j = A2 + (size_t)j * lda2;
    k_panel<true><<<1, kThreads, ((size_t)row * jb + kPanelExtra) * sizeof(double), s>>>(
        row, jb, A1j, lda1, A2j, lda2, TAU + j, nullptr, rest > 0 ? w.X : nullptr);
    if (rest == 0) break;
    const double *t = w.X + (size_t)row * jb, *head = t + kMaxW;
    sub_dlarft(s, row, jb, w.X, row, t, w.T, kMaxW, w.G, false, true);
    sub_dssrfb(s, jb, row, jb, rest, w.X, row, w.T, kMaxW, A1j + (size_t)jb * lda1, lda1, A2j + (size_t)jb * lda2,
               lda2, w.D, w.D2, nullptr, 0, 0, head);
  }
}

}  // namespace tk
}  // namespace hqr

using hqr::tk::Call;
using hqr::tk::extent;

extern "C" {

void* tile_init(char type, int tile_row, int tile_col) {
  (void)type;   // tile_kernel.c:19-25 allocates doubles whatever the type
  return calloc((size_t)tile_row * tile_col * 3, sizeof(double));
}

// tile_kernel.c:138-218.  row < col is rejected (HQR_ERR_INVALID): the
// reference's loop then walks the diagonal past the last row.
void tile_sub_dgeqr2(const int row, const int col, double* A, const int lda, double* TAU, double* Y,
                     double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  if (row < col || lda < row) {
    hqr::report_error("tile_sub_dgeqr2", HQR_ERR_INVALID);
    return;
  }
  Call call("tile_sub_dgeqr2");
  double* dA = call.arg(A, extent(lda, row, col), true);
  double* dT = call.arg(TAU, col, true);
  double* dY = call.arg(Y, extent(lda, row, col), true);
  const size_t w = call.scratch(hqr::tk::PanelScratch::size(col));
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dgeqr2(call.stream(), row, col, call.view(A, dA), lda, call.view(TAU, dT), call.view(Y, dY), base + w);
  call.launched();
}

// tile_kernel.c:654-716
void tile_sub_dtsqr2(const int row, const int col, double* A1, const int lda1, double* A2, const int lda2,
                     double* TAU, double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  Call call("tile_sub_dtsqr2");
  double* d1 = call.arg(A1, extent(lda1, col, col), true);
  double* d2 = call.arg(A2, extent(lda2, row, col), true);
  double* dt = call.arg(TAU, col, true);
  const size_t w = call.scratch(hqr::tk::PanelScratch::size(col));
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dtsqr2(call.stream(), row, col, call.view(A1, d1), lda1, call.view(A2, d2), lda2,
                      call.view(TAU, dt), base + w);
  call.launched();
}

// tile_kernel.c:220-262
void tile_sub_dlarft(const int row, const int col, const double* Y, const int lda, const double* TAU, double* T,
                     const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  Call call("tile_sub_dlarft");
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dtau = call.arg(TAU, col, false);
  double* dT = call.arg(T, extent(ldt, col, col), true);
  const size_t g = call.scratch((size_t)col * col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dlarft(call.stream(), row, col, call.view(Y, dy), lda, call.view(TAU, dtau), call.view(T, dT), ldt,
                      base + g);
  call.launched();
}

// tile_kernel.c:264-311
void tile_sub_dlarfb(const int row, const int Y_col, const int A_col, const double* Y, const int ldy,
                     const double* T, const int ldt, double* A, const int lda, double* work) {
  (void)work;
  if (row <= 0 || Y_col <= 0 || A_col <= 0) return;
  Call call("tile_sub_dlarfb");
  double* dy = call.arg(Y, extent(ldy, row, Y_col), false);
  double* dT = call.arg(T, extent(ldt, Y_col, Y_col), false);
  double* dA = call.arg(A, extent(lda, row, A_col), true);
  const size_t d = call.scratch((size_t)Y_col * A_col), d2 = call.scratch((size_t)Y_col * A_col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dlarfb(call.stream(), row, Y_col, A_col, call.view(Y, dy), ldy, call.view(T, dT), ldt,
                      call.view(A, dA), lda, base + d, base + d2, 0);
  call.launched();
}

// tile_kernel.c:313-363
void tile_sub_dssrfb(const int over_row, const int under_row, const int Y_col, const int A_col, const double* Y,
                     const int ldy, const double* T, const int ldt, double* A1, const int lda1, double* A2,
                     const int lda2, double* work) {
  (void)work;
  if (over_row <= 0 || under_row <= 0 || Y_col <= 0 || A_col <= 0) return;
  Call call("tile_sub_dssrfb");
  double* dy = call.arg(Y, extent(ldy, under_row, Y_col), false);
  double* dT = call.arg(T, extent(ldt, Y_col, Y_col), false);
  double* d1 = call.arg(A1, extent(lda1, over_row, A_col), true);
  double* d2 = call.arg(A2, extent(lda2, under_row, A_col), true);
  const size_t d = call.scratch((size_t)over_row * A_col), dd = call.scratch((size_t)Y_col * A_col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dssrfb(call.stream(), over_row, under_row, Y_col, A_col, call.view(Y, dy), ldy, call.view(T, dT),
                      ldt, call.view(A1, d1), lda1, call.view(A2, d2), lda2, base + d, base + dd, nullptr, 0, 0);
  call.launched();
}

// tile_kernel.c:28-57.  Quirk kept: only the diagonal T blocks are built.
void tile_dgeqrt(const int row, const int col, const int block, double* A, const int lda, double* TAU, double* Y,
                 double* T, const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0 || block <= 0) return;
  if (row < col || lda < row || ldt < col) {   // as tile_sub_dgeqr2
    hqr::report_error("tile_dgeqrt", HQR_ERR_INVALID);
    return;
  }
  Call call("tile_dgeqrt");
  double* dA = call.arg(A, extent(lda, row, col), true);
  double* dtau = call.arg(TAU, col, true);
  double* dY = call.arg(Y, extent(lda, row, col), true);
  double* dT = call.arg(T, extent(ldt, col, col), true);
  const size_t g = call.scratch((size_t)col * col);
  const size_t d = call.scratch((size_t)row * col), d2 = call.scratch((size_t)row * col);
  const size_t w = call.scratch(hqr::tk::PanelScratch::size(col));
  double* base = call.bind();
  if (!base) return;
  A = call.view(A, dA);
  TAU = call.view(TAU, dtau);
  Y = call.view(Y, dY);
  T = call.view(T, dT);
  cudaStream_t s = call.stream();
  int i;
  for (i = 0; i < col - block; i += block) {
    hqr::tk::sub_dgeqr2(s, row - i, block, A + i * lda + i, lda, TAU + i, Y + i * lda + i, base + w);
    hqr::tk::sub_dlarft(s, row - i, block, Y + i * lda + i, lda, TAU + i, T + i * ldt + i, ldt, base + g);
    hqr::tk::sub_dlarfb(s, row - i, block, col - i - block, Y + i * lda + i, lda, T + i * ldt + i, ldt,
                        A + (i + block) * lda + i, lda, base + d, base + d2, 0);
  }
  hqr::tk::sub_dgeqr2(s, row - i, col - i, A + i * lda + i, lda, TAU + i, Y + i * lda + i, base + w);
  hqr::tk::sub_dlarft(s, row - i, col - i, Y + i * lda + i, lda, TAU + i, T + i * ldt + i, ldt, base + g);
  call.launched();
}

// tile_kernel.c:60-104
void tile_dtsqrt(const int row, const int col, const int block, double* A1, const int lda1, double* A2,
                 const int lda2, double* TAU, double* T, const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0 || block <= 0) return;
  Call call("tile_dtsqrt");
  double* d1 = call.arg(A1, extent(lda1, col, col), true);
  double* d2 = call.arg(A2, extent(lda2, row, col), true);
  double* dtau = call.arg(TAU, col, true);
  double* dT = call.arg(T, extent(ldt, col, col), true);
  const size_t g = call.scratch((size_t)col * col);
  const size_t d = call.scratch((size_t)block * col), dd = call.scratch((size_t)block * col);
  const size_t w = call.scratch(hqr::tk::PanelScratch::size(col));
  double* base = call.bind();
  if (!base) return;
  A1 = call.view(A1, d1);
  A2 = call.view(A2, d2);
  TAU = call.view(TAU, dtau);
  T = call.view(T, dT);
  cudaStream_t s = call.stream();
  int i;
  for (i = 0; i < col - block; i += block) {
    hqr::tk::sub_dtsqr2(s, row, block, A1 + i + i * lda1, lda1, A2 + i * lda2, lda2, TAU + i, base + w);
    hqr::tk::sub_dlarft(s, row, block, A2 + i * lda2, lda2, TAU + i, T + i * ldt + i, ldt, base + g);
    hqr::tk::sub_dssrfb(s, block, row, block, col - i - block, A2 + i * lda2, lda2, T + i + i * ldt, ldt,
                        A1 + i + (i + block) * lda1, lda1, A2 + (i + block) * lda2, lda2, base + d, base + dd,
                        nullptr, 0, 0);
  }
  if (col % block > 0) {
    i = block * (col / block);
    hqr::tk::sub_dtsqr2(s, row, col % block, A1 + i + i * lda1, lda1, A2 + i * lda2, lda2, TAU + i, base + w);
    hqr::tk::sub_dlarft(s, row, col % block, A2 + i * lda2, lda2, TAU + i, T + i * ldt + i, ldt, base + g);
  } else {
    i = col - block;
    hqr::tk::sub_dtsqr2(s, row, block, A1 + i + i * lda1, lda1, A2 + i * lda2, lda2, TAU + i, base + w);
    hqr::tk::sub_dlarft(s, row, block, A2 + i * lda2, lda2, TAU + i, T + i * ldt + i, ldt, base + g);
  }
  call.launched();
}

// tile_kernel.c:106-119
void tile_dlarfb(const int row, const int col, double* A, const int lda, const double* Y, const double* T,
                 const int ldt, double* work) {
  tile_sub_dlarfb(row, col, col, Y, lda, T, ldt, A, lda, work);
}

// tile_kernel.c:121-136
void tile_dssrfb(const int row, const int col, double* A1, double* A2, const int lda, const double* Y,
                 const double* T, const int ldt, double* work) {
  tile_sub_dssrfb(row, row, col, col, Y, lda, T, ldt, A1, lda, A2, lda, work);
}

// tile_kernel.c:368-437.  block < 2: the full lower T; 2 <= block < col: the
// coupling of the existing diagonal blocks; block >= col: T untouched.
void tile_dlarft(const int row, const int col, const int block, const double* Y, const int lda, const double* TAU,
                 double* T, const int ldt, double* work) {
  if (block < 2) {
    tile_sub_dlarft(row, col, Y, lda, TAU, T, ldt, work);
    return;
  }
  if (block >= col || row <= 0) return;
  Call call("tile_dlarft");
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dT = call.arg(T, extent(ldt, col, col), true);
  const int ldg = (col / block) * block + block;
  const size_t g = call.scratch((size_t)col * ldg), t1 = call.scratch((size_t)col * block);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::k_dlarft_block<<<1, hqr::kThreads, 0, call.stream()>>>(row, col, block, call.view(Y, dy), lda,
                                                                    call.view(T, dT), ldt, base + g, ldg,
                                                                    base + t1);
  call.launched();
}

// tile_kernel.c:439-476: A1 update of tile_dssrfb, W kept in upper_mat (ld row).
void tile_dssrfb_head(const int row, const int col, double* A1, double* A2, const int lda, const double* Y,
                      const double* T, const int ldt, double* upper_mat) {
  if (row <= 0 || col <= 0) return;
  Call call("tile_dssrfb_head");
  double* d1 = call.arg(A1, extent(lda, row, col), true);
  double* d2 = call.arg(A2, extent(lda, row, col), false);
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dT = call.arg(T, extent(ldt, col, col), false);
  double* du = call.arg(upper_mat, (size_t)row * col, true);
  const size_t d = call.scratch((size_t)row * col), dd = call.scratch((size_t)col * col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dssrfb(call.stream(), row, row, col, col, call.view(Y, dy), lda, call.view(T, dT), ldt,
                      call.view(A1, d1), lda, call.view(A2, d2), lda, base + d, base + dd,
                      call.view(upper_mat, du), 1, 0);
  call.launched();
}

// tile_kernel.c:478-499: A2 -= Y W with W from tile_dssrfb_head.
void tile_dssrfb_tail(const int row, const int col, double* A2, const int lda, const double* Y, double* upper_mat) {
  if (row <= 0 || col <= 0) return;
  Call call("tile_dssrfb_tail");
  double* d2 = call.arg(A2, extent(lda, row, col), true);
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* du = call.arg(upper_mat, (size_t)row * col, false);
  if (!call.bind()) return;
  hqr::tk::sub_dssrfb(call.stream(), row, row, col, col, call.view(Y, dy), lda, nullptr, 0, nullptr, 0,
                      call.view(A2, d2), lda, nullptr, nullptr, call.view(upper_mat, du), 2, 0);
  call.launched();
}

// tile_kernel.c:501-601: tile_dlarfb with T read row-major (the transpose of
// the lower part of the column-major T).
void tile_return_dlarfb(const int row, const int col, double* A, const int lda, const double* Y, const double* T,
                        const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  Call call("tile_return_dlarfb");
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dT = call.arg(T, extent(ldt, col, col), false);
  double* dA = call.arg(A, extent(lda, row, col), true);
  const size_t d = call.scratch((size_t)col * col), d2 = call.scratch((size_t)col * col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dlarfb(call.stream(), row, col, col, call.view(Y, dy), lda, call.view(T, dT), ldt, call.view(A, dA),
                      lda, base + d, base + d2, 1);
  call.launched();
}

// tile_kernel.c:603-650: tile_dssrfb with T read row-major.
void tile_return_dssrfb(const int row, const int col, double* A1, double* A2, const int lda, const double* Y,
                        const double* T, const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  Call call("tile_return_dssrfb");
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dT = call.arg(T, extent(ldt, col, col), false);
  double* d1 = call.arg(A1, extent(lda, row, col), true);
  double* d2 = call.arg(A2, extent(lda, row, col), true);
  const size_t d = call.scratch((size_t)row * col), dd = call.scratch((size_t)col * col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dssrfb(call.stream(), row, row, col, col, call.view(Y, dy), lda, call.view(T, dT), ldt,
                      call.view(A1, d1), lda, call.view(A2, d2), lda, base + d, base + dd, nullptr, 0, 1);
  call.launched();
}

// Declared at tile_kernel.h:216 of the reference but never defined there:
// tile_sub_dlarft's T (built from a zeroed T), stored transposed in the upper
// triangle of T (ld ldt) as the tile_return_* kernels read it.
void tile_return_dlarft(const int row, const int col, const double* Y, const int lda, const double* TAU, double* T,
                        const int ldt, double* work) {
  (void)work;
  if (row <= 0 || col <= 0) return;
  Call call("tile_return_dlarft");
  double* dy = call.arg(Y, extent(lda, row, col), false);
  double* dtau = call.arg(TAU, col, false);
  double* dT = call.arg(T, extent(ldt, col, col), true);
  const size_t g = call.scratch((size_t)col * col);
  double* base = call.bind();
  if (!base) return;
  hqr::tk::sub_dlarft(call.stream(), row, col, call.view(Y, dy), lda, call.view(TAU, dtau), call.view(T, dT), ldt,
                      base + g, false, true, true);
  call.launched();
}

}  // extern "C"
