// hqr_tile_fp64.cuh -- FP64 tile kernels of the tiled Householder QR, run by
// one CTA of kThreads threads on CUDA cores.
//
// These restate, as block-cooperative CUDA, the four PLASMA CORE kernels that
// Hybrid_tile_QR calls (Hybrid_tile_QR.c:985 CORE_dgeqrt, :1135 CORE_dtsqrt,
// :1276 CORE_dormqr, :1356 CORE_dtsmqr):
//   * reflectors follow LAPACK dlarfg: beta = -sign(alpha)*||[alpha; x]||,
//     tau = 0 when x = 0, with the safe-minimum rescaling for tiny columns;
//   * the factorization and its updates run in w-column inner blocks
//     (w = min(IB, 32)); each block's w x w upper-triangular T is stored as a
//     diagonal block of the panel tile's NB x NB T (the full T, whose diagonal
//     w x w blocks are exactly the IB-blocked T of the LAPACK dgeqrt layout);
//   * a block reflector is applied as W = V^T C, W = T^T W, C -= V W.
//
// Shared memory holds the panel / the column block being updated; V and T are
// streamed from global memory (L2) in row chunks.  FP64 throughput on GB300 is
// ~1 TFLOP/s per GPU, so the kernels are FP64-issue bound and favour simple
// conflict-free shared-memory access over register blocking.
#pragma once
#include <cfloat>
#include "hqr_common.cuh"

namespace hqr {

constexpr int kMaxW = 32;      // inner block width
constexpr int kRC = 128;       // V row chunk staged per pass
constexpr int kRedSlots = 32;  // block-reduction scratch: kWarps partials, then 4 broadcasts
constexpr int kBcast = kWarps; // first broadcast slot
constexpr int kSplitItems = 256;   // at most this many (output, split) items in W = V^T C
static_assert(kWarps + 4 <= kRedSlots, "reduction scratch");

// Shape of the tile kernels for one (NB, IB) configuration.
struct TileShape {
  int NB;   // tile order
  int w;    // inner block width = min(IB, kMaxW)
  int CB;   // columns per LARFB/SSRFB column-block task
  int RC;   // V row chunk
  // columns of a strip of a panel block's own trailing update: the tile's
  // nominal column block, also where the update tasks are narrower (300 x 4
  // tiles of order 256, whole panel blocks in the first step: factorization 414
  // ms, 517 with the update tasks' 8 columns)
  int PB;
};

// Shared-memory carve-up, in doubles.  Computed identically on host and device.
struct SmemPlan {
  int off_c1, off_c2, off_vb, off_vt, off_t, off_g, off_w, off_w2, off_part, off_red, off_tau, off_scal;
  int total;
  __host__ __device__ static SmemPlan make(const TileShape& s) {
    SmemPlan p;
    const int NB = s.NB, w = s.w, CB = s.CB, PB = s.PB;
    // One region serves, one at a time: the GEQRT/TSQRT panel (NB x w), the
    // LARFB column block (NB x CB), the SSRFB pair A1|A2 (2 x NB x CB) and the
    // TSQRT trailing strip R-rows|A2 (w x PB + NB x PB).
    int region = NB * w;
    if (2 * NB * CB > region) region = 2 * NB * CB;
    if (w * PB + NB * PB > region) region = w * PB + NB * PB;
    int o = 0;
    p.off_c1 = o;
    p.off_c2 = o + NB * CB;                // SSRFB A2
    o += region;
    p.off_vb = o; o += (s.RC + 1) * w;     // V row chunk (ld RC+1)
    p.off_vt = o; o += w * w;              // unit-lower top of V / TSQRT R block
    p.off_t = o; o += w * w;               // T block
    p.off_g = o; o += w * w;               // Gram scratch of the T-block build
    p.off_w = o; o += w * (CB > PB ? CB : PB);
    p.off_w2 = o; o += w * (CB > PB ? CB : PB);
    p.off_part = o; o += 8 * kSplitItems;  // split-K partials (<= kSplitItems items x 8)
    p.off_red = o; o += kRedSlots;         // block reductions (kWarps) + broadcasts (4)
    p.off_tau = o; o += kMaxW;
    p.off_scal = o; o += kMaxW;            // factor of each panel column's stored x (v = x scal)
    p.total = o;
    return p;
  }
};

// ---------------------------------------------------------------------------
// Reflector generation (LAPACK dlarfg), block-cooperative.
// alpha: shared scalar; x: shared vector of n elements (unit stride).
// On return *alpha = beta, x is scaled to v(1:n), *tau_out = tau.
// ---------------------------------------------------------------------------
// Range constants of the panel arithmetic R (double; float for the FP32-class
// panels of HQR_PREC_FP32): the smallest normal number and the unit roundoff
// of dlarfg's safe minimum, the magnitudes whose squares stay in range (plain
// path), and the range of a sum of squares whose square root needs no
// scaling.  The panel kernels hold their tile in shared memory as R and
// convert once on the way in and out (the stored values are R's).
template <typename R> struct PanelReal;
template <> struct PanelReal<double> {
  static constexpr double kMin = DBL_MIN, kEps = DBL_EPSILON, kBig = 1e140, kTiny = 1e-140;
  static constexpr double kSsLo = 1e-290, kSsHi = 1e290;
};
template <> struct PanelReal<float> {
  static constexpr float kMin = FLT_MIN, kEps = FLT_EPSILON, kBig = 1e17f, kTiny = 1e-17f;
  static constexpr float kSsLo = 1e-34f, kSsHi = 1e34f;
};

// The scalar part of dlarfg for alpha = a, ||x|| = xnorm, ss = ||x||^2; plain:
// ss lies where its square root needs no scaling.  beta = -sign(a) ||[a; x]||,
// tau = (beta - a) / beta, scal = 1 / (a - beta) (x is scaled by scal after
// knt rescalings by 1/safmin, as LAPACK does for tiny columns).
template <typename R>
__device__ __forceinline__ void larfg_scalars(R a, R xnorm, R ss, bool plain, R& tau, R& scal, int& knt,
                                              R& beta) {
  using K = PanelReal<R>;
  tau = R(0);
  beta = a;
  scal = R(1);
  knt = 0;
  const R aa = fabs(a);
  if (xnorm != R(0) && plain && aa < K::kBig && (aa > K::kTiny || a == R(0))) {
    // dlapy2(alpha, ||x||) as sqrt(alpha^2 + ||x||^2): no overflow or
    // underflow in this range, one square root instead of two
    beta = -copysign(sqrt(fma(a, a, ss)), a);
    tau = (beta - a) / beta;
    scal = R(1) / (a - beta);
  } else if (xnorm != R(0)) {
    const R safmin = K::kMin / (K::kEps * R(0.5));
    const R rsafmn = R(1) / safmin;
    R xn = xnorm;
    beta = -copysign(hypot(a, xn), a);
    while (fabs(beta) < safmin && knt < 20) {
      knt++;
      a *= rsafmn;
      xn *= rsafmn;
      beta = -copysign(hypot(a, xn), a);
    }
    tau = (beta - a) / beta;
    scal = R(1) / (a - beta);
    for (int j = 0; j < knt; j++) beta *= safmin;
  }
}

// dlarfg on [alpha; x] by one warp (x: n contiguous shared doubles); every
// lane computes the (identical) scalars.
template <typename R>
__device__ void warp_larfg(R* alpha, R* x, int n, R* tau_out) {
  using K = PanelReal<R>;
  const int lane = threadIdx.x & 31;
  R ss = R(0);
  for (int r = lane; r < n; r += 32) {
    const R v = x[r];
    ss = fma(v, v, ss);
  }
  ss = warp_sum(ss);
  R xnorm;
  bool plain = false;
  if (ss == R(0)) {
    xnorm = R(0);
  } else if (ss >= K::kSsLo && ss <= K::kSsHi) {
    xnorm = sqrt(ss);
    plain = true;
  } else {
    R amax = R(0);
    for (int r = lane; r < n; r += 32) amax = fmax(amax, fabs(x[r]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    R s2 = R(0);
    for (int r = lane; r < n; r += 32) {
      const R v = x[r] / amax;
      s2 = fma(v, v, s2);
    }
    s2 = warp_sum(s2);
    xnorm = amax * sqrt(s2);
  }
  R tau, scal, beta;
  int knt;
  larfg_scalars(*alpha, xnorm, ss, plain, tau, scal, knt, beta);
  if (tau != R(0)) {
    const R rsafmn = R(1) / (K::kMin / (K::kEps * R(0.5)));
    for (int r = lane; r < n; r += 32) {
      R v = x[r];
      for (int j = 0; j < knt; j++) v *= rsafmn;
      x[r] = v * scal;
    }
  }
  __syncwarp();
  if (lane == 0) {
    *alpha = beta;
    *tau_out = tau;
  }
  __syncwarp();
}

// The warp that runs work item `it` of a panel column step: item 0 (the next
// column, whose reflector is on the critical path) has warp 0 to itself, the
// other items go round the remaining warps.
__device__ __forceinline__ bool panel_item_mine(int it, int warp) {
  return it == 0 ? warp == 0 : (warp != 0 && (it - 1) % (kWarps - 1) == warp - 1);
}

// Unblocked QR of the triangle-on-square panel [R; A] (R w x w, upper part
// used; A m x w dense), the per-column loop of CORE_dtsqrt, with the Gram
// matrix of the reflectors for the T build: G(b, c) = v_b . v_c, b < c (ld w).
// Column c's reflector acts on [R(c,c); A(:,c)]; A(:, c) becomes v_c.  At
// step c, the warp that applies reflector c to column c + 1 also forms
// reflector c + 1 (warp_larfg), the other warps apply reflector c to the
// remaining columns and compute G(:, c): one barrier per column.
template <typename RT = double>
__device__ void panel_qr_ts_fused(RT* R, int ldr, RT* A, int lda, int m, int w, RT* tau,
                                  RT* G) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) warp_larfg(R, A, m, tau);
  __syncthreads();
  for (int c = 0; c < w; c++) {
    const RT t = tau[c];
    const RT* ac = A + (size_t)c * lda;
    const int nupd = w - 1 - c;   // items 0..nupd-1: columns c+1..w-1; then G(b, c), b < c
    for (int it = 0; it < nupd + c; it++) {
      if (!panel_item_mine(it, warp)) continue;
      if (it < nupd) {
        const int j = c + 1 + it;
        RT* aj = A + (size_t)j * lda;
        if (t != RT(0)) {
          RT* rcj = R + c + (size_t)j * ldr;
          const RT r0 = *rcj;
          RT s = RT(0);
          for (int r = lane; r < m; r += 32) s = fma(ac[r], aj[r], s);
          s = (warp_sum(s) + r0) * t;
          if (lane == 0) *rcj = r0 - s;
          for (int r = lane; r < m; r += 32) aj[r] = fma(-s, ac[r], aj[r]);
        }
        if (it == 0) {
          __syncwarp();
          warp_larfg(R + j + (size_t)j * ldr, aj, m, tau + j);
        }
      } else {
        const int b = it - nupd;
        const RT* vb = A + (size_t)b * lda;
        RT s = RT(0);
        for (int r = lane; r < m; r += 32) s = fma(vb[r], ac[r], s);
        s = warp_sum(s);
        if (lane == 0) G[b + c * w] = s;
      }
    }
    __syncthreads();
  }
}

// Unblocked QR of a shared panel (dgeqr2 semantics, P m x w, ld ldp, m >= w)
// with the Gram matrix of the unit-lower reflectors, G(b, c) = v_b . v_c =
// P(c, b) + sum_{r > c} P(r, b) P(r, c), b < c (ld w); the same one-barrier
// column step as panel_qr_ts_fused.
template <typename RT = double>
__device__ void panel_qr_ge_fused(RT* P, int ldp, int m, int w, RT* tau, RT* G) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) warp_larfg(P, P + 1, m - 1, tau);
  __syncthreads();
  for (int c = 0; c < w; c++) {
    const RT t = tau[c];
    const RT* pc = P + (size_t)c * ldp;
    const int nupd = w - 1 - c;
    for (int it = 0; it < nupd + c; it++) {
      if (!panel_item_mine(it, warp)) continue;
      if (it < nupd) {
        const int j = c + 1 + it;
        RT* pj = P + (size_t)j * ldp;
        if (t != RT(0)) {
          const RT pcj = pj[c];
          RT s = RT(0);
          for (int r = c + 1 + lane; r < m; r += 32) s = fma(pc[r], pj[r], s);
          s = (warp_sum(s) + pcj) * t;
          if (lane == 0) pj[c] = pcj - s;
          for (int r = c + 1 + lane; r < m; r += 32) pj[r] = fma(-s, pc[r], pj[r]);
        }
        if (it == 0) {
          __syncwarp();
          warp_larfg(pj + j, pj + j + 1, m - j - 1, tau + j);
        }
      } else {
        const int b = it - nupd;
        const RT* pb = P + (size_t)b * ldp;
        RT s = RT(0);
        for (int r = c + 1 + lane; r < m; r += 32) s = fma(pb[r], pc[r], s);
        s = warp_sum(s);
        if (lane == 0) G[b + c * w] = s + pb[c];
      }
    }
    __syncthreads();
  }
}

// T (w x w upper, ld w) of a block of w reflectors (dlarft 'F','C') from tau
// and the Gram G(b, c), b < c: T(c, c) = tau_c, T(0:c, c) = -tau_c T(0:c,
// 0:c) G(0:c, c).  One warp, lane a owns row a of T: a row depends only on
// itself, so no synchronisation between the columns.
template <typename RT = double>
__device__ void t_from_gram(const RT* G, const RT* tau, RT* T, int w) {
  const int a = threadIdx.x & 31;
  if (a >= w) return;
  for (int c = 0; c < w; c++) {
    RT v;
    if (a < c) {
      RT s = RT(0);
      for (int b = a; b < c; b++) s = fma(T[a + b * w], G[b + c * w], s);
      v = (tau[c] == RT(0)) ? RT(0) : -tau[c] * s;
    } else {
      v = (a == c) ? tau[c] : RT(0);
    }
    T[a + c * w] = v;
  }
}

// T block (dlarft 'F','C') of a w-column block whose V is stored in shared
// memory.  unit: V is unit lower (rows 0..w-1 hold the unit triangle, V(c,c)
// = 1 implicit); otherwise V is dense (TS block, top part = identity).
// G (w x w scratch) receives the needed Gram entries.  T (w x w, ld w) output.
inline __device__ void build_t_block(const double* V, int ldv, int m, int w, bool unit, const double* tau,
                              double* G, double* T) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npairs = w * (w - 1) / 2;
  for (int p = warp; p < npairs; p += kWarps) {
    // decode p -> (a, c) with a < c
    int c = 1, base = 0;
    while (base + c <= p) { base += c; c++; }
    const int a = p - base;
    const double* va = V + (size_t)a * ldv;
    const double* vc = V + (size_t)c * ldv;
    double s = 0.0;
    const int r0 = unit ? c + 1 : 0;
    for (int r = r0 + lane; r < m; r += 32) s = fma(va[r], vc[r], s);
    s = warp_sum(s);
    if (lane == 0) G[a + c * w] = unit ? s + va[c] : s;
  }
  __syncthreads();
  for (int c = 0; c < w; c++) {
    const double tc = tau[c];
    const int a = threadIdx.x;
    if (a < c) {
      double s = 0.0;
      for (int b = a; b < c; b++) s = fma(T[a + b * w], G[b + c * w], s);
      T[a + c * w] = (tc == 0.0) ? 0.0 : -tc * s;
    } else if (a == c) {
      T[c + c * w] = tc;
    } else if (a < w) {
      T[a + c * w] = 0.0;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// The FP64 panel column loop.  On this part an FP64 warp instruction holds its
// SM sub-partition's FP64 pipe for about 65 cycles and returns after 60 (55
// for an addition), a correctly rounded sqrt or division takes about 600, and
// a shuffle sum of a warp 530: the loop is a chain of such latencies, and the
// pipe of each sub-partition is busy with the other columns meanwhile.  So:
//  * warp sums are taken in integers (warp_sums_fixed): no FP64 instruction;
//  * the reflector's scalars come from Newton steps on FP32 seeds;
//  * the dots with a column start before its scalars are known: x stays
//    unscaled (v = x scal, applied when the panel is stored);
//  * warp 0 computes the scalars alone, in a sub-partition that only the T
//    recurrence (warp 4) shares; six worker warps do the columns.
// Measured: a TSQRT block of NB 128, w 16 in the 32768 x 2048 split
// factorization takes 126 us, 176 us with the loop it replaces (each column's
// update, norm and scalars in turn on one warp, FP64 shuffle sums).
// ---------------------------------------------------------------------------

// N sums over the warp, one double per lane each, every lane gets them: each
// value as an integer multiple of 2^-57 of its sum's largest binade (rounded
// to nearest, so off by less than the first rounding of an FP64 addition of
// the two largest), summed exactly by three integer warp reductions of 22, 22
// and 14 bits, and rounded once to nearest.  Sums whose largest exponent
// leaves no room for this (near the ends of the range; infinities and NaN)
// take the FP64 shuffle sum.
template <int N>
__device__ __forceinline__ void warp_sums_fixed(double (&v)[N]) {
  const unsigned full = 0xffffffffu;
  unsigned hi[N], lo[N];
  int E[N];
  bool fits = true;
#pragma unroll
  for (int q = 0; q < N; q++) {
    hi[q] = (unsigned)__double2hiint(v[q]);
    lo[q] = (unsigned)__double2loint(v[q]);
    const unsigned top = __reduce_max_sync(full, (hi[q] & 0x7fffffffu) | (lo[q] != 0u ? 1u : 0u));
    E[q] = (int)(top >> 20);
    fits = fits && (top == 0u || (E[q] >= 128 && E[q] <= 1900));
  }
  if (!fits) {
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = warp_sum(v[q]);
    return;
  }
#pragma unroll
  for (int q = 0; q < N; q++) {
    const int e = (int)((hi[q] >> 20) & 0x7ffu);
    // the 53-bit significand at bits 5..57, shifted right by E - e, then by one with rounding
    const unsigned long long mant =
        e == 0 ? 0ULL : ((((unsigned long long)((hi[q] & 0xfffffu) | 0x100000u)) << 32) | lo[q]) << 5;
    const unsigned long long mag = ((mant >> min(E[q] - e, 62)) + 1ULL) >> 1;
    const long long F = (int)hi[q] < 0 ? -(long long)mag : (long long)mag;
    const unsigned s0 = __reduce_add_sync(full, (unsigned)F & 0x3fffffu);
    const unsigned s1 = __reduce_add_sync(full, (unsigned)(F >> 22) & 0x3fffffu);
    const int s2 = __reduce_add_sync(full, (int)(F >> 44));
    const long long sum = ((long long)s2 << 44) + ((long long)s1 << 22) + (long long)s0;   // |sum| < 2^62
    const unsigned long long sg = (unsigned long long)(sum >> 63);
    const unsigned long long ax = ((unsigned long long)sum ^ sg) - sg;
    const int lz = __clzll((long long)ax);
    const unsigned long long u = ax << (lz & 63);               // leading one at bit 63
    const unsigned long long m = (u >> 11) + ((u >> 10) & 1ULL);   // 53 bits (a carry bumps the exponent)
    const int ex = E[q] + 7 - lz;                               // biased exponent of the leading one
    const unsigned long long bits = (m + ((unsigned long long)(ex - 1) << 52)) | (sg << 63);
    v[q] = ax == 0ULL ? 0.0 : __longlong_as_double((long long)bits);
  }
}

// The FP32 image of a non-negative double in FP32's normal range, truncated
// (smaller: 0), and the double of a positive normal float: integer operations.
__device__ __forceinline__ float f32_of(int hi, int lo) {
  const int h = hi - (896 << 20);
  return h < (1 << 20) ? 0.0f : __uint_as_float(((unsigned)h << 3) | ((unsigned)lo >> 29));
}
__device__ __forceinline__ double f64_of(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)(b >> 3) + (896 << 20), (int)(b << 29));
}

// beta, tau and scal of larfg_scalars' plain case (n2 = a^2 + ss within
// [1e-290, 1e290]) without FP64 square root or division: f = n2 / 4^h in [1,
// 4); s = sqrt(f) by coupled Newton steps on sqrt and its inverse from an FP32
// seed (Goldschmidt's iteration, residual taken with an FMA); 1 / (|a| 2^-h +
// s) from an FP32 seed by one third-order (Householder) step.  Against the
// exact values, restated on the host for 2 10^7 pairs a, ss with seeds up to
// two units off: tau 1.5, beta 0.9, scal 2.8 units in the last place at most;
// with square root and divisions 2.2, 0.9 and 2.8.
__device__ __forceinline__ void larfg_newton(double a, double ss, double& tau, double& scal, double& beta) {
  const double n2 = fma(a, a, ss);
  const int hi = __double2hiint(n2), lo = __double2loint(n2);
  const int h = ((hi >> 20) - 1023) >> 1;
  const int fhi = hi - (h << 21);
  const double f = __hiloint2double(fhi, lo);
  const double as = fabs(a) * __hiloint2double((1023 - h) << 20, 0);   // |a| 2^-h
  const float ff = f32_of(fhi, lo);
  const float yf = rsqrtf(ff);
  const double y0 = f64_of(yf);
  const double x0 = f64_of(__fdividef(1.0f, fmaf(ff, yf, f32_of(__double2hiint(as), __double2loint(as)))));
  const double g0 = f * y0, h0 = __hiloint2double(__double2hiint(y0) - (1 << 20), __double2loint(y0));   // y0 / 2
  const double r0 = fma(-g0, h0, 0.5);
  const double g1 = fma(g0, r0, g0), h1 = fma(h0, r0, h0);
  const double s = fma(fma(-g1, g1, f), h1, g1);           // sqrt(f)
  const double den = as + s;
  const double y1 = __hiloint2double(__double2hiint(h1) + (1 << 20), __double2loint(h1));   // 2 h1
  const double y = fma(y1, fma(-s, y1, 1.0), y1);          // 1 / sqrt(f)
  const double e = fma(-den, x0, 1.0);
  const double x = fma(x0, fma(e, e, e), x0);              // 1 / den
  tau = fma(as, y, 1.0);                                   // (beta - a) / beta = 1 + |a| / ||.||
  beta = -copysign(__hiloint2double(__double2hiint(s) + (h << 20), __double2loint(s)), a);
  scal = copysign(__hiloint2double(__double2hiint(x) - (h << 20), __double2loint(x)), a);
}

// Named barriers of the panel loop (0: __syncthreads, 1: the split engine's slicers).
constexpr int kBarColumn = 2, kBarStep = 3, kBarScalars = 4;
template <int ID, int N>
__device__ __forceinline__ void bar_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory"); }
template <int ID, int N>
__device__ __forceinline__ void bar_arrive() { asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory"); }

constexpr int kPanelWorkers = kWarps - 2;                                        // warps 1, 2, 3, 5, 6, 7
constexpr int kPanelItems = 3;       // columns of one worker taken at a time
constexpr int kPanelGroups = (kMaxW - 1 + kPanelWorkers * kPanelItems - 1) / (kPanelWorkers * kPanelItems);
constexpr int kPanelRows = 4;        // rows per lane taken at a time: chunks of 128
// The range of the loop's columns, as high words: with x_c unscaled, its dots,
// Gram entries and factors stay in range where no element reaches 2^450 and the
// other column is not much below 2^-400.  Elements are looked at when the panel
// is loaded.  A column's size is looked at in its own step only, which covers
// the steps before: a reflection keeps the norm of the rows it acts on, so
// rows c.. of column j were in step c at least as large as [alpha; x] is in step
// j > c.  Panels outside take the general loop.
__host__ __device__ constexpr unsigned kHiExp(int e) { return (unsigned)(1023 + e) << 20; }   // high word of 2^e
constexpr unsigned kPanelMaxHi = kHiExp(450), kColumnMinHi = kHiExp(-400);
__device__ __forceinline__ unsigned magnitude(double v) {   // the high word of |v|; 0 for zero alone
  return ((unsigned)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u);
}

// TS: unblocked QR of the triangle-on-square panel [R; A] (R w x w, upper part
// used; A m x w dense), the per-column loop of CORE_dtsqrt: column c's
// reflector acts on [R(c,c); A(:,c)].  !TS: of the m x w panel A itself (dgeqr2
// semantics, R = A, ldr = lda): on A(c:, c).  On return column c of A (below
// the diagonal for !TS) holds x_c with v_c = x_c scal[c], tau[c], the w x w
// upper T (ld w) of the block reflector (dlarft 'F','C'); G is scratch.
// Every |element| is below 2^450.  wide: w ints of scratch.  Returns false, the
// panel in an undefined state, at the first column that is below 2^-400 and
// not zero (the same in every thread).
//
// Step c: warp 0 waits for column c (updated first by worker 0), takes its
// norm and scalars; the workers meanwhile take the dots of x_c with every
// other column -- those right of c, to be updated, and those left of it, for
// the Gram entry G(b, c) = v_b . v_c; with the scalars they update their
// columns; warp 4 forms T's column c during step c + 1 (T(0:c, c) = -tau_c
// T(0:c, 0:c) G(0:c, c)).
//
// Larfg: the reflector's convention (LapackLarfg, or tile_kernel.h's): the two
// numbers of column c that scalars() puts into tau[c] and scal[c], and update()'s
// change of a column from its dot with x_c: r_c -= s, a -= f x_c.  nref:
// reflectors formed (columns from there on are updated only).  GRAM false: no
// Gram entries and no T.
struct LapackLarfg {
  static constexpr bool kSplitFactor = false;
  // false: alpha and x below 2^-400, read off the high words: an FP64 comparison
  // is an FP64 instruction too.  ss = 0: H = I.
  __device__ static bool scalars(double a, double ss, double& tau, double& scal, double& beta) {
    const unsigned sh = (unsigned)__double2hiint(ss), ah = (unsigned)__double2hiint(a) & 0x7fffffffu;
    tau = 0.0;
    scal = 1.0;
    beta = a;
    if (sh < kHiExp(-800) && ah < kColumnMinHi) return false;
    if ((sh | (unsigned)__double2loint(ss)) != 0u) larfg_newton(a, ss, tau, scal, beta);
    return true;
  }
  __device__ static bool moves(double tau) { return __double_as_longlong(tau) != 0; }   // (tau = 0 is +0)
  // d = x . a, t: tau (of a Gram entry: the other column's scal).  v = x scal
  __device__ static void update(double& d, double r, double t, double scal, double& s, double& f) {
    s = fma(scal, d, r) * t;
    f = s * scal;
  }
};
// By one warp: whether [alpha; x] is zero, and the column's elements r (n of
// them, at most 32) above alpha are each zero or at least 2^-400: the column
// was then zero or large enough in every step, and H = I.
__device__ __forceinline__ bool zero_column(double alpha, const double* x, int m, const double* r, int n) {
  const int lane = threadIdx.x & 31;
  unsigned t = magnitude(alpha);
  for (int i = lane; i < m; i += 32) t |= magnitude(x[i]);
  if (lane < n && magnitude(r[lane]) < kColumnMinHi) t |= magnitude(r[lane]);
  return __reduce_or_sync(0xffffffffu, t) == 0u;
}
template <bool TS, class Larfg = LapackLarfg, bool GRAM = true>
__device__ __forceinline__ bool panel_qr(double* R, int ldr, double* A, int lda, int m, int w, int nref,
                                         double* tau, double* scal, int* wide, double* G, double* T) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kParty = (kPanelWorkers + 1) * 32;                 // the workers and warp 0
  constexpr int kStepParty = (kPanelWorkers + (GRAM ? 1 : 0)) * 32;   // the workers (and warp 4)
  bool ok = true;
  if (warp == 0) {
    for (int c = 0; c < nref; c++) {
      if (c > 0) bar_sync<kBarColumn, 64>();
      double* x = A + (size_t)c * lda;
      double* al = TS ? R + c + (size_t)c * ldr : x + c;
      const int r0 = TS ? 0 : c + 1;
      const double a = *al;
      double ssv[1] = {0.0};
      for (int rb = r0 & ~127; rb < m; rb += 32 * kPanelRows) {
        double xv[kPanelRows];
#pragma unroll
        for (int i = 0; i < kPanelRows; i++) {
          const int r = rb + 32 * i + lane;
          xv[i] = (r >= r0 && r < m) ? x[r] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kPanelRows; i++)
          if (rb + 32 * i < m && rb + 32 * i + 31 >= r0) ssv[0] = fma(xv[i], xv[i], ssv[0]);
      }
      warp_sums_fixed(ssv);
      const double ss = ssv[0];
      double t, sc, beta;
      if (!Larfg::scalars(a, ss, t, sc, beta)) ok = zero_column(a, x + r0, m - r0, R + (size_t)c * ldr, c);
      __syncwarp();
      if (lane == 0) {
        tau[c] = t;
        scal[c] = sc;
        wide[c] = ok ? 0 : 1;
        *al = beta;
      }
      __syncwarp();
      bar_arrive<kBarScalars, kParty>();
      if (!ok) break;
    }
  } else if (warp == 4) {
    for (int c = 0; GRAM && c < nref; c++) {
      bar_sync<kBarStep, kStepParty>();
      ok = wide[c] == 0;
      if (!ok) break;
      double s = 0.0;
      if (lane < c)
        for (int b = 0; b < c; b++) s = fma(lane <= b ? T[lane + b * w] : 0.0, G[b + c * w], s);
      const double tc = tau[c];   // tau = 0 is +0
      const bool zero = __double_as_longlong(tc) == 0;
      if (lane < w) T[lane + c * w] = lane < c ? (zero ? 0.0 : -tc * s) : (lane == c ? tc : 0.0);
      __syncwarp();
    }
  } else {
    const int wi = warp < 4 ? warp - 1 : warp - 2;
    for (int c = 0; c < nref; c++) {
      // items 0 .. w - 2 - c: columns c + 1 .. w - 1; then columns 0 .. c - 1
      const int nupd = w - 1 - c, items = GRAM ? w - 1 : nupd;
      const int r0 = TS ? 0 : c + 1;
      const double* x = A + (size_t)c * lda;
      double acc[kPanelGroups][kPanelItems];
      auto item = [&](int g, int q) { return wi + (g * kPanelItems + q) * kPanelWorkers; };
      auto column = [&](int it) { return it < nupd ? c + 1 + it : it - nupd; };
      // lane q of a group's first kPanelItems lanes owns item q's scalars
      double rc[kPanelGroups], mul[kPanelGroups];
#pragma unroll
      for (int g = 0; g < kPanelGroups; g++) {
        const int it = item(g, lane < kPanelItems ? lane : 0);
        rc[g] = mul[g] = 0.0;
        if (it < items && (it < nupd || !TS)) rc[g] = R[c + (size_t)column(it) * ldr];
        if (it < items && it >= nupd) mul[g] = scal[it - nupd];
      }
#pragma unroll
      for (int g = 0; g < kPanelGroups; g++) {
        if (item(g, 0) >= items) break;
        const double* aq[kPanelItems];   // (past the last item: column c, the result unused)
#pragma unroll
        for (int q = 0; q < kPanelItems; q++) {
          acc[g][q] = 0.0;
          aq[q] = A + (size_t)(item(g, q) < items ? column(item(g, q)) : c) * lda;
        }
        for (int rb = r0 & ~127; rb < m; rb += 32 * kPanelRows) {
          double xv[kPanelRows], av[kPanelItems][kPanelRows];
#pragma unroll
          for (int i = 0; i < kPanelRows; i++) {
            const int r = rb + 32 * i + lane;
            const bool in = r >= r0 && r < m;
            xv[i] = in ? x[r] : 0.0;
#pragma unroll
            for (int q = 0; q < kPanelItems; q++) av[q][i] = in ? aq[q][r] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < kPanelRows; i++)
            if (rb + 32 * i < m && rb + 32 * i + 31 >= r0)
#pragma unroll
              for (int q = 0; q < kPanelItems; q++)
                if (q < kPanelItems - 1 || item(g, q) < items) acc[g][q] = fma(xv[i], av[q][i], acc[g][q]);
        }
        warp_sums_fixed(acc[g]);
      }
      bar_sync<kBarScalars, kParty>();
      ok = wide[c] == 0;
      if (!ok) {
        bar_sync<kBarStep, kStepParty>();   // warp 4 looks at wide[c] too
        break;
      }
      const double t = tau[c], sc = scal[c];
      const bool moves = Larfg::moves(t);
#pragma unroll
      for (int g = 0; g < kPanelGroups; g++) {
        if (item(g, 0) >= items) break;
        const int mine = item(g, lane < kPanelItems ? lane : 0);
        double d = acc[g][0];
#pragma unroll
        for (int q = 1; q < kPanelItems; q++) d = lane == q ? acc[g][q] : d;
        // update: s = tau (v_c . a_j + r_cj); Gram: G(b, c) = v_b . v_c
        double s, f;
        Larfg::update(d, rc[g], mine < nupd ? t : mul[g], sc, s, f);
        if (lane < kPanelItems && mine < items) {
          if (mine < nupd)
            R[c + (size_t)(c + 1 + mine) * ldr] = rc[g] - s;
          else
            G[mine - nupd + c * w] = s;
        }
#pragma unroll
        for (int q = 0; q < kPanelItems; q++) {
          const int it = item(g, q);
          if (it >= nupd) break;
          const double fq = __shfl_sync(0xffffffffu, f, q);
          double* aj = A + (size_t)(c + 1 + it) * lda;
          bool whole = moves;   // a -= f x with f as one factor
          if (Larfg::kSplitFactor) {
            // a factor that is not in range is two, a -= (t x) d, and so is one
            // whose products can be exact (its low word is zero): the column is
            // then a short multiple of x, 1 or 2 of it, say, and would become
            // exactly zero instead of rounding errors (see the convention)
            const unsigned fh = (unsigned)__double2hiint(fq) & 0x7fffffffu;
            whole = fh >= kHiExp(-960) && fh < kHiExp(960) && __double2loint(fq) != 0;
            const double dq = __shfl_sync(0xffffffffu, d, q);
            for (int r = r0 + lane; r < m && !whole; r += 32) aj[r] = fma(-(t * x[r]), dq, aj[r]);
          }
          for (int rb = r0 & ~127; rb < m && whole; rb += 32 * kPanelRows) {
            double xv[kPanelRows], av[kPanelRows];
#pragma unroll
            for (int i = 0; i < kPanelRows; i++) {
              const int r = rb + 32 * i + lane;
              const bool in = r >= r0 && r < m;
              xv[i] = in ? x[r] : 0.0;
              av[i] = in ? aj[r] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < kPanelRows; i++) {
              const int r = rb + 32 * i + lane;
              if (rb + 32 * i < m && rb + 32 * i + 31 >= r0) {
                const double y = fma(-fq, xv[i], av[i]);
                if (r >= r0 && r < m) aj[r] = y;
              }
            }
          }
          if (it == 0 && c + 1 < nref) {
            __syncwarp();
            bar_arrive<kBarColumn, 64>();
          }
        }
      }
      bar_sync<kBarStep, kStepParty>();
    }
  }
  __syncthreads();
  return ok;
}

// ---------------------------------------------------------------------------
// Apply the transpose of one w-column block reflector H = I - V T V^T,
// V = [Vt; Vb], to [Ct; Cb] held in shared memory:
//     W = Vt^T Ct + Vb^T Cb;  W = T^T W;  Ct -= Vt W;  Cb -= Vb W
// (notrans: H itself, W = T W).
// Vt: w x w unit lower (unit_top) or the identity; Vb: mb x w.  V and T are
// read from global memory (ld ldv / ldt), or, with `resident` (mb <= RC), are
// in shared memory already: T in sT (zero below the diagonal), Vb in sVb (ld
// RC + 1), Vt in sVt.  ncol must be a multiple of 8.
// v_col0 >= 0: Vb is upper triangular (a TT merge's reflectors, stored in the
// upper triangle of a tile whose lower part holds other data): element
// (mb_off + r, c) is used when mb_off + r <= v_col0 + c, else taken as zero.
// ---------------------------------------------------------------------------
template <typename RT = double>
__device__ void apply_block_t(const double* __restrict__ gV, int ldv, int mb_off,
                              const double* __restrict__ gT, int ldt, int w, int mb, bool unit_top,
                              RT* Ct, int ldct, RT* Cb, int ldcb, int ncol, RT* smem,
                              const SmemPlan& sp, int RC, bool notrans = false, int v_col0 = -1,
                              bool resident = false) {
  RT* sVb = smem + sp.off_vb;
  RT* sVt = smem + sp.off_vt;
  RT* sT = smem + sp.off_t;
  RT* sW = smem + sp.off_w;
  RT* sW2 = smem + sp.off_w2;
  RT* sPart = smem + sp.off_part;
  const int tid = threadIdx.x;
  const int ldvs = RC + 1;

  // T block and the unit-lower top of V
  for (int e = tid; e < w * w && !resident; e += kThreads) {
    const int r = e % w, c = e / w;
    sT[e] = (r <= c) ? RT(ldg_cg(gT + r + (size_t)c * ldt)) : RT(0);
    if (unit_top) sVt[e] = (r > c) ? RT(ldg_cg(gV + r + (size_t)c * ldv)) : (r == c ? RT(1) : RT(0));
  }

  // ---- W = Vt^T Ct + Vb^T Cb -------------------------------------------
  const int G8 = ncol >> 3;
  const int outs = w * G8;                       // items per split
  int S = kSplitItems / (outs > 0 ? outs : 1);
  if (S < 1) S = 1;
  const int item = tid;
  const int a = item % w;
  const int g = (item / w) % (G8 > 0 ? G8 : 1);
  const int s = item / outs;
  const bool active = (outs > 0) && (item < outs * S) && (s < S);
  RT acc[8];
#pragma unroll
  for (int q = 0; q < 8; q++) acc[q] = RT(0);
  for (int r0 = 0; r0 < mb; r0 += RC) {
    const int rc = min(RC, mb - r0);
    __syncthreads();
    for (int e = tid; e < rc * w && !resident; e += kThreads) {
      const int r = e % rc, c = e / rc;
      sVb[r + c * ldvs] = (v_col0 < 0 || mb_off + r0 + r <= v_col0 + c)
                              ? RT(ldg_cg(gV + mb_off + r0 + r + (size_t)c * ldv)) : RT(0);
    }
    __syncthreads();
    if (active) {
      const RT* cb = Cb + r0 + (size_t)(8 * g) * ldcb;
      for (int r = s; r < rc; r += S) {
        const RT v = sVb[r + a * ldvs];
#pragma unroll
        for (int q = 0; q < 8; q++) acc[q] = fma(v, cb[r + (size_t)q * ldcb], acc[q]);
      }
    }
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int q = 0; q < 8; q++) sPart[(s * w + a) * 8 * G8 + g * 8 + q] = acc[q];
  }
  __syncthreads();
  for (int e = tid; e < w * ncol; e += kThreads) {
    const int aa = e % w, j = e / w;
    RT v = RT(0);
    for (int ss = 0; ss < S; ss++) v += sPart[(ss * w + aa) * 8 * G8 + j];
    RT top = Ct[aa + (size_t)j * ldct];
    if (unit_top)
      for (int r = aa + 1; r < w; r++) top = fma(sVt[r + aa * w], Ct[r + (size_t)j * ldct], top);
    sW[aa + j * w] = v + top;
  }
  __syncthreads();

  // ---- W2 = T^T W (notrans: T W) --------------------------------------------
  for (int e = tid; e < w * ncol; e += kThreads) {
    const int aa = e % w, j = e / w;
    RT v = RT(0);
    if (notrans)
      for (int b = aa; b < w; b++) v = fma(sT[aa + b * w], sW[b + j * w], v);
    else
      for (int b = 0; b <= aa; b++) v = fma(sT[b + aa * w], sW[b + j * w], v);
    sW2[aa + j * w] = v;
  }
  __syncthreads();

  // ---- Ct -= Vt W2 ----------------------------------------------------------
  for (int e = tid; e < w * ncol; e += kThreads) {
    const int aa = e % w, j = e / w;
    RT v = sW2[aa + j * w];
    if (unit_top)
      for (int b = 0; b < aa; b++) v = fma(sVt[aa + b * w], sW2[b + j * w], v);
    Ct[aa + (size_t)j * ldct] -= v;
  }

  // ---- Cb -= Vb W2 ----------------------------------------------------------
  // from the last chunk, which is still staged, back to the first
  const int last = (mb - 1) / RC * RC;
  for (int r0 = last; r0 >= 0; r0 -= RC) {
    const int rc = min(RC, mb - r0);
    __syncthreads();
    for (int e = tid; e < rc * w && r0 != last; e += kThreads) {
      const int r = e % rc, c = e / rc;
      sVb[r + c * ldvs] = (v_col0 < 0 || mb_off + r0 + r <= v_col0 + c)
                              ? RT(ldg_cg(gV + mb_off + r0 + r + (size_t)c * ldv)) : RT(0);
    }
    if (r0 != last) __syncthreads();
    for (int e = tid; e < rc * G8; e += kThreads) {
      const int r = e % rc, gg = e / rc;
      RT acc2[8];
#pragma unroll
      for (int q = 0; q < 8; q++) acc2[q] = RT(0);
      for (int b = 0; b < w; b++) {
        const RT v = sVb[r + b * ldvs];
#pragma unroll
        for (int q = 0; q < 8; q++) acc2[q] = fma(v, sW2[b + (8 * gg + q) * w], acc2[q]);
      }
      RT* cb = Cb + r0 + r + (size_t)(8 * gg) * ldcb;
#pragma unroll
      for (int q = 0; q < 8; q++) cb[(size_t)q * ldcb] -= acc2[q];
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Task bodies.  All tile pointers are global (ld = NB).  T tiles are NB x NB;
// the factorization writes their diagonal w x w blocks.
// ---------------------------------------------------------------------------

template <typename RT = double>
__device__ void load_block(RT* s, int lds, const double* g, int ldg, int m, int n) {
  for (int e = threadIdx.x; e < m * n; e += kThreads) {
    const int r = e % m, c = e / m;
    s[r + (size_t)c * lds] = RT(ldg_cg(g + r + (size_t)c * ldg));
  }
}
template <typename RT = double>
__device__ void store_block(double* g, int ldg, const RT* s, int lds, int m, int n) {
  for (int e = threadIdx.x; e < m * n; e += kThreads) {
    const int r = e % m, c = e / m;
    stg_cg(g + r + (size_t)c * ldg, double(s[r + (size_t)c * lds]));
  }
}
// The upper part (row r <= col0 + c) of an m x n block, zero below; and its
// store (a TT merge's panel columns).
template <typename RT = double>
__device__ void load_block_upper(RT* s, int lds, const double* g, int ldg, int m, int n, int col0) {
  for (int e = threadIdx.x; e < m * n; e += kThreads) {
    const int r = e % m, c = e / m;
    s[r + (size_t)c * lds] = (r <= col0 + c) ? RT(ldg_cg(g + r + (size_t)c * ldg)) : RT(0);
  }
}
template <typename RT = double>
__device__ void store_block_upper(double* g, int ldg, const RT* s, int lds, int m, int n, int col0) {
  for (int e = threadIdx.x; e < m * n; e += kThreads) {
    const int r = e % m, c = e / m;
    if (r <= col0 + c) stg_cg(g + r + (size_t)c * ldg, double(s[r + (size_t)c * lds]));
  }
}

// The high words of the largest |element| of the m x n blocks loaded so far:
// *top (shared, zeroed before) collects it over the CTA's threads.
__device__ __forceinline__ void note_top(unsigned top, unsigned* s_top) {
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) atomicMax(s_top, top);
}
__device__ __forceinline__ unsigned top_of(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
// load_block / load_block_upper (col0 >= 0) of an FP64 panel block; returns
// this thread's largest high word.
__device__ __forceinline__ unsigned load_panel(double* s, int lds, const double* g, int ldg, int m, int n,
                                               int col0 = -1) {
  unsigned top = 0;
#pragma unroll 4
  for (int e = threadIdx.x; e < m * n; e += kThreads) {
    const int r = e % m, c = e / m;
    const double v = (col0 < 0 || r <= col0 + c) ? ldg_cg(g + r + (size_t)c * ldg) : 0.0;
    s[r + (size_t)c * lds] = v;
    top = max(top, top_of(v));
  }
  return top;
}
// The general FP64 column loops (panels with elements of 2^450 and above,
// infinities or NaN, or columns below 2^-400), their T, and scal = 1: their
// columns are v itself.
template <bool TS>
__device__ __noinline__ void panel_qr_general(double* R, int ldr, double* A, int lda, int m, int w, double* tau,
                                              double* scal, double* G, double* T) {
  if (TS)
    panel_qr_ts_fused(R, ldr, A, lda, m, w, tau, G);
  else
    panel_qr_ge_fused(A, lda, m, w, tau, G);
  if (threadIdx.x < 32) t_from_gram(G, tau, T, w);
  if (threadIdx.x < w) scal[threadIdx.x] = 1.0;
  __syncthreads();
}

// Inner block b of CORE_dgeqrt(NB, NB, IB, A, NB, T, NB, TAU): the QR of
// columns [b w, (b+1) w) from row b w down (blocks 0..b-1 done), its T block,
// and (trailing) its application to the columns right of it.  It writes rows
// >= b w of the tile only: rows [b w, (b+1) w) of R are final afterwards.
template <typename RT = double>
__device__ void task_geqrt_blk(double* A, double* T, double* tau_g, const TileShape& sh, double* smem,
                               const SmemPlan& sp, int b, bool trailing = true) {
  const int NB = sh.NB, w = sh.w;
  constexpr bool kFp64 = sizeof(RT) == sizeof(double);
  RT* sm = reinterpret_cast<RT*>(smem);
  RT* sP = sm + sp.off_c1;
  RT* sTau = sm + sp.off_tau;
  RT* sG = sm + sp.off_g;
  RT* sTb = sm + sp.off_t;
  bool resident = false;   // V and T left in shared memory for the trailing update
  {
    const int i0 = b * w;
    const int m = NB - i0;
    int* wide = reinterpret_cast<int*>(sm + sp.off_red);
    unsigned* s_top = reinterpret_cast<unsigned*>(wide + kMaxW);
    if (kFp64 && threadIdx.x == 0) *s_top = 0u;
    __syncthreads();
    if constexpr (kFp64) {
      double* scal = sm + sp.off_scal;
      note_top(load_panel(sP, NB, A + i0 + (size_t)i0 * NB, NB, m, w), s_top);
      __syncthreads();
      bool general = *s_top >= kPanelMaxHi;
      if (!general && !panel_qr<false>(sP, NB, sP, NB, m, w, w, sTau, scal, wide, sG, sTb)) {
        general = true;
        load_panel(sP, NB, A + i0 + (size_t)i0 * NB, NB, m, w);
        __syncthreads();
      }
      if (general) panel_qr_general<false>(sP, NB, sP, NB, m, w, sTau, scal, sG, sTb);
      // R and V = x scal to the tile; V also to the trailing update's buffers
      resident = m - w <= sh.RC;
      double* sVb = sm + sp.off_vb;
      double* sVt = sm + sp.off_vt;
      for (int e = threadIdx.x; e < m * w; e += kThreads) {
        const int r = e % m, c = e / m;
        double v = sP[r + (size_t)c * NB];
        if (r > c) v *= scal[c];
        stg_cg(A + i0 + r + (size_t)(i0 + c) * NB, v);
        if (r < w)
          sVt[r + c * w] = r > c ? v : (r == c ? 1.0 : 0.0);
        else if (resident)
          sVb[r - w + c * (sh.RC + 1)] = v;
      }
    } else {
      load_block(sP, NB, A + i0 + (size_t)i0 * NB, NB, m, w);
      __syncthreads();
      panel_qr_ge_fused(sP, NB, m, w, sTau, sG);
      if (threadIdx.x < 32) t_from_gram(sG, sTau, sTb, w);
      __syncthreads();
      store_block(A + i0 + (size_t)i0 * NB, NB, sP, NB, m, w);
    }
    store_block(T + i0 + (size_t)i0 * NB, NB, sTb, w, w, w);
    for (int e = threadIdx.x; e < w; e += kThreads) stg_cg(tau_g + i0 + e, double(sTau[e]));
    __syncthreads();
    for (int c0 = trailing ? i0 + w : NB; c0 < NB; c0 += sh.PB) {
      const int ncol = min(sh.PB, NB - c0);
      RT* sC = sm + sp.off_c1;
      __syncthreads();
      load_block(sC, NB, A + i0 + (size_t)c0 * NB, NB, m, ncol);
      __syncthreads();
      apply_block_t(A + i0 + (size_t)i0 * NB, NB, w, T + i0 + (size_t)i0 * NB, NB, w, m - w, true,
                    sC, NB, sC + w, NB, ncol, sm, sp, sh.RC, false, -1, resident);
      store_block(A + i0 + (size_t)c0 * NB, NB, sC, NB, m, ncol);
    }
  }
  __syncthreads();
}

// Inner block b of CORE_dtsqrt(NB, NB, IB, A1, NB, A2, NB, T, NB, TAU): A1
// holds R (upper part) above the GEQRT's V (strict lower part, left
// untouched).  The QR of [R(bw:(b+1)w, bw:(b+1)w); A2(:, bw:(b+1)w)] (blocks
// 0..b-1 of this tile done), its T block, and its application to the columns
// right of it.  Of A1 it touches rows [b w, (b+1) w) only, and those rows are
// touched by no other block of this TSQRT: once block b is done here, block b
// of the TSQRT of the next tile below may run.
// a2_upper: the TT merge (CORE_dttqrt): A2 is upper triangular (the R of a
// domain's top tile; its strict lower part holds that tile's GEQRT reflectors
// and is neither read nor written).  The reflectors keep A2's shape, so the
// same arithmetic on A2 with zeros below the diagonal is exact, and only the
// upper triangle is stored back.
template <typename RT = double>
__device__ void task_tsqrt_blk(double* A1, double* A2, double* T, double* tau_g, const TileShape& sh,
                               double* smem, const SmemPlan& sp, int b, bool a2_upper = false,
                               bool trailing = true) {
  const int NB = sh.NB, w = sh.w;
  constexpr bool kFp64 = sizeof(RT) == sizeof(double);
  RT* sm = reinterpret_cast<RT*>(smem);
  RT* sA = sm + sp.off_c1;     // NB x w panel of A2
  RT* sR = sm + sp.off_vt;     // w x w block of R
  RT* sTau = sm + sp.off_tau;
  RT* sG = sm + sp.off_g;
  RT* sTb = sm + sp.off_t;
  bool resident = false;   // V and T left in shared memory for the trailing update
  {
    const int i0 = b * w;
    int* wide = reinterpret_cast<int*>(sm + sp.off_red);
    unsigned* s_top = reinterpret_cast<unsigned*>(wide + kMaxW);
    if (kFp64 && threadIdx.x == 0) *s_top = 0u;
    __syncthreads();
    if constexpr (kFp64) {
      double* scal = sm + sp.off_scal;
      // R's strictly lower part (the GEQRT's V) is neither used nor counted
      auto load = [&]() {
        const unsigned top = load_panel(sA, NB, A2 + (size_t)i0 * NB, NB, NB, w, a2_upper ? i0 : -1);
        return max(top, load_panel(sR, w, A1 + i0 + (size_t)i0 * NB, NB, w, w, 0));
      };
      note_top(load(), s_top);
      __syncthreads();
      bool general = *s_top >= kPanelMaxHi;
      if (!general && !panel_qr<true>(sR, w, sA, NB, NB, w, w, sTau, scal, wide, sG, sTb)) {
        general = true;
        load();
        __syncthreads();
      }
      if (general) panel_qr_general<true>(sR, w, sA, NB, NB, w, sTau, scal, sG, sTb);
      // V = x scal to the tile (a merge: its upper triangle) and to the
      // trailing update's buffer
      resident = NB <= sh.RC;
      double* sVb = sm + sp.off_vb;
      for (int e = threadIdx.x; e < NB * w; e += kThreads) {
        const int r = e % NB, c = e / NB;
        const double v = sA[r + (size_t)c * NB] * scal[c];
        if (!a2_upper || r <= i0 + c) stg_cg(A2 + r + (size_t)(i0 + c) * NB, v);
        if (resident) sVb[r + c * (sh.RC + 1)] = v;
      }
    } else {
      if (a2_upper)
        load_block_upper(sA, NB, A2 + (size_t)i0 * NB, NB, NB, w, i0);
      else
        load_block(sA, NB, A2 + (size_t)i0 * NB, NB, NB, w);
      load_block(sR, w, A1 + i0 + (size_t)i0 * NB, NB, w, w);
      __syncthreads();
      panel_qr_ts_fused(sR, w, sA, NB, NB, w, sTau, sG);
      if (threadIdx.x < 32) t_from_gram(sG, sTau, sTb, w);
      __syncthreads();
      if (a2_upper)
        store_block_upper(A2 + (size_t)i0 * NB, NB, sA, NB, NB, w, i0);
      else
        store_block(A2 + (size_t)i0 * NB, NB, sA, NB, NB, w);
    }
    for (int e = threadIdx.x; e < w * w; e += kThreads) {
      const int r = e % w, c = e / w;
      if (r <= c) stg_cg(A1 + i0 + r + (size_t)(i0 + c) * NB, double(sR[r + c * w]));
    }
    store_block(T + i0 + (size_t)i0 * NB, NB, sTb, w, w, w);
    for (int e = threadIdx.x; e < w; e += kThreads) stg_cg(tau_g + i0 + e, double(sTau[e]));
    __syncthreads();
    for (int c0 = trailing ? i0 + w : NB; c0 < NB; c0 += sh.PB) {
      const int ncol = min(sh.PB, NB - c0);
      RT* sCt = sm + sp.off_c1;  // w x ncol rows of R (the panel area is free now)
      RT* sCb = sm + sp.off_c1 + w * sh.PB;  // NB x ncol of A2 after the R rows
      __syncthreads();
      // A TT merge's block reflectors reach rows < i0 + w of A2 only: the rows
      // below belong to the domain top's own later blocks, which its chain may
      // still be updating, so they are neither read nor written here.
      const int mrows = a2_upper ? i0 + w : NB;
      load_block(sCt, w, A1 + i0 + (size_t)c0 * NB, NB, w, ncol);
      load_block(sCb, NB, A2 + (size_t)c0 * NB, NB, mrows, ncol);
      __syncthreads();
      apply_block_t(A2 + (size_t)i0 * NB, NB, 0, T + i0 + (size_t)i0 * NB, NB, w, mrows, false, sCt, w,
                    sCb, NB, ncol, sm, sp, sh.RC, false, a2_upper ? i0 : -1, resident);
      store_block(A1 + i0 + (size_t)c0 * NB, NB, sCt, w, w, ncol);
      store_block(A2 + (size_t)c0 * NB, NB, sCb, NB, mrows, ncol);
    }
  }
  __syncthreads();
}

// Columns [cbeg, cbeg + cols) of the trailing update of inner block b of a panel
// tile, as a task of its own: of a GEQRT (A2 null: V and C in the tile A1, on
// rows >= b w) or of a TSQRT (rows [b w, (b+1) w) of R in A1, all of A2).
template <typename RT = double>
__device__ void task_trailing(double* A1, double* A2, const double* T, const TileShape& sh, double* smem,
                              const SmemPlan& sp, int b, int cbeg, int cols) {
  const int NB = sh.NB, w = sh.w;
  RT* sm = reinterpret_cast<RT*>(smem);
  const int i0 = b * w;
  const int m = A2 ? NB : NB - i0;
  const double* V = A2 ? A2 + (size_t)i0 * NB : A1 + i0 + (size_t)i0 * NB;
  for (int c0 = cbeg; c0 < cbeg + cols; c0 += sh.PB) {
    const int ncol = min(sh.PB, cbeg + cols - c0);
    RT* sCt = sm + sp.off_c1;                                // the w x ncol rows of R (GEQRT: with the rows below)
    RT* sCb = A2 ? sCt + w * sh.PB : sCt + w;
    const int ldt = A2 ? w : NB;
    double* top = A1 + i0 + (size_t)c0 * NB;
    __syncthreads();
    load_block(sCt, ldt, top, NB, A2 ? w : m, ncol);
    if (A2) load_block(sCb, NB, A2 + (size_t)c0 * NB, NB, m, ncol);
    __syncthreads();
    apply_block_t(V, NB, A2 ? 0 : w, T + i0 + (size_t)i0 * NB, NB, w, A2 ? m : m - w, !A2, sCt, ldt, sCb, NB, ncol,
                  sm, sp, sh.RC);
    store_block(top, NB, sCt, ldt, A2 ? w : m, ncol);
    if (A2) store_block(A2 + (size_t)c0 * NB, NB, sCb, NB, m, ncol);
  }
  __syncthreads();
}

// CORE_dormqr(Left, Trans, NB, ncol, NB, IB, V, NB, T, NB, C, NB) on columns
// [c0, c0+ncol) of C (notrans: CORE_dormqr(Left, NoTrans, ...), the inner
// blocks in reverse order).
inline __device__ void task_larfb(const double* V, const double* T, double* C, int c0, int ncol,
                           const TileShape& sh, double* smem, const SmemPlan& sp, bool notrans = false) {
  const int NB = sh.NB, w = sh.w;
  double* sC = smem + sp.off_c1;
  __syncthreads();
  load_block(sC, NB, C + (size_t)c0 * NB, NB, NB, ncol);
  __syncthreads();
  for (int b = 0; b < NB / w; b++) {
    const int i0 = (notrans ? NB / w - 1 - b : b) * w;
    apply_block_t(V + i0 + (size_t)i0 * NB, NB, w, T + i0 + (size_t)i0 * NB, NB, w, NB - i0 - w, true,
                  sC + i0, NB, sC + i0 + w, NB, ncol, smem, sp, sh.RC, notrans);
  }
  store_block(C + (size_t)c0 * NB, NB, sC, NB, NB, ncol);
  __syncthreads();
}

// CORE_dtsmqr(Left, Trans, NB, ncol, NB, ncol, NB, IB, A1, NB, A2, NB, V, NB,
// T, NB) on columns [c0, c0+ncol) of A1 and A2 (notrans: Left, NoTrans, the
// inner blocks in reverse order).  v_upper: CORE_dttmqr, V is the upper
// triangle (with the diagonal) of its tile.
inline __device__ void task_ssrfb(double* A1, double* A2, const double* V, const double* T, int c0,
                           int ncol, const TileShape& sh, double* smem, const SmemPlan& sp,
                           bool notrans = false, bool v_upper = false) {
  const int NB = sh.NB, w = sh.w;
  double* s1 = smem + sp.off_c1;
  double* s2 = smem + sp.off_c2;
  __syncthreads();
  load_block(s1, NB, A1 + (size_t)c0 * NB, NB, NB, ncol);
  load_block(s2, NB, A2 + (size_t)c0 * NB, NB, NB, ncol);
  __syncthreads();
  for (int b = 0; b < NB / w; b++) {
    const int i0 = (notrans ? NB / w - 1 - b : b) * w;
    apply_block_t(V + (size_t)i0 * NB, NB, 0, T + i0 + (size_t)i0 * NB, NB, w, NB, false, s1 + i0, NB,
                  s2, NB, ncol, smem, sp, sh.RC, notrans, v_upper ? i0 : -1);
  }
  store_block(A1 + (size_t)c0 * NB, NB, s1, NB, NB, ncol);
  store_block(A2 + (size_t)c0 * NB, NB, s2, NB, NB, ncol);
  __syncthreads();
}

}  // namespace hqr
