// hqr_oztasks.cuh -- tile tasks of the split-precision path (NB = 128).
//
// A block reflector H = I - [I; V] T [I; V]^T applied as H^T (the
// factorization, Q^T C; CORE_dtsmqr / CORE_dormqr) or as H (Q generation)
// to a column block [C_top; C_bot] needs W2 = M (C_top + V^T C_bot), M = T^T
// or T, then C_top -= W2 and C_bot -= V W2.  With Z = M V^T prepared once per
// panel tile, W2 = Z C_bot + M C_top is ONE product of K = 256:
//
//   OZPREP(i,k): T from V and TAU (LAPACK dlarft, forward, columnwise -- the
//     full NB x NB T Hybrid_make_Q rebuilds with IB = NB,
//     Hybrid_make_Q.c:124-130,159-163; G = V^T V on the tensor cores, the
//     recurrence in shared memory), Z = M V^T on the tensor cores, and the
//     sliced left operands X1 = [Z | M] (128 x 256, one row exponent per row
//     over both halves) and V.
//   OZAPPLY: one 64-column block of an SSRFB (V dense) or LARFB (V unit
//     lower, no C_top) as two products:
//       W2 = [Z | M] [C_bot; C_top]   (LARFB: Z C)  -> C_top -= W2
//       C_bot -= V W2,
//     with W2 kept in shared memory between them: two epilogues per task.
#pragma once
#include "hqr_ozaki.cuh"

namespace hqr {

// Slots of a panel tile's prepared operands (operand_bytes() each) and of
// their row exponents (kK ints each): X1 = [Z | M] (slots 0-1: 16 K chunks,
// one exponent per row in slot 0), V (slot 2), and slot 3, scratch of the
// preparation (V^T, then M with its own exponents).
constexpr size_t kOzX = 0, kOzV = 2, kOzS = 3;

// T upper triangular, packed by columns in shared memory: T(a, b) (a <= b)
// at b (b + 1) / 2 + a.  As a left operand: X = T^T (transposed) or X = T.
struct PackedTAcc {
  const double* t;
  bool transposed;
  __device__ __forceinline__ double operator()(int r, int k) const {
    if (transposed) return (k <= r) ? t[r * (r + 1) / 2 + k] : 0.0;   // T^T(r, k) = T(k, r)
    return (r <= k) ? t[k * (k + 1) / 2 + r] : 0.0;
  }
};

// T recurrence (dlarft 'F','C', k = NB = 128) in shared memory,
//   T(c, c) = tau_c;  T(0:c, c) = -tau_c T(0:c, 0:c) G(0:c, c)  (zero when tau_c = 0),
// by doubling: first the diagonal 16 x 16 blocks (each row runs its own scalar
// recurrence over its own row: no barrier), then for H = 16, 32, 64 the block
// of every pair of neighbouring H x H diagonal blocks,
//   T12 = -T11 (G12 T22),
// the same sums regrouped (tau_c = 0 leaves column c zero either way).  The
// FP64 pipe bounds it (an FMA of a warp per 16 cycles of the SM; 350 kFMA are
// 178 kcycles), so each product is laid out for full warps that skip the
// triangle's zeros: the lanes run along the dense side, a thread's H / 4 sums
// along the triangular one, four apart, which gives every warp the same work,
// four of them at a time: loops whose bodies need no branch per term keep the
// loads ahead of the FMAs (all H / 4 sums at once with a branch per term took
// 403 kcycles).  210 kcycles; by block columns of 16 it took 310.
// sG: strictly upper part of G = V^T V, packed: G(b, c) (b < c) at c (c - 1) / 2 + b.
// sT: the result, packed upper: T(a, b) (a <= b) at b (b + 1) / 2 + a.
// sX: 64 x kLdX doubles of scratch.
constexpr int kLdX = 65;
// Sixteen terms of four sums: acc[i] += x(d) y(d, i), d = 0..15; with DIAG only
// the terms of a triangular block, d <= 4 i + res (UPPER) or d >= 4 i + res.
template <bool DIAG, bool UPPER, class X, class Y>
__device__ __forceinline__ void t_terms(double (&acc)[4], int res, X x, Y y) {
#pragma unroll
  for (int d = 0; d < 16; d++) {
    const double xd = x(d);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (DIAG && (UPPER ? i < d / 4 : i > d / 4)) continue;
      const double yd = y(d, i);
      const bool in = !DIAG || i != d / 4 || (UPPER ? d % 4 <= res : d % 4 >= res);
      acc[i] = fma(in ? xd : 0.0, in ? yd : 0.0, acc[i]);
    }
  }
}
template <int H>
__device__ __forceinline__ void t_double(const double* sG, double* sT, double* sX) {
  constexpr int L = H < 32 ? H : 32, NB = H / 16;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // the pair of blocks, this lane's dense index, this thread's residue mod 4
  const int pair = H == 64 ? 0 : H == 32 ? w >> 2 : w >> 1;
  const int dense = (H == 64 ? (w & 1) * 32 : 0) + lane % L;
  const int res = H == 64 ? w >> 1 : H == 32 ? w & 3 : (w & 1) * 2 + lane / L;
  const int b1 = pair * 2 * H, b2 = b1 + H;
  double* X = sX + pair * H;   // (the pairs' columns side by side: H * pairs = 64)
  auto T = [&](int a, int b) -> double& { return sT[b * (b + 1) / 2 + a]; };
  // X(r, j) = sum_{d <= j} G12(r, d) T22(d, j): r = dense, j = 16 jb + 4 i + res
#pragma unroll 1
  for (int jb = 0; jb < NB; jb++) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    auto g = [&](int db) {
      return [=](int d) { const int c = b2 + 16 * db + d; return sG[c * (c - 1) / 2 + b1 + dense]; };
    };
    auto t = [&](int db) {
      return [=](int d, int i) { return T(b2 + 16 * db + d, b2 + 16 * jb + 4 * i + res); };
    };
#pragma unroll 1
    for (int db = 0; db < jb; db++) t_terms<false, true>(acc, res, g(db), t(db));
    t_terms<true, true>(acc, res, g(jb), t(jb));
#pragma unroll
    for (int i = 0; i < 4; i++) X[dense * kLdX + 16 * jb + 4 * i + res] = acc[i];
  }
  __syncthreads();
  // T12(r, j) = -sum_{d >= r} T11(r, d) X(d, j): j = dense, r = 16 rb + 4 i + res
#pragma unroll 1
  for (int rb = 0; rb < NB; rb++) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    auto x = [&](int db) { return [=](int d) { return X[(16 * db + d) * kLdX + dense]; }; };
    auto t = [&](int db) {
      return [=](int d, int i) { return T(b1 + 16 * rb + 4 * i + res, b1 + 16 * db + d); };
    };
    t_terms<true, false>(acc, res, x(rb), t(rb));
#pragma unroll 1
    for (int db = rb + 1; db < NB; db++) t_terms<false, false>(acc, res, x(db), t(db));
#pragma unroll
    for (int i = 0; i < 4; i++) T(b1 + 16 * rb + 4 * i + res, b2 + dense) = -acc[i];
  }
  __syncthreads();
}
inline __device__ void t_recurrence(const double* sG, double* sT, double* sX, const double* tau) {
  constexpr int K = oz::kK, BS = 16;
  const int tid = threadIdx.x;
  if (tid < K) {
    // row `tid` of its block: every T(tid, d) goes to the sums of the later columns
    const int b = tid / BS, a = tid % BS;
    const double my_tau = __ldcg(tau + tid);
    double acc[BS];
#pragma unroll
    for (int c = 0; c < BS; c++) acc[c] = 0.0;
#pragma unroll
    for (int d = 0; d < BS; d++) {
      const int gd = b * BS + d;
      const double td = __shfl_sync(0xffffffffu, my_tau, d, BS);
      if (d >= a) {
        const double t = d == a ? td : td == 0.0 ? 0.0 : -td * acc[d];
        sT[gd * (gd + 1) / 2 + tid] = t;
#pragma unroll
        for (int c = d + 1; c < BS; c++) {
          const int gc = b * BS + c;
          acc[c] = fma(t, sG[gc * (gc - 1) / 2 + gd], acc[c]);
        }
      }
    }
  }
  __syncthreads();
  t_double<16>(sG, sT, sX);
  t_double<32>(sG, sT, sX);
  t_double<64>(sG, sT, sX);
}

// Shape of a panel tile's reflectors V.
enum VKind : int {
  kVDense = 0,       // TSQRT: the whole tile
  kVUnitLower = 1,   // GEQRT: strictly below the diagonal, unit diagonal
  kVUpper = 2,       // TT merge: the upper triangle with the diagonal
};

// OZPREP of panel tile V (global, NB x NB, of shape vkind) with TAU tau.
// G: NB x NB global scratch (it ends holding M).  slices / exps: this tile's
// prepared operands and row exponents; M = T^T (applying H^T) or, with
// t_transposed false, T (applying H).  sm: the CTA's dynamic shared memory
// (oz::kSmemBytes).  False on a device time-out.
inline __device__ bool task_ozprep(const double* V, const double* tau, double* G, int vkind,
                                   uint8_t* slices, int* exps, uint8_t* sm, uint32_t tmem,
                                   unsigned* err, bool t_transposed) {
  using namespace oz;
  constexpr size_t ob = operand_bytes();
  uint8_t* X1 = slices + kOzX * ob;
  uint8_t* XV = slices + kOzV * ob;
  uint8_t* XS = slices + kOzS * ob;
  // Z (FP64, ld kK) waits in X1's last 4 chunks until X1 is sliced
  double* Zs = reinterpret_cast<double*>(X1 + 12 * (size_t)kAChunkBytes);
  static_assert(12 * kAChunkBytes + kK * kK * 8 == 2 * operand_bytes(), "Z scratch");
  const int kv = vkind == kVUnitLower ? kUnitLower : vkind == kVUpper ? kUpperIncl : kDense;
  // 1. V^T (scratch) and V from a shared-memory copy of the tile
  {
    double* sV = reinterpret_cast<double*>(sm);
    int* sE = reinterpret_cast<int*>(sm + kLdT * kK * 8);
    stage_tile(sV, V);
    const int kt = vkind == kVUnitLower ? kUnitUpper : vkind == kVUpper ? kLowerIncl : kDense;
    slice_left(StagedAcc{sV, kLdT, 1, kt}, XS, exps + kOzS * kK, sE);
    slice_left(StagedAcc{sV, 1, kLdT, kv}, XV, exps + kOzV * kK, sE);
  }
  // 2. G = V^T V on the tensor cores, by 64-column blocks, into G (global)
  {
    Ctx c;
    ctx_init(c, sm, tmem, err);
    for (int cb = 0; cb < kK / kN; cb++) {
      prefetch(c, XS);
      stage_y(c, V + (size_t)cb * kN * kK, kK, vkind == kVDense ? -1 : cb * kN, vkind == kVUpper);
      if (!product(c, XS, (cb + 1 < kK / kN) ? XS : nullptr, exps + kOzS * kK, kEpiStore,
                   G + (size_t)cb * kN * kK, kK, nullptr, 0))
        return false;
    }
    ctx_release(c);
  }
  __threadfence_block();
  // 3. T in shared memory
  double* sG = reinterpret_cast<double*>(sm);
  double* sT = sG + kK * (kK - 1) / 2;
  int* sE = reinterpret_cast<int*>(sT + kK * (kK + 1) / 2);
  double* sX = reinterpret_cast<double*>(sE + kK);
  static_assert((kK * (kK - 1) / 2 + kK * (kK + 1) / 2) * 8 + kK * 4 + 64 * kLdX * 8 <= kSmemBytes,
                "T recurrence scratch");
  // a warp packs 16 columns, four columns' loads in flight
  for (int c0 = threadIdx.x >> 5; c0 < kK; c0 += 4 * kWarps) {
    double v[4][kK / 32];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int q = 0; q < kK / 32; q++) {
        const int c = c0 + i * kWarps, r = 32 * q + (threadIdx.x & 31);
        v[i][q] = r < c ? __ldcg(G + r + (size_t)c * kK) : 0.0;
      }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int q = 0; q < kK / 32; q++) {
        const int c = c0 + i * kWarps, r = 32 * q + (threadIdx.x & 31);
        if (r < c) sG[c * (c - 1) / 2 + r] = v[i][q];
      }
  }
  __syncthreads();
  t_recurrence(sG, sT, sX, tau);
  // 4. M to G (global, its last use of G was above) and sliced with its own
  //    row exponents into the scratch slot (V^T is not needed any more)
  {
    const PackedTAcc m{sT, t_transposed};
    for (int e = threadIdx.x; e < kK * kK; e += kThreads) stg_cg(G + e, m(e % kK, e / kK));
    slice_left(m, XS, exps + kOzS * kK, sE);
  }
  // 5. Z = M V^T on the tensor cores, into Zs
  {
    Ctx c;
    ctx_init(c, sm, tmem, err);
    for (int cb = 0; cb < kK / kN; cb++) {
      prefetch(c, XS);
      stage_yt(c, V, cb * kN, kv);
      if (!product(c, XS, (cb + 1 < kK / kN) ? XS : nullptr, exps + kOzS * kK, kEpiStore,
                   Zs + (size_t)cb * kN * kK, kK, nullptr, 0))
        return false;
    }
    ctx_release(c);
  }
  __threadfence_block();
  // 6. row exponents of X1 = [Z | M] over both halves
  //    (threads 0..127 scan Z's rows, threads 128..255 M's)
  static_assert(kThreads == 2 * kK, "one thread per row and half");
  int* sE1 = reinterpret_cast<int*>(sm);
  if (threadIdx.x < kK) sE1[threadIdx.x] = 0;
  __syncthreads();
  {
    const int r = threadIdx.x % kK;
    const double* src = threadIdx.x < kK ? Zs : G;
    int e = 0;
#pragma unroll 8
    for (int k = 0; k < kK; k++) e = max(e, biased_exp(__ldcg(src + r + (size_t)k * kK)));
    atomicMax(sE1 + r, e);
  }
  __syncthreads();
  if (threadIdx.x < kK) exps[kOzX * kK + threadIdx.x] = sE1[threadIdx.x];
  // 7. X1: Z into chunks 0-7 (all of Zs read before chunks 12-15 are written),
  //    then M into chunks 8-15
  slice_cols(GlobalAcc{Zs}, X1, sE1, kK);
  slice_cols(GlobalAcc{G}, X1 + (size_t)kChunks * kAChunkBytes, sE1, kK);
  return true;
}

// `chunks` 64-column blocks of the update, one after the other.  Ctop: A1 block
// (SSRFB) or nullptr (LARFB); Cbot: A2 block (SSRFB) or the C block (LARFB); ld
// NB.  Returns false on a device time-out (error word already set).  G: t-groups
// of the products (8: FP64-level; 4: the reduced form, see oz::product).
template <int G = oz::kGroups>
inline __device__ bool task_ozapply(oz::Ctx& c, const uint8_t* slices, const int* exps, double* Ctop,
                                    double* Cbot, int chunks) {
  using namespace oz;
  constexpr size_t ob = operand_bytes();
  const uint8_t* X1 = slices + kOzX * ob;
  const uint8_t* XV = slices + kOzV * ob;
  prefetch<G>(c, X1);
  for (int cc = 0; cc < chunks; cc++) {
    // the right operand [C_bot; C_top]: C_bot staged, C_top loaded after chunk 7;
    // column exponents over both
    stage_y(c, Cbot, kK, -1, false, Ctop);
    if (!product<G>(c, X1, XV, exps + kOzX * kK, kEpiToYSubTop, nullptr, 0, Ctop, kK, Ctop ? 2 * kChunks : kChunks,
                    Ctop))
      return false;
    if (!product<G>(c, XV, cc + 1 < chunks ? X1 : nullptr, exps + kOzV * kK, kEpiSubInto, Cbot, kK, nullptr, 0))
      return false;
    Cbot += kN * kK;
    if (Ctop) Ctop += kN * kK;
  }
  ctx_release(c);
  return true;
}

}  // namespace hqr
