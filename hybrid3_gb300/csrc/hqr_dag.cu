// hqr_dag.cu -- host side of the device DAG: geometry, workspace and launches
// of the persistent executor for the factorization and the Q^T application.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "hqr_dag.cuh"
#include "hqr_internal.h"

namespace hqr {

// Task ids of the plain FP64 factorization with nc column blocks per update
// tile and no trailing-update tasks, and the scratch that hqr_geqrf_noalloc
// carves for n_ids ids.
static size_t coarse_task_ids(const Geometry& g, int nc) {
  return (size_t)g.steps * g.MT * (g.NB / g.w) + (size_t)g.steps * g.NT * g.MT * nc;
}
ExternalLayout external_layout(const Geometry& g, size_t n_ids) {
  ExternalLayout l{};
  auto carve = [&](size_t b) {
    const size_t at = l.bytes;
    l.bytes += (b + 255) & ~size_t(255);
    return at;
  };
  l.T = carve((size_t)g.M * g.N * sizeof(double));
  l.cnt = carve(n_ids * sizeof(int));
  l.qhi = carve(n_ids * sizeof(int));
  l.qlo = carve(n_ids * sizeof(int));
  l.ctl = carve(kExternalCtlBytes);
  l.stats = carve(kExternalStatsBytes);
  return l;
}

int make_geometry(long M, long N, int NB, int IB, Geometry* g, size_t smem_limit) {
  if (NB < 16 || NB > kMaxNB || NB % 16 != 0) return HQR_ERR_UNSUPPORTED;
  if (M <= 0 || N <= 0 || M % NB != 0 || N % NB != 0) return HQR_ERR_INVALID;
  if (IB <= 0 || IB > NB) return HQR_ERR_INVALID;
  g->M = M;
  g->N = N;
  g->NB = NB;
  g->IB = IB;
  g->MT = (int)(M / NB);
  g->NT = (int)(N / NB);
  g->steps = std::min(g->MT, g->NT);
  // inner block: the largest divisor of NB that is <= min(IB, 32) and a multiple of 8
  int w = std::min(IB, kMaxW);
  w -= w % 8;
  while (w > 8 && NB % w != 0) w -= 8;
  if (w < 8) w = 8;
  g->w = w;
  // column block of the update tasks: the widest multiple of 8 dividing NB,
  // at most 64 and at most NB*CB*8 <= 64 KiB, whose shared-memory plan fits
  const size_t smem_cap = smem_limit ? smem_limit : 227 * 1024 - 256;   // room for static shared memory
  int cb = (8192 / NB) > 64 ? 64 : 8192 / NB;
  if (cb > NB) cb = NB;
  cb -= cb % 8;
  for (; cb >= 8; cb -= 8) {
    if (NB % cb != 0) continue;
    TileShape sh{NB, w, cb, NB >= 512 ? 64 : kRC, cb};
    if ((size_t)SmemPlan::make(sh).total * sizeof(double) <= smem_cap) break;
  }
  if (cb < 8) return HQR_ERR_UNSUPPORTED;
  g->CB = cb;
  g->NC = NB / cb;
  TileShape sh{NB, w, cb, NB >= 512 ? 64 : kRC, cb};
  SmemPlan sp = SmemPlan::make(sh);
  g->smem_bytes = (size_t)sp.total * sizeof(double);
  if (g->smem_bytes > smem_cap) return HQR_ERR_UNSUPPORTED;
  if ((long long)g->steps * g->MT * (g->NB / g->w + 1) + (long long)g->steps * g->NT * g->MT * g->NC >
      0x3fffffffLL)
    return HQR_ERR_UNSUPPORTED;
  return HQR_OK;
}

static TileShape shape_of(const Geometry& g) {
  return TileShape{g.NB, g.w, g.CB, g.NB >= 512 ? 64 : kRC, g.CB};
}

int dag_workspace_reserve(DagWorkspace* ws, size_t n_ids) {
  if (ws->cap_ids >= n_ids && ws->ctl) return HQR_OK;
  dag_workspace_free(ws);
  if (cudaMalloc(&ws->cnt, n_ids * sizeof(int)) != cudaSuccess) return HQR_ERR_NOMEM;
  if (cudaMalloc(&ws->qhi, n_ids * sizeof(int)) != cudaSuccess) return HQR_ERR_NOMEM;
  if (cudaMalloc(&ws->qlo, n_ids * sizeof(int)) != cudaSuccess) return HQR_ERR_NOMEM;
  if (cudaMalloc(&ws->ctl, kCtlWords * sizeof(unsigned)) != cudaSuccess) return HQR_ERR_NOMEM;
  if (cudaMalloc(&ws->stats, 2 * kNumStats * sizeof(unsigned long long)) != cudaSuccess)
    return HQR_ERR_NOMEM;
  if (cudaMemset(ws->ctl, 0, kCtlWords * sizeof(unsigned)) != cudaSuccess) return HQR_ERR_CUDA;
  ws->cap_ids = n_ids;
  return HQR_OK;
}

void dag_workspace_free(DagWorkspace* ws) {
  if (ws->cnt) cudaFree(ws->cnt);
  if (ws->qhi) cudaFree(ws->qhi);
  if (ws->qlo) cudaFree(ws->qlo);
  if (ws->ctl) cudaFree(ws->ctl);
  if (ws->stats) cudaFree(ws->stats);
  *ws = DagWorkspace{};
}

// Per-device caches: cudaFuncSetAttribute applies to the current device only,
// and the SM count is a property of the device, so both are kept per device
// ordinal (devices beyond kCacheDevices are simply not cached).
constexpr int kCacheDevices = 64;
static int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

int dag_sm_count() {
  static int n[kCacheDevices] = {};
  const int dev = current_device();
  const bool cached = dev >= 0 && dev < kCacheDevices;
  if (cached && n[dev] > 0) return n[dev];
  int v = 0;
  cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev < 0 ? 0 : dev);
  if (v <= 0) v = 1;
  if (cached) n[dev] = v;
  return v;
}

// The largest dynamic shared memory a kernel has been opted in to, per device
// (one record a kernel: a smaller opt-in would take a larger one back).
struct SmemOptIn {
  std::mutex mu;
  size_t bytes[kCacheDevices] = {};
};
// Opt `kernel` in to smem bytes of dynamic shared memory on the current device
// (once per device and size); extra(): further attribute calls made with it.
template <class Kernel, class Extra>
static cudaError_t opt_in(SmemOptIn& o, Kernel kernel, size_t smem, Extra extra) {
  const int dev = current_device();
  std::lock_guard<std::mutex> lk(o.mu);
  if (dev >= 0 && dev < kCacheDevices && smem <= o.bytes[dev]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = extra();
  if (e == cudaSuccess && dev >= 0 && dev < kCacheDevices) o.bytes[dev] = smem;
  return e;
}
template <class Kernel>
static cudaError_t opt_in(SmemOptIn& o, Kernel kernel, size_t smem) {
  return opt_in(o, kernel, smem, [] { return cudaSuccess; });
}

static size_t dag_smem_bytes(const Geometry& g, bool oz) {
  size_t b = g.smem_bytes;
  if (oz) b = std::max(b, (size_t)oz::kSmemBytes);
  return b;
}

template <bool OZ, int G = 8, bool P32 = false>
static int launch_exec(const DagParams& p, const Geometry& g, cudaStream_t stream) {
  static SmemOptIn opted;
  const size_t smem = dag_smem_bytes(g, OZ);
  {
    const cudaError_t e = opt_in(opted, dag_exec_kernel<OZ, false, G, P32>, smem);
    if (e != cudaSuccess) return record_cuda_error(e, "cudaFuncSetAttribute(dag_exec_kernel)");
  }
  const int grid = std::min(dag_sm_count(), std::max(1, p.n_tasks));
  dag_exec_kernel<OZ, false, G, P32><<<grid, kThreads, smem, stream>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return record_cuda_error(e, "dag_exec_kernel launch");
  return HQR_OK;
}

// reserve: ids to reserve the scheduler's tables for, at least this run's.
static int run_dag(DagParams& p, DagWorkspace* ws, const Geometry& g, cudaStream_t stream, long long reserve = 0) {
  p.sp = SmemPlan::make(p.sh);
  p.n_ids = id_end(p);
  int rc = dag_workspace_reserve(ws, (size_t)std::max((long long)p.n_ids, reserve));
  if (rc != HQR_OK) return rc;
  p.cnt = ws->cnt;
  p.qhi = ws->qhi;
  p.qlo = ws->qlo;
  p.ctl = ws->ctl;
  p.stats = ws->stats;
  // control words: queue heads/tails and the done counter start at zero; the
  // error word is kept (cleared by dag_status) so a failure is never lost.
  cudaError_t e0 = cudaMemsetAsync(ws->ctl, 0, kErr * sizeof(unsigned), stream);
  if (e0 == cudaSuccess)
    e0 = cudaMemsetAsync(ws->stats, 0, 2 * kNumStats * sizeof(unsigned long long), stream);
  if (e0 != cudaSuccess) return record_cuda_error(e0, "DAG workspace reset");
  const int blocks = (p.n_ids + 255) / 256;
  dag_init_kernel<<<blocks, 256, 0, stream>>>(p);
  dag_seed_kernel<<<blocks, 256, 0, stream>>>(p);
  if (!p.oz) return launch_exec<false>(p, g, stream);
  if (p.oz_groups == 8) return launch_exec<true, 8>(p, g, stream);
  return p.oz_p32 ? launch_exec<true, 4, true>(p, g, stream) : launch_exec<true, 4>(p, g, stream);
}

// The steps from which on a flat-tree factorization cuts its panel blocks'
// trailing updates into tasks of their own: those whose panel chain, not their
// update work, sets the pace, that is with at most `tiles` update tiles ((NT -
// i - 1) (MT - i - 1)) left.  Before them the additional tasks cost more than
// the shorter chain gains.  Measured, against whole panel blocks: FP64 n =
// 2048, NB 256: factorization 73 -> 38 ms; n = 4096: 155 -> 118 ms; split n =
// 3072 (against blocks that released their dependents in phases): QR + Q 35.7
// -> 28.4 ms; split n = 16384 unchanged.  FP32 panels: fine_tiles_fp32.
//
// Such a task takes a part of a block's w columns: the chain through a tile is
// its panel blocks and the first part after each, and a part of 8 / 16 / 32
// columns takes 52 / 84 / 156 us at tile order 256 (8 / 16: 13 / 22 us at 128).
// Parts of 8 cost a third more work than blocks of 32, so they are taken where
// there are at most two panel tiles to an SM (factorization, ms, parts of 8 /
// 16 / whole blocks: FP64 n = 2048, NB 256: 25.7 / 27.2 / 31.4, n = 4096: 112.2
// / 113.4 / 116.9; 1000 x 615, NB 96, with its solve: 6.53 / 6.87 / 7.59; split
// n = 3072: 21.4 / - / 22.2; but 594 panel tiles: FP64 38400 x 1024, NB 256:
// 118 / 112.2 / 111.8, split 19200 x 512: 18.2 / - / 14.6), and FP64 parts of
// 16 beyond that.
//
// FP32 panel blocks take half the time and are latency, not work, and the
// scheduler hands out about two of the small tasks a microsecond.  They are cut
// by what the whole factorization is: `load` is its work on every SM (an update
// 50 us, a panel tile 1 ms) over its chain (a tile down a column 105 us, a step
// 660 us).  Small loads: in every step; matrices that are not tall gain somewhat
// longer, and up to a load of 1 in their last steps (300 tiles left); none
// beyond.  Factorization, ms, none / from 300 tiles on / all steps, in tiles:
//   load to 0.45: 4 x 4 3.49 / 2.91 / 2.92, 30 x 6 7.88 / 6.01 / 5.98, 100 x 3
//     12.5 / 7.5 / 7.5, 256 x 4 29.5 / 29.7 / 19.5, 1000 x 2 103 / 105 / 54, 64 x 8
//     13.2 / 13.0 / 11.1, 40 x 40 39.3 / 37.3 / 36.0, 12 x 80 11.7 / 11.1 / 9.8
//   0.52 .. 1: 32 x 64 31.9 / 31.1 / 28.3, 48 x 48 47.7 / 45.7 / 47.6, 64 x 64 73.7
//     / 72.4 / 82.8; tall 400 x 8 48.5 / 48.8 / 56.5, 128 x 16 28.5 / 29.0 / 36.9
//   above 1: 256 x 32 106 / 109 / 155, 256 x 64 293 / 296 / 396
struct FineSteps {
  int from = 0, sub = 1;
  long long ids = 0, tasks = 0;
};
constexpr long long kFineTilesSplit = 6000, kFineTilesFp64 = 600;
static long long fine_tiles_fp32(const Geometry& g) {   // -1: no such steps
  double work = 0.0;
  for (int i = 0; i < g.steps; i++) work += (g.MT - i) * (1000.0 + 50.0 * (g.NT - 1 - i));
  const double load = work / (dag_sm_count() * (105.0 * g.MT + 660.0 * g.steps));
  const bool tall = g.MT > 3 * g.steps;
  return load <= (tall ? 0.45 : 0.53) ? 0x7fffffffLL : load <= 1.0 && !tall ? 300 : -1;
}
static FineSteps fine_steps(const Geometry& g, bool split, bool fp32 = false, bool parts = true) {
  FineSteps f;
  const long long nblk = g.NB / g.w, tiles = fp32 ? fine_tiles_fp32(g) : split ? kFineTilesSplit : kFineTilesFp64;
  while (f.from < g.steps && (long long)(g.NT - f.from - 1) * (g.MT - f.from - 1) > tiles) f.from++;
  if (nblk < 2) return f;
  long long panels = 0;
  for (int i = f.from; i < g.steps; i++) panels += g.MT - i;
  const int part = panels <= 2LL * dag_sm_count() && !fp32 ? 8 : split ? g.w : 16;
  if (parts && g.w % part == 0) f.sub = g.w / part;
  f.ids = (long long)(g.steps - f.from) * g.MT * nblk * nblk * f.sub;
  for (int i = f.from; i < g.steps; i++) f.tasks += (g.MT - i) * nblk * (nblk - 1) / 2 * f.sub;
  if ((long long)coarse_task_ids(g, split ? 2 : g.NC) + f.ids > 0x3fffffffLL) {
    if (f.sub > 1) return fine_steps(g, split, fp32, false);
    f.ids = f.tasks = 0;
  }
  return f;
}

// Columns per FP64 update task: the tile's nominal block (g.CB), or fewer
// where the longest chain of updates (`path` tasks) sets the pace rather than
// all `tiles` of them (`cols` columns of data each) on every SM.  A task of cb
// columns takes cb + c0 column times: c0 is 12 us and 6 us an inner block, in
// columns of NB^2 / 1700 us each, and at least 4; 20 for tiles of order 512,
// whose V goes through shared memory in chunks of 64 rows (us a link of Q^T C's
// chain, CB 64 / 32 / 16 / 8: NB 32, w 8 - / 40.9 / 35.5 / 35.8, w 32 - / 40.2 /
// 29.7 / 23.9; NB 64, w 16 175 / 98 / 64 / 51; NB 128 - / 310 / 169 / 103; NB 512
// - / - / 1241 / 969).
//
// Q generation and the applications (`apply`) start with few tiles or end with
// few, so that chain and work overlap in part only: three tenths of the smaller
// count too, a gain has to be 8 %, and tiles of order 512 stay at their nominal
// 16 columns unless the work stays below nine tenths of the chain and the tasks
// of one of its links (a tile, on all CT tile columns of C) are one wave (ms,
// nominal / 8 columns, MT x NT on CT: 192 tasks a link, 1 x 1 on 3 1.65 / 2.41,
// 2 x 1 on 3 4.40 / 6.75; 128 a link, 3 x 2 on 2 9.91 / 8.96, 3 x 3 on 2 11.45 /
// 10.13).  A factorization's chain has its panel blocks besides, and its tasks are
// narrowed as if chain and work overlapped.  (ms, nominal / the narrower block
// that the plain maximum takes: Q, 4 x 4 tiles of order 512 20.0 / 26.6; 20 x 20
// of 32 1.69 / 1.89; 14 x 14 of 32 1.18 / 1.33, 1.04 with 16 columns.)  Tiles of
// order 16 have nothing to cut (factorization of 20 x 20: 1.89 ms, 2.06 cut).
static int update_columns(const Geometry& g, long long tiles, long long path, int cols, int CT) {
  const bool apply = CT > 0;   // (0: a factorization)
  const double c0 =
      g.NB >= 512 ? 20.0 : std::max(4.0, 1700.0 * (12.0 + 6.0 * (g.NB / g.w)) / ((double)g.NB * g.NB));
  int best = g.CB;
  double t_best = 0.0;
  for (int cb = g.CB; cb >= (g.NB < 32 ? g.CB : 8); cb -= 8) {
    const long long tasks = tiles * ((cols + cb - 1) / cb);
    if (g.CB % cb != 0 || tasks > 0x0fffffffLL) continue;
    const double chain = (double)path, work = (double)tasks / dag_sm_count();
    const long long link = (long long)CT * ((cols + cb - 1) / cb);
    if (apply && g.NB >= 512 && cb < g.CB && (work > 0.9 * chain || link > dag_sm_count())) continue;
    const double t = (cb + c0) * (std::max(chain, work) + (apply ? 0.3 : 0.0) * std::min(chain, work));
    if (cb == g.CB || t < (apply ? 0.92 : 0.95) * t_best) {
      best = cb;
      t_best = t;
    }
  }
  return best;
}
static void set_columns(DagParams& p, const Geometry& g, int cb, int cols) {
  p.sh = shape_of(g);
  if (p.oz) return;
  p.sh.CB = cb;
  if (p.mode != kModeFactor) p.sh.PB = cb;
  p.NC = (cols + cb - 1) / cb;
  p.count_every = g.CB / cb;
}
// The same for C <- Q^T C or Q C on CT tile columns (ccols > 0: that many
// columns hold data; in a single tile column only their blocks are tasks).
static void set_apply_columns(DagParams& p, const Geometry& g, long long tiles, long long path, int CT,
                              long long ccols) {
  const int cols = CT == 1 && ccols > 0 && ccols < g.NB ? (int)ccols : g.NB;
  set_columns(p, g, update_columns(g, tiles, path, cols, CT), cols);
}

// The FP64 factorization's update columns and fine steps.  The allocation-free
// entry point runs the same tasks, hence with the same rounding: where its
// scratch holds the plain tasks' ids but not these, both take the plain ones.
struct FactorTasks {
  int cb;
  FineSteps fine;
  size_t ids;
};
static FactorTasks factor_tasks(const Geometry& g) {
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)(g.NT - 1 - i) * (g.MT - i);
  FactorTasks f{update_columns(g, tiles, g.MT + g.steps, g.NB, 0), fine_steps(g, false), 0};
  f.ids = coarse_task_ids(g, g.NB / f.cb) + (size_t)f.fine.ids;
  auto fits = [&](size_t ids) { return external_layout(g, ids).bytes <= kNoAllocScratchBytes; };
  if (fits(coarse_task_ids(g, g.NC))) {
    if (f.fine.sub > 1 && !fits(f.ids)) {
      f.fine = fine_steps(g, false, false, false);
      f.ids = coarse_task_ids(g, g.NB / f.cb) + (size_t)f.fine.ids;
    }
    if (!fits(f.ids))
      f = FactorTasks{g.CB, FineSteps{}, coarse_task_ids(g, g.NC)};
  }
  return f;
}

// 64-column chunks per split update task, run one after the other.  Two (a
// whole 128-column tile) halve the number of update tasks and with them the
// scheduling round trips (a queue claim and the dependents' releases, about 6
// us per task).  One, where the longest chain of whole-tile updates (`path`
// tasks) takes longer than all `tiles` of them on every SM: the chain's time
// halves (Q^T C and Q C, n = 8192, 512 columns: 21.5 -> 13.3 ms together, now
// 11.4).  C with data in one chunk only (ccols) has nothing to cut.
static int oz_chunks(long long tiles, long long path, long long ccols = 0) {
  return (ccols > 0 && ccols <= oz::kN) || tiles >= path * dag_sm_count() ? 2 : 1;
}
static void set_oz(DagParams& p, const Geometry& g, const OzWorkspace* oz, int chunks) {
  if (oz && oz->slices) {
    p.oz = 1;
    p.oz_groups = oz->groups;
    p.oz_p32 = oz->fp32_panels;
    p.oz_cpt = chunks;
    p.NC = g.NB / oz::kN / p.oz_cpt;
    p.slices = oz->slices;
    p.sexp = oz->sexp;
  } else {
    p.oz = 0;
    p.NC = g.NC;
  }
}

// The most task ids that Q generation or an application to up to NT tile columns
// takes on the plan of factorization f (`chain` tasks down a column).  The
// factorization reserves the scheduler's tables for them as well: a later call
// on the plan then allocates nothing, so that it can be captured into a graph,
// keeps the addresses that an earlier graph holds, and loses no status that has
// not been read yet.  Their tasks can be narrower than the factorization's.
static long long plan_apply_ids(const DagParams& f, const Geometry& g, int chain) {
  long long below = 0, q_tiles = 0;   // tiles of one column; of Q generation
  for (int i = 0; i < g.steps; i++) {
    below += g.MT - i;
    q_tiles += (long long)(g.NT - i) * (g.MT - i);
  }
  const long long path = chain + g.steps;
  auto ids = [&](long long tiles, int CT) {
    long long nc = f.oz ? g.NB / oz::kN / oz_chunks(tiles, path) : g.NB / update_columns(g, tiles, path, g.NB, CT);
    if (!f.oz && CT == 1) nc = g.NB / 8;   // (few right-hand sides in one tile column: any width)
    return g.steps * ((long long)g.MT + f.dmax + ((long long)g.MT + f.dmax) * CT * nc);
  };
  long long most = g.M == g.N ? ids(q_tiles, g.NT) : 0;
  for (int CT = 1; CT <= g.NT; CT++) most = std::max(most, ids(CT * below, CT));
  return most;
}

// Domains and merge storage of a domain tree (tw null or tw->S == 0: flat).
static void set_tree(DagParams& p, const Geometry& g, const TreeWorkspace* tw) {
  if (!tw || tw->S <= 0 || tw->S >= g.MT) {
    p.tree = 0;
    p.dmax = 0;
    return;
  }
  p.tree = tw->S;
  p.dmax = (g.MT + tw->S - 1) / tw->S;
  p.T2 = tw->T2;
  p.TAU2 = tw->TAU2;
  p.slices2 = tw->slices2;
  p.sexp2 = tw->sexp2;
}
static long long merges_of_step(const DagParams& p, int i) { return n_domains(p, i) - 1; }

int launch_factor(const Geometry& g, DagWorkspace* ws, double* dA, double* dT, double* dTAU,
                  long long timeout_ns, cudaStream_t stream, const OzWorkspace* ozw,
                  const TreeWorkspace* tw) {
  DagParams p{};
  p.mode = kModeFactor;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = g.NT;
  p.steps = g.steps;
  p.J = g.NT;
  p.A = dA;
  p.T = dT;
  p.TAU = dTAU;
  p.C = dA;
  p.timeout_ns = timeout_ns;
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)(g.NT - 1 - i) * (g.MT - i);
  const int chain = tw && tw->S > 0 && tw->S < g.MT ? tw->S + (g.MT + tw->S - 1) / tw->S : g.MT;   // tasks down a column
  set_oz(p, g, ozw, oz_chunks(tiles, chain + g.steps));
  p.prep = p.oz;
  p.nblk = g.NB / g.w;
  set_tree(p, g, tw);
  FineSteps fine;
  int cb = g.CB;
  if (p.tree == 0 && p.oz) fine = fine_steps(g, true, p.oz_p32 != 0);
  if (p.tree == 0 && !p.oz) {
    const FactorTasks f = factor_tasks(g);
    fine = f.fine;
    cb = f.cb;
  }
  set_columns(p, g, cb, g.NB);
  p.fine_from = fine.from;
  p.fine_ids = (int)fine.ids;
  p.fine_sub = fine.sub;
  // tasks: per step i, nblk inner blocks of each of the MT-i panel tiles [+ one
  // OZPREP per panel tile] + NC*(NT-1-i)*(MT-i) updates; a tree adds per merge
  // nblk blocks [+ one OZPREP] + NC*(NT-1-i) merge updates; a fine step nblk
  // (nblk - 1) / 2 trailing updates per panel tile
  long long n = fine.tasks;
  for (int i = 0; i < g.steps; i++) {
    const long long m = merges_of_step(p, i);
    n += (long long)(g.MT - i) * (p.nblk + (p.prep ? 1 : 0)) + (long long)p.NC * (g.NT - 1 - i) * (g.MT - i);
    n += m * (p.nblk + (p.prep ? 1 : 0)) + m * p.NC * (g.NT - 1 - i);
  }
  p.n_tasks = (int)n;
  return run_dag(p, ws, g, stream, plan_apply_ids(p, g, chain));
}

int launch_apply_qt(const Geometry& g, DagWorkspace* ws, const double* dA, double* dT,
                    const double* dTAU, double* dC, int CT, bool rebuild_t, long long timeout_ns,
                    cudaStream_t stream, const OzWorkspace* ozw, long long ccols) {
  if (CT <= 0) return HQR_ERR_INVALID;
  DagParams p{};
  p.mode = kModeApplyQt;
  p.c_cols = ccols;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = CT;
  p.steps = g.steps;
  p.J = CT;
  p.A = const_cast<double*>(dA);
  p.T = dT;
  p.TAU = const_cast<double*>(dTAU);
  p.C = dC;
  p.timeout_ns = timeout_ns;
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)CT * (g.MT - i);
  set_oz(p, g, ozw, oz_chunks(tiles, g.MT + g.steps, ccols));
  set_apply_columns(p, g, tiles, g.MT + g.steps, CT, ccols);
  p.prep = 0;
  p.nblk = 1;
  // rebuild_t: panel tasks rebuild each panel tile's T (FP64: its diagonal
  // blocks) or prepared operands (split) from V and TAU; else the updates use
  // those the factorization left in dT / the slice store
  p.skip_panels = rebuild_t ? 0 : 1;
  long long n = 0;
  for (int i = 0; i < g.steps; i++) n += (rebuild_t ? (g.MT - i) : 0) + (long long)p.NC * CT * (g.MT - i);
  p.n_tasks = (int)n;
  return run_dag(p, ws, g, stream);
}

int launch_apply_qt_tree(const Geometry& g, DagWorkspace* ws, const double* dA, double* dT,
                         const double* dTAU, double* dC, int CT, long long timeout_ns, cudaStream_t stream,
                         const OzWorkspace* ozw, const TreeWorkspace* tw) {
  if (CT <= 0 || !tw || tw->S <= 0) return HQR_ERR_INVALID;
  DagParams p{};
  p.mode = kModeApplyQt;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = CT;
  p.steps = g.steps;
  p.J = CT;
  p.A = const_cast<double*>(dA);
  p.T = dT;
  p.TAU = const_cast<double*>(dTAU);
  p.C = dC;
  p.timeout_ns = timeout_ns;
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)CT * (g.MT - i);
  set_oz(p, g, ozw, oz_chunks(tiles, tw->S + (g.MT + tw->S - 1) / tw->S + g.steps));
  set_apply_columns(p, g, tiles, tw->S + (g.MT + tw->S - 1) / tw->S + g.steps, CT, 0);
  p.prep = 0;
  p.nblk = 1;
  p.skip_panels = 1;   // the T factors / slices of the factorization on this plan
  set_tree(p, g, tw);
  long long n = 0;
  for (int i = 0; i < g.steps; i++) n += (long long)p.NC * CT * ((g.MT - i) + merges_of_step(p, i));
  p.n_tasks = (int)n;
  return run_dag(p, ws, g, stream);
}

int launch_build_q(const Geometry& g, DagWorkspace* ws, const double* dA, double* dT, const double* dTAU,
                   double* dQ, bool rebuild_t, long long timeout_ns, cudaStream_t stream, const OzWorkspace* ozw) {
  if (g.M != g.N) return HQR_ERR_INVALID;
  DagParams p{};
  p.mode = kModeBuildQ;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = g.NT;
  p.steps = g.steps;
  p.J = g.NT;
  p.A = const_cast<double*>(dA);
  p.T = dT;
  p.TAU = const_cast<double*>(dTAU);
  p.C = dQ;
  p.timeout_ns = timeout_ns;
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)(g.NT - i) * (g.MT - i);
  set_oz(p, g, ozw, oz_chunks(tiles, g.MT + g.steps));
  set_columns(p, g, update_columns(g, tiles, g.MT + g.steps, g.NB, g.NT), g.NB);
  p.prep = 0;
  p.nblk = 1;
  p.skip_panels = rebuild_t ? 0 : 1;   // as in launch_apply_qt (split: T from its own slot)
  // per step i: MT - i panel tasks (when rebuilding) and NC (NT - i) (MT - i) updates
  long long n = 0;
  for (int i = 0; i < g.steps; i++)
    n += (rebuild_t ? (g.MT - i) : 0) + (long long)p.NC * (g.NT - i) * (g.MT - i);
  p.n_tasks = (int)n;
  return run_dag(p, ws, g, stream);
}

int launch_apply_q(const Geometry& g, DagWorkspace* ws, const double* dA, double* dT, const double* dTAU,
                   double* dC, int CT, bool rebuild_t, long long timeout_ns, cudaStream_t stream,
                   const OzWorkspace* ozw, long long ccols) {
  if (CT <= 0) return HQR_ERR_INVALID;
  DagParams p{};
  p.mode = kModeApplyQ;
  p.c_cols = ccols;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = CT;
  p.steps = g.steps;
  p.J = CT;
  p.A = const_cast<double*>(dA);
  p.T = dT;
  p.TAU = const_cast<double*>(dTAU);
  p.C = dC;
  p.timeout_ns = timeout_ns;
  long long tiles = 0;
  for (int i = 0; i < g.steps; i++) tiles += (long long)CT * (g.MT - i);
  set_oz(p, g, ozw, oz_chunks(tiles, g.MT + g.steps, ccols));
  set_apply_columns(p, g, tiles, g.MT + g.steps, CT, ccols);
  p.prep = 0;
  p.nblk = 1;
  p.skip_panels = rebuild_t ? 0 : 1;
  long long n = 0;
  for (int i = 0; i < g.steps; i++) n += (rebuild_t ? (g.MT - i) : 0) + (long long)p.NC * CT * (g.MT - i);
  p.n_tasks = (int)n;
  return run_dag(p, ws, g, stream);
}

// --- batches of independent matrices (FP64) ---------------------------------------
size_t mat_desc_bytes() { return sizeof(MatDesc); }

// The per-matrix fields of a batch launch (factorization, or C <- Q^T C with
// the T factors the factorization left), plus that matrix's id / task counts.
// C <- Q^T C covers the first nrhs columns of C: ceil(nrhs / NB) tile
// columns; fewer than NB right-hand sides take the narrowest column blocks
// (a multiple of 8 dividing NB, at most the factorization's) that hold them.
static DagParams batch_matrix_params(bool apply, const Geometry& g, int nrhs) {
  DagParams p{};
  p.mode = apply ? kModeApplyQt : kModeFactor;
  p.MT = g.MT;
  p.NT = g.NT;
  p.NC = g.NC;
  p.steps = g.steps;
  p.CT = g.NT;
  p.nblk = g.NB / g.w;
  p.sh = shape_of(g);
  if (apply) {
    p.skip_panels = 1;
    p.nblk = 1;
    p.CT = (nrhs + g.NB - 1) / g.NB;
    if (nrhs < g.NB) {
      int cb = (nrhs + 7) / 8 * 8;
      while (cb < g.CB && g.NB % cb != 0) cb += 8;
      if (cb > g.CB) cb = g.CB;
      p.sh.CB = p.sh.PB = cb;
      p.NC = (nrhs + cb - 1) / cb;
    }
  }
  p.J = p.CT;
  p.sp = SmemPlan::make(p.sh);
  return p;
}
static long long batch_matrix_tasks(bool apply, const DagParams& p) {
  long long n = 0;
  for (int i = 0; i < p.steps; i++) {
    if (apply)
      n += (long long)p.NC * p.CT * (p.MT - i);
    else
      n += (long long)(p.MT - i) * p.nblk + (long long)p.NC * (p.NT - 1 - i) * (p.MT - i);
  }
  return n;
}

long long batch_ids(bool apply, const Geometry& g, int nrhs) {
  return id_end(batch_matrix_params(apply, g, nrhs));
}

int batch_describe(bool apply, int count, const Geometry* gs, const int* order, double* const* A,
                   double* const* T, double* const* TAU, double* const* C, int nrhs, void* desc, int* n_ids,
                   int* n_tasks) {
  MatDesc* d = static_cast<MatDesc*>(desc);
  long long ids = 0, tasks = 0;
  for (int i = 0; i < count; i++) {
    const int b = order ? order[i] : i;
    const DagParams p = batch_matrix_params(apply, gs[b], nrhs);
    MatDesc m{};
    m.MT = p.MT;
    m.NT = p.NT;
    m.CT = p.CT;
    m.NC = p.NC;
    m.steps = p.steps;
    m.J = p.J;
    m.nblk = p.nblk;
    m.sh = p.sh;
    m.sp = p.sp;
    m.A = A[b];
    m.T = T[b];
    m.TAU = TAU[b];
    m.C = apply ? C[b] : A[b];
    m.id_base = (int)ids;
    ids += id_end(p);
    tasks += batch_matrix_tasks(apply, p);
    if (ids > 0x3fffffffLL) return HQR_ERR_UNSUPPORTED;
    m.id_end = (int)ids;
    d[i] = m;
  }
  *n_ids = (int)ids;
  *n_tasks = (int)tasks;
  return HQR_OK;
}

size_t batch_two_cta_smem() {
  static size_t v = 0;
  if (v == 0) {
    int dev = 0, per_sm = 0;
    cudaFuncAttributes fa{};
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaFuncGetAttributes(&fa, dag_exec_kernel<false, true>);
    // per CTA: the dynamic part, the kernel's static part and 1 KiB the system reserves
    const long long b = (long long)per_sm / 2 - (long long)fa.sharedSizeBytes - 1024;
    v = b > 0 ? (size_t)b : 1;
  }
  return v;
}

int launch_batch(bool apply, int count, const void* d_desc, int n_ids, int n_tasks, size_t smem,
                 int ctas_per_sm, DagWorkspace* ws, long long timeout_ns, cudaStream_t stream) {
  if (count <= 0 || n_tasks <= 0) return HQR_ERR_INVALID;
  DagParams p{};
  p.mode = apply ? kModeApplyQt : kModeFactor;
  p.skip_panels = apply ? 1 : 0;
  p.n_mats = count;
  p.mats = static_cast<const MatDesc*>(d_desc);
  p.n_ids = n_ids;
  p.n_tasks = n_tasks;
  p.timeout_ns = timeout_ns;
  int rc = dag_workspace_reserve(ws, (size_t)n_ids);
  if (rc != HQR_OK) return rc;
  p.cnt = ws->cnt;
  p.qhi = ws->qhi;
  p.qlo = ws->qlo;
  p.ctl = ws->ctl;
  p.stats = ws->stats;
  cudaError_t e = cudaMemsetAsync(ws->ctl, 0, kErr * sizeof(unsigned), stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(ws->stats, 0, 2 * kNumStats * sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return record_cuda_error(e, "DAG workspace reset");
  static SmemOptIn opted;
  int occ = 1;
  e = opt_in(opted, dag_exec_kernel<false, true>, smem, [] {
    return cudaFuncSetAttribute(dag_exec_kernel<false, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
  });
  if (e != cudaSuccess) return record_cuda_error(e, "cudaFuncSetAttribute(dag_exec_kernel batch)");
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, dag_exec_kernel<false, true>, kThreads, smem);
  if (e != cudaSuccess) return record_cuda_error(e, "occupancy of dag_exec_kernel batch");
  if (occ < 1) return HQR_ERR_UNSUPPORTED;
  if (ctas_per_sm > 0) occ = std::min(occ, ctas_per_sm);
  dag_init_batch_kernel<<<count, 256, 0, stream>>>(p);
  dag_seed_batch_kernel<<<count, 256, 0, stream>>>(p);
  const int grid = std::min(occ * dag_sm_count(), std::max(1, n_tasks));
  dag_exec_kernel<false, true><<<grid, kThreads, smem, stream>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return record_cuda_error(e, "dag_exec_kernel batch launch");
  return HQR_OK;
}

bool oz_supported(const Geometry& g) { return g.NB == oz::kK; }

// The split path rebuilds every panel tile's full T from V and TAU, which do
// not depend on the inner block width of the FP64 panels: those run with the
// narrower w = 16, whose column loop is shorter (about 13 % faster GEQRT and
// TSQRT at NB = 128, the factorization's critical path).
int narrow_panels(Geometry* g) {
  if (g->w <= 16) return HQR_OK;
  g->w = 16;
  const SmemPlan sp = SmemPlan::make(shape_of(*g));
  g->smem_bytes = (size_t)sp.total * sizeof(double);
  return HQR_OK;
}

static size_t panel_tiles(const Geometry& g) {
  return panel_slot(g.MT, g.steps, g.steps);   // slots of every (k, i), k >= i, i < steps
}
size_t oz_slice_bytes(const Geometry& g) { return panel_tiles(g) * oz::panel_slice_bytes(); }
size_t oz_panel_bytes() { return oz::panel_slice_bytes(); }
size_t oz_exp_bytes(const Geometry& g) { return panel_tiles(g) * oz::kSlots * (size_t)g.NB * sizeof(int); }
size_t oz_exp_bytes_per_panel(int NB) { return (size_t)oz::kSlots * NB * sizeof(int); }

size_t tree_slots(const Geometry& g, int S) {
  if (S <= 0 || S >= g.MT) return 0;
  return (size_t)g.steps * ((g.MT + S - 1) / S);
}

size_t factor_task_ids(const Geometry& g) { return factor_tasks(g).ids; }

int launch_factor_external(const Geometry& g, const ExternalScratch& x, double* dA, double* dTAU,
                           long long timeout_ns, cudaStream_t stream) {
  static_assert(kExternalCtlBytes == kCtlWords * sizeof(unsigned), "control words");
  static_assert(kExternalStatsBytes == 2 * kNumStats * sizeof(unsigned long long), "stats");
  DagParams p{};
  p.mode = kModeFactor;
  p.MT = g.MT;
  p.NT = g.NT;
  p.CT = g.NT;
  p.steps = g.steps;
  p.J = g.NT;
  p.nblk = g.NB / g.w;
  const FactorTasks f = factor_tasks(g);
  const FineSteps& fine = f.fine;
  set_columns(p, g, f.cb, g.NB);
  p.sp = SmemPlan::make(p.sh);
  p.fine_from = fine.from;
  p.fine_ids = (int)fine.ids;
  p.fine_sub = fine.sub;
  p.n_ids = (int)f.ids;
  long long n = fine.tasks;
  for (int i = 0; i < g.steps; i++)
    n += (long long)(g.MT - i) * p.nblk + (long long)p.NC * (g.NT - 1 - i) * (g.MT - i);
  p.n_tasks = (int)n;
  p.A = dA;
  p.T = x.T;
  p.TAU = dTAU;
  p.C = dA;
  p.cnt = x.cnt;
  p.qhi = x.qhi;
  p.qlo = x.qlo;
  p.ctl = x.ctl;
  p.stats = x.stats;
  p.timeout_ns = timeout_ns;
  const int blocks = (p.n_ids + 255) / 256;
  dag_init_kernel<<<blocks, 256, 0, stream>>>(p);
  dag_seed_kernel<<<blocks, 256, 0, stream>>>(p);
  return launch_exec<false>(p, g, stream);
}

int external_status(const ExternalScratch& x, cudaStream_t stream) {
  unsigned ctl[kCtlWords];
  cudaError_t e = cudaMemcpyAsync(ctl, x.ctl, sizeof(ctl), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return record_cuda_error(e, "DAG execution (stream synchronize)");
  if (ctl[kErr] != 0u) return (ctl[kErr] & kErrTimeout) ? HQR_ERR_TIMEOUT : HQR_ERR_DEVICE;
  return HQR_OK;
}

int dag_status(DagWorkspace* ws, cudaStream_t stream) {
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return record_cuda_error(e, "DAG execution (stream synchronize)");
  unsigned ctl[kCtlWords];
  e = cudaMemcpy(ctl, ws->ctl, sizeof(ctl), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return record_cuda_error(e, "DAG status read");
  if (ctl[kErr] != 0u) {
    cudaMemset(ws->ctl + kErr, 0, sizeof(unsigned));
    if (ctl[kErr] & kErrTimeout) return HQR_ERR_TIMEOUT;
    return HQR_ERR_DEVICE;
  }
  return HQR_OK;
}

int dag_stats(DagWorkspace* ws, unsigned long long out[14], cudaStream_t stream) {
  if (cudaStreamSynchronize(stream) != cudaSuccess) return HQR_ERR_CUDA;
  if (cudaMemcpy(out, ws->stats, 14 * sizeof(unsigned long long), cudaMemcpyDeviceToHost) !=
      cudaSuccess)
    return HQR_ERR_CUDA;
  return HQR_OK;
}

}  // namespace hqr
