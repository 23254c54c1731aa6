// Persistent per-energy-point engine for sm_100a.
//
// One team (a CTA, or a cluster of up to 16 CTAs when a call has few points)
// owns one (energy, k) point at a time and runs its complete solve:
// Sancho-Rubio decimation per contact, contact self-energies, the backward
// gsmr sweep, Gr(1,1), then (by mode) the Caroli transmission, the full
// retarded sweep with the diagonal spectral density, or the elastic
// dephasing SCBA loop with the lesser sweep, Meir-Wingreen and layer
// currents.  Teams pull points from a global queue, so all energy x k points
// of a call (and all SCBA iterations of each point) run in one launch, or in
// one for the contacts and one for the rest, with no host synchronisation;
// per-point convergence (decimation, SCBA) is
// decided on the device.
//
// Reference routines (libNEGF): decimation src/contselfenergy.F90:271-340,
// contact self-energy :445-491/:552-566, build_ESH src/iterative.F90:1956,
// gsmr/Gr/Gn sweeps src/iterative_cpu.F90:51-372, transmissions :399-583,
// DOS src/iterative.F90:1821-1952, elastic SCBA :289-363 with
// src/elphdd.F90:108-276 and src/scba.F90:120-147, Meir-Wingreen and layer
// current src/iterative.F90:382-461.
#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "program.cuh"

namespace negf {

static_assert(kGemmSmemBytes + (int)sizeof(GemmDesc) <= kSmemMain,
              "GEMM staging ring and descriptor must fit the main shared-memory region");

size_t engine_smem_bytes(int nmax) { return smem_bytes_for(nmax); }

// ---------------------------------------------------------------- helpers (primitive kernels)
__device__ __forceinline__ void gemm(int M, int N, int K, Operand A, Operand B, double2* C, int ldc,
                                     double2 alpha, double2 beta, SmemMap& sm, bool want_max = false) {
  long long t0 = sm.tr.start();
  Epilogue e = epi_store(C, ldc, alpha, beta);
  if (want_max) {
    if (threadIdx.x == 0) *sm.maxv = 0.0;
    __syncthreads();
    e.maxabs = sm.maxv;
  }
  cta_gemm(M, N, K, A, B, e, sm.main);
  sm.tr.stop(TR_GEMM, t0);
}

__device__ __forceinline__ int zinv(int n, const double2* A, double2* out, double2* ws, SmemMap& sm) {
  return cta_zinv(n, A, out, ws, sm.main, sm.inv);
}

// zinv, then the residual probe and up to two Newton steps
// X <- X + X (I - A X) where the probe exceeds kInvProbeTol (the engine's
// refine block); R and Xn are n x n scratch (R null: no probe).
// *nearly_singular (optional): the probe's condition estimate exceeds
// kSensitiveCond.
__device__ __noinline__ int zinv_refined(int n, const double2* A, double2* X, double2* ws, double2* R, double2* Xn,
                                         SmemMap& sm, bool* nearly_singular = nullptr) {
  const int bad = zinv(n, A, X, ws, sm);
  if (nearly_singular) *nearly_singular = false;
  const double2 one = make_double2(1, 0), mone = make_double2(-1, 0);
  const int nn = n * n;
  for (int k = 0; k < 2 && R; ++k) {
    double kap = 0.0;
    const double e = team_inv_probe(n, A, X, sm.main, sm.main + n, sm.maxv, &kap);
    if (k == 0 && nearly_singular && kap > kSensitiveCond) *nearly_singular = true;
    if (!(e > kInvProbeTol) || !(e <= 1.7976931348623157e308)) break;
    for (int q = team_tid(); q < nn; q += team_threads()) R[q] = make_double2((q % n) == (q / n) ? 1.0 : 0.0, 0.0);
    team_sync();
    gemm(n, n, n, opN(A, n), opN(X, n), R, n, mone, one, sm);     // R = I - A X
    team_copy(Xn, X, nn);
    team_sync();
    gemm(n, n, n, opN(X, n), opN(R, n), Xn, n, one, one, sm);     // X + X R
    team_copy(X, Xn, nn);
    team_sync();
  }
  return bad;
}

// Sancho-Rubio decimation (src/contselfenergy.F90:271-340) by one team.
// In: Ao, Bo, Co in slot 0, 2, 3 (consumed).  Out: surface GF in *go_out
// (one of the slots).  wave: CTAs that run at once.  Returns a status.
__device__ __noinline__ int cta_decimation(int L, const Ws& w, double tol, int max_iter, int& ncyc, double2** go_out,
                              int wave, SmemMap& sm) {
  double2* Ao = w.slot(0);
  double2* Aos = w.slot(1);
  double2* Go = w.slot(4);
  double2* Sf = w.slot(6);
  double2* D = w.slot(13);
  const int nn = L * L;
  int st = ST_OK;
  team_copy(Aos, Ao, nn);
  team_sync();
  bool ok = false, done = false;
  int it;
  // the engine's products, side by side in the parts of a team; with more CTAs
  // than run at once the products in vain would cost more than the latency
  // (160 of order 256: 82.8 ms one after another, 85.8 side by side)
  const int gw = (int)gridDim.x > wave ? 1 : min(team_size(), 4);
  int ib = 2, ib1 = 11, ic = 3, ic1 = 7;
  auto run = [&](int first, int of) {
    const int size = team_size() / of, rank = team_rank();
    const DecProduct p = dec_product(w, first + rank / size, ib, ib1, ic, ic1, gw);
    Epilogue e = epi_store(p.C, L, make_double2(p.alpha, 0.0), make_double2(0.0, 0.0));
    if (p.flag) {
      if (threadIdx.x == 0) *sm.maxv = 0.0;
      __syncthreads();
      e.maxabs = sm.maxv;
      e.idle_max = p.flag == 2;
    }
    gemm_run_any(gemm_desc_publish(L, L, L, opN(p.A, L), opN(p.B, L), e, sm.main, rank % size, size), sm.main);
  };
  for (it = 1; it <= max_iter; ++it) {
    if (zinv_refined(L, Ao, Go, w.inv(), w.slot(8), w.slot(9), sm)) st = ST_SINGULAR;
    run(4, min(gw, 2));                           // X = Go Co (and Y = Go Bo)
    run(0, gw);                                   // C1 = Co X (and Self = Bo X; B1 = Bo Y, D = -Co Y)
    const double mx = *sm.maxv;
    if (!(mx <= 1.7976931348623157e308)) break;   // Inf / NaN: will not converge (NOT_CONVERGED)
    if (mx <= tol) {
      if (ok) { done = true; break; }
      ok = true;
    } else {
      ok = false;
    }
    if (gw == 1) run(5, 1);
    for (int q = gw; q < 4; q += gw) run(q, gw);
    for (int q = team_tid(); q < nn; q += team_threads()) {
      Aos[q] = csub(Aos[q], Sf[q]);
      Ao[q] = cadd(D[q], csub(Ao[q], Sf[q]));
    }
    team_sync();
    { int t = ib; ib = ib1; ib1 = t; t = ic; ic = ic1; ic1 = t; }   // Bo = B1, Co = C1
  }
  ncyc = done ? it : max_iter + 1;
  if (!done && st == ST_OK) st = ST_NOT_CONVERGED;
  if (zinv_refined(L, Aos, Go, w.inv(), w.slot(8), w.slot(9), sm)) st = ST_SINGULAR;
  *go_out = Go;
  return st;
}

// ---------------------------------------------------------------- engine kernel
// Persistent: each team pulls points from the queue inside engine_step() and
// runs the heavy steps it returns.  The product loop is inlined here and the
// kernel keeps nothing in registers across engine_step() (its state is in
// local memory, the shared-memory map in shared memory), so the loop is
// register-allocated as in a kernel of its own.  The inversion leaves are
// separately compiled routines (leaf_dev.cu).
__global__ void __launch_bounds__(kThreads, 2) k_engine(EngineArgs a) {
  extern __shared__ __align__(16) char smem_raw[];
  __shared__ SmemMap smap;
  if (threadIdx.x == 0) {
    smap = map_smem(smem_raw, a.nmax);
    if (!a.trace) smap.tr.acc = nullptr;
    smap.inv.tr = smap.tr;
  }
  __syncthreads();
  if (a.trace && threadIdx.x < TR_NPHASE) smap.tr.acc[threadIdx.x] = 0;
  __syncthreads();
  const long long t_all = a.trace ? clock64() : 0;
  EngineCtl c;
  c.prog.pc = 0;
  c.prog.p = 0;
  c.in_inv = 0;
  c.open = -1;
  for (;;) {
    const int st = engine_step(a, c, smap);
    if (st == STEP_DONE) break;
    if (st == STEP_GEMM) {
      const GemmDesc* d = reinterpret_cast<const GemmDesc*>(smap.main + kGemmDescOffset);
      if (d->tile == kTile) cta_gemm_body<kTile>(d, smap.main);
      else gemm_run_small(d, smap.main);
    } else if (st == STEP_ROWS) {
      rows_run(c.ip, smap.main, smap.inv);
    } else {
      leaf_run(c.ip, smap.main, smap.inv);
    }
  }
  team_sync();   // no member's shared memory is read any more
  if (a.trace) {
    if (threadIdx.x == 0) smap.tr.acc[TR_TOTAL] += clock64() - t_all;
    __syncthreads();
    if (threadIdx.x < TR_NPHASE) atomicAdd(a.trace + threadIdx.x, (unsigned long long)smap.tr.acc[threadIdx.x]);
  }
}

int64_t engine_contact_elems(int nmax) { return (int64_t)S_SIG * nmax * nmax; }

int64_t engine_slots(int mode, int nbl_max, int ncont_max) {
  int64_t s = S_SIG + ncont_max;
  if (mode == MODE_T || mode == MODE_DOS) s += nbl_max + ncont_max;   // gsmr, Gr(cb,cb)
  else if (mode == MODE_RHO) s += nbl_max + 2 * ncont_max;             // + gs per contact
  else s += 8 * (int64_t)nbl_max + ncont_max;                     // GN arrays, gs per contact
  return s;
}

int64_t engine_ws_elems(int mode, int nbl_max, int ncont_max, int nmax) {
  const int64_t Q = (int64_t)nmax * nmax;
  int64_t e = engine_slots(mode, nbl_max, ncont_max) * Q;
  if (mode == MODE_GN) e += 2 * (int64_t)nbl_max * nmax + 16;  // sigma_r, sigma_n vectors
  return e;
}

// Kernels whose limits have been raised, by device.
static std::mutex g_opt_mu;
static std::set<std::pair<const void*, int>> g_opted;

cudaError_t team_opt_in(const void* kernel, size_t smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_opt_mu);
  if (g_opted.count({kernel, dev})) return cudaSuccess;
  if (smem == 0) smem = engine_smem_bytes(kMaxOrder);
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) g_opted.insert({kernel, dev});
  return e;
}

void team_opt_out(const void* kernel) {
  int dev = 0;
  cudaGetLastError();
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  std::lock_guard<std::mutex> lk(g_opt_mu);
  g_opted.erase({kernel, dev});
}

cudaLaunchConfig_t team_config(int teams, int team, size_t smem, cudaStream_t s, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(teams * team);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  if (team > 1) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = team;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  return cfg;
}

cudaError_t launch_engine(const EngineArgs& a, int teams, int team, cudaStream_t s) {
  cudaLaunchAttribute attr;
  return team_launch(team_config(teams, team, engine_smem_bytes(a.nmax), s, &attr), k_engine, 0, a);
}

// Clusters of `team` CTAs that run at once on the current device (0: none),
// queried once per device and size.  Asked of the engine, and taken for the
// inverse and the decimation too: all have two CTAs to an SM, of the same
// threads, registers and shared memory.
static int resident_teams(int team) {
  static std::mutex mu;
  static int known[64][5];   // count + 1
  int dev = 0, lg = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  while ((1 << lg) < team) ++lg;
  std::lock_guard<std::mutex> lk(mu);
  if (known[dev][lg] == 0) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = team_config(1, team, engine_smem_bytes(kMaxOrder), nullptr, &attr);
    for (int attempt = 0; attempt < 2; ++attempt) {   // again with the limits raised afresh (see team_launch)
      int n = 0;
      cudaError_t e = team_opt_in((const void*)k_engine);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, k_engine, &cfg);
      if (e == cudaSuccess) {
        known[dev][lg] = n + 1;
        break;
      }
      team_opt_out((const void*)k_engine);
    }
    if (known[dev][lg] == 0) return 0;   // asked again by the next call
  }
  return known[dev][lg] - 1;
}

// The team size whose measured cost for `work` problems is least.  Three
// figures make up the cost (T solves of orders 32 .. 384, 1 .. 400 points,
// every team size timed):
//  - the time of one problem alone, relative to one CTA.  Products and
//    updates split over the team, the elimination's panels do not: order 256
//    takes 0.58, 0.33, 0.23, 0.18 of the time in teams of 2, 4, 8, 16 (171 ->
//    29 ms for a point of 3 layers), order 128 0.64 .. 0.32, order 64 0.71 at
//    best (one panel, four output tiles), order 32 nothing;
//  - the slowdown when the teams share SMs.  Two CTAs on an SM run 1.6 times
//    as long as one, as soon as any SM has two; teams of 4 and more leave the
//    FP64 pipe less idle time to share (2.05 times with every SM holding two)
//    and are placed two to an SM before every SM has one.  The numbers of CTAs
//    at which this sets in were measured on 148 SMs and scale with the SMs;
//  - the waves.  One or two CTAs per problem wait for the last wave; larger
//    teams drift apart over the waves and lose less.
// Examples (us per call, one CTA per problem -> chosen): n = 384, 12 points
// 825000 -> 195000 (16); n = 97, 48 points 28200 -> 16050 (4); n = 256, 320
// points 400000 -> 362000 (2); 296 points stay with one CTA (278000; 304000
// in teams of 2).
static double team_cost(int work, int n, int max_ctas, int sms, int lg, TeamShape* shape) {
  static const double kAlone[3][5] = {{1.0, 0.90, 0.71, 0.70, 0.70},    // n <= 80
                                      {1.0, 0.64, 0.45, 0.385, 0.32},   // n <= 150
                                      {1.0, 0.58, 0.33, 0.225, 0.18}};
  const int team = 1 << lg;
  if (team > 1 && n <= 40) return -1.0;
  int teams = std::min(max_ctas / team, team > 1 ? resident_teams(team) : max_ctas);
  if (teams < 1) return -1.0;
  const double waves = (double)work / teams;
  teams = std::min(teams, std::max(1, work));
  const double c = 148.0 * teams * team / sms;   // CTAs per 148 SMs
  double share = 1.0, w = 1.0;
  if (team <= 2) {
    if (c > 148.0) share = 1.6;
    const double whole = (double)(int)waves, frac = waves - whole;
    if (waves > 1.0) w = whole + (frac > 0.0 ? (team == 1 ? 0.4 + 0.45 * frac : 0.3 + 0.55 * frac) : 0.0);
  } else {
    if (c > 192.0) share = 1.42 + 0.63 * (c - 192.0) / 104.0;
    else if (c > 148.0) share = 1.35 + 0.07 * (c - 148.0) / 44.0;
    else if (c > 100.0) share = 1.0 + 0.35 * (c - 100.0) / 48.0;
    if (waves > 1.0) w = 0.35 + 0.68 * waves;
  }
  *shape = TeamShape{team, teams};
  return kAlone[n <= 80 ? 0 : (n <= 150 ? 1 : 2)][lg] * share * w;
}

static double best_team(int work, int n, int max_ctas, int sms, TeamShape* best) {
  double best_cost = -1.0;
  *best = TeamShape{1, std::max(1, std::min(work, max_ctas))};
  for (int lg = 0; lg <= 4; ++lg) {
    TeamShape t;
    const double c = team_cost(work, n, max_ctas, sms, lg, &t);
    if (c >= 0.0 && (best_cost < 0.0 || c < best_cost)) {
      best_cost = c;
      *best = t;
    }
  }
  return best_cost;
}

TeamShape team_shape(int work, int n, int max_ctas, int sms) {
  TeamShape t;
  best_team(work, n, max_ctas, sms, &t);
  return t;
}

// Problems a little above one full wave of the best team size leave most CTAs
// idle in the second wave, although larger teams would finish it sooner: up to
// two waves, the full one and the rest run as two launches where the costs
// above say 5 % or more (below that the drain of the first launch takes the
// gain).  320 points of order 256 with DOS (12 layers): 566 -> 539 ms;
// 160 points of order 128: 31.6 -> 29.5, of order 97: 27.1 -> 25.7.  Beyond two waves the
// points' different decimation counts smear the waves and the split gained
// nothing (600 points of order 128: 88.7 -> 92.6 ms with it).
TeamPlan team_plan(int work, int n, int max_ctas, int sms) {
  TeamPlan pl;
  pl.parts = 1;
  pl.count[0] = work;
  pl.count[1] = 0;
  double cost = 0.95 * best_team(work, n, max_ctas, sms, &pl.shape[0]);
  pl.shape[1] = pl.shape[0];
  for (int lg = 0; lg <= 4; ++lg) {
    TeamShape t, rest;
    if (team_cost(work, n, max_ctas, sms, lg, &t) < 0.0 || work <= t.teams || work % t.teams == 0) continue;
    if (work > 2 * t.teams) continue;
    const int whole = work / t.teams * t.teams;
    const double c = team_cost(whole, n, max_ctas, sms, lg, &t) + best_team(work - whole, n, max_ctas, sms, &rest);
    if (c < cost) {
      cost = c;
      pl.parts = 2;
      pl.count[0] = whole;
      pl.count[1] = work - whole;
      pl.shape[0] = t;
      pl.shape[1] = rest;
    }
  }
  return pl;
}

// ---------------------------------------------------------------- primitives
// CTA (x, b) of the grid: output tiles (of tile x tile elements) x, x + gridDim.x, ... of product b.
__global__ void __launch_bounds__(kThreads, 2)
    k_zgemm_batched(int m, int n, int k, double2 alpha, const double2* A, int64_t sA, const double2* B,
                    int64_t sB, double2 beta, double2* C, int64_t sC, int dagger, int tile) {
  extern __shared__ __align__(16) char smem_raw[];
  SmemMap sm = map_smem(smem_raw, 1);
  sm.tr.acc = nullptr;
  const int64_t b = blockIdx.y;
  Operand Ao = (dagger == 1) ? opC(A + b * sA, k) : opN(A + b * sA, m);
  Operand Bo = (dagger == 2) ? opC(B + b * sB, n) : opN(B + b * sB, k);
  const GemmDesc* d = gemm_desc_publish(m, n, k, Ao, Bo, epi_store(C + b * sC, m, alpha, beta), sm.main, blockIdx.x,
                                        gridDim.x, tile);
  if (d->tile == kTile) cta_gemm_body<kTile>(d, sm.main);
  else gemm_run_small(d, sm.main);
}

// SMs of the current device, asked once per device.
int device_sms() {
  static std::mutex mu;
  static int known[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  std::lock_guard<std::mutex> lk(mu);
  if (known[dev] == 0 && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
    known[dev] = n;
  return known[dev] > 0 ? known[dev] : 148;
}

// Whether some problem's C (nc elements) shares memory with its own operand A (na elements).
static bool in_place(const double2* A, int64_t sA, int64_t na, const double2* C, int64_t sC, int64_t nc, int batch) {
  constexpr int64_t kElem = sizeof(double2);
  const int64_t first = reinterpret_cast<intptr_t>(C) - reinterpret_cast<intptr_t>(A);
  const int64_t last = first + (int64_t)(batch - 1) * (sC - sA) * kElem;   // of the last problem; linear between
  return std::min(first, last) < na * kElem && std::max(first, last) > -nc * kElem;
}

// The output tile of a batch of m x n products, a tile per CTA.  Small tiles
// spread few products over more SMs, but cost 0.46 of a large one's time for a
// quarter of its elements, so they lose as soon as the large ones fill the GPU.
// Where C has at most 32 rows or columns, half of a large tile's warps idle: it
// takes 0.66 alone (a small one 0.33), 1.5 times that beside another one, 0.5 in
// a full GPU.  CTAs that share an SM share its FP64 pipe: 1.95 times the time with
// two large tiles, 1.7 with two small ones, and in proportion beyond that.  us,
// small and large tiles, one per CTA: order 64, 74 products 12.9 and 16.8, 148:
// 22.1 and 16.8, 296: 39.4 and 26.0; order 128, 100: 87.7 and 65.2; order 300, 6:
// 78.4 and 94.5, 10: 118 and 96.
static int zgemm_tile(int batch, int m, int n, int sms) {
  const double big = (double)((m + kTile - 1) / kTile) * ((n + kTile - 1) / kTile);
  const double small = (double)((m + kSmallTile - 1) / kSmallTile) * ((n + kSmallTile - 1) / kSmallTile);
  const bool narrow = m <= kSmallTile || n <= kSmallTile;
  const double work_big = narrow ? 0.66 : 1.0, work_small = narrow ? 0.33 : 0.46;
  auto time = [&](double ctas, double two) {
    const double x = ctas * batch / sms;
    return x <= 1.0 ? 1.0 : (x <= 2.0 ? two : two * (0.5 * x + 0.2));
  };
  if (big * batch > 4.0 * sms)   // two waves of large tiles: the work alone decides
    return (narrow ? 0.5 : 1.0) * big <= 0.46 * small ? kTile : kSmallTile;
  return work_big * time(big, narrow ? 1.5 : 1.95) <= 0.98 * work_small * time(small, 1.7) ? kTile : kSmallTile;
}

cudaError_t launch_zgemm_batched(int batch, int m, int n, int k, double2 alpha, const double2* A, int64_t sA,
                                 const double2* B, int64_t sB, double2 beta, double2* C, int64_t sC,
                                 int dagger, cudaStream_t s) {
  // A tile per CTA (one CTA per product left all but `batch` SMs idle: 6
  // products of order 300 1604 -> 82 us), up to a number of CTAs per SM beyond
  // which a CTA runs through several tiles of a product and loads the next
  // tile's operands behind this one's epilogue: the shorter the product, the
  // more that counts beside the spread (900 products of 128 x 128: K = 16 103 us
  // with two tiles per CTA, 122 with one; K = 128 509 and 484).
  const int sms = device_sms();
  int T = zgemm_tile(batch, m, n, sms);
  const int64_t per_sm = std::min(48, 4 * ((k + TK - 1) / TK) + 4);
  int64_t want = (per_sm * sms + batch - 1) / batch;
  // C in the place of A or B: up to order 64 one CTA holds the whole product in
  // one tile and has read all operands when it stores, so such calls stay with it.
  if (m <= kTile && n <= kTile &&
      (in_place(A, sA, (int64_t)m * k, C, sC, (int64_t)m * n, batch) ||
       in_place(B, sB, (int64_t)k * n, C, sC, (int64_t)m * n, batch))) {
    T = m <= kSmallTile && n <= kSmallTile ? kSmallTile : kTile;
    want = 1;
  }
  const int64_t tiles = (int64_t)((m + T - 1) / T) * ((n + T - 1) / T);
  const int split = (int)std::max<int64_t>(1, std::min(tiles, want));
  for (int b0 = 0; b0 < batch; b0 += 65535) {   // gridDim.y limit
    const int nb = std::min(65535, batch - b0);
    cudaLaunchConfig_t cfg = team_config(1, 1, engine_smem_bytes(1), s, nullptr);
    cfg.gridDim = dim3(split, nb);
    const cudaError_t e = team_launch(cfg, k_zgemm_batched, 0, m, n, k, alpha, A + b0 * sA, sA, B + b0 * sB, sB, beta,
                                      C + b0 * sC, sC, dagger, T);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// per matrix: the inversion's own buffers, then two n x n refinement buffers
size_t zinv_batched_work_elems(int n) { return zinv_ws_elems(n) + 2 * (size_t)n * n; }

// One team per matrix: the inverses of the problems map[b], b < batch (map
// null: b), matrices sA / sX complex elements apart; work (may be null where
// the inversion needs no buffers: then no residual probe) holds batch slots
// of wstride.  info[p] gets the zgetrf-style singular column (0 = none).
__global__ void __launch_bounds__(kThreads, 2)
    k_zinv_mapped(int n, const double2* A, int64_t sA, double2* X, int64_t sX, const int* map, int* info,
                  double2* work, int64_t wstride, int* sens) {
  extern __shared__ __align__(16) char smem_raw[];
  SmemMap sm = map_smem(smem_raw, n);
  sm.tr.acc = nullptr;
  const int b = blockIdx.x / team_size();
  const int64_t p = map ? map[b] : b;
  double2* wb = work ? work + (int64_t)b * wstride : nullptr;
  double2* R = work ? wb + zinv_ws_elems(n) : nullptr;
  bool near_sing = false;
  int inf = zinv_refined(n, A + p * sA, X + p * sX, wb, R, R ? R + (int64_t)n * n : nullptr, sm, &near_sing);
  if (lead() && info) info[p] = inf;
  if (lead() && sens && near_sing) sens[p] = 1;
  team_sync();   // no member's shared memory is read any more
}

// Teams for a batch of inverses alone.  Their panels do not split over a team,
// so a team's other CTAs mostly wait in the places of other matrices: with more
// matrices than SMs one CTA each, with more than half as many one (up to order
// 128, four leaves) or two.  ms by this rule and by the teams that suit a
// decimation: order 256, 100 matrices 1.88 and 2.36, 250: 2.85 and 3.80, 297: 4.40
// and 5.82; order 128, 170: 0.49 and 0.68; order 257, 100: 3.3 and 4.7.
TeamShape zinv_shape(int batch, int n, int max_ctas, int sms) {
  if (2 * batch > sms) {
    const int team = batch > sms || n <= 128 ? 1 : 2;
    if (team == 1 || resident_teams(team) >= 1) return TeamShape{team, std::min(batch, max_ctas / team)};
  }
  return team_shape(batch, n, max_ctas, sms);
}

cudaError_t launch_zinv_mapped(int batch, int n, const double2* A, int64_t sA, double2* X, int64_t sX,
                               const int* map, int* info, double2* work, cudaStream_t s, int* sens) {
  if (batch <= 0) return cudaSuccess;
  const TeamShape t = zinv_shape(batch, n, 2 * device_sms(), device_sms());
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = team_config(batch, t.team, engine_smem_bytes(n), s, &attr);
  return team_launch(cfg, k_zinv_mapped, 0, n, A, sA, X, sX, map, info, work,
                     (int64_t)zinv_batched_work_elems(n), sens);
}

cudaError_t launch_zinv_batched(int batch, int n, const double2* A, double2* Ainv, int* info, double2* work,
                                cudaStream_t s) {
  const int64_t nn = (int64_t)n * n;
  return launch_zinv_mapped(batch, n, A, nn, Ainv, nn, nullptr, info, work, s, nullptr);
}

__host__ __device__ inline size_t dec_work_elems(int n) { return (size_t)(S_INV + 3) * n * n; }
size_t decimation_batched_work_elems(int n) { return dec_work_elems(n); }

__global__ void __launch_bounds__(kThreads, 2)
    k_decimation_batched(int n, const double2* Ao, const double2* Bo, const double2* Co, double2* Go, int* ncyc,
                         double tol, int max_iter, double2* work, int wave) {
  extern __shared__ __align__(16) char smem_raw[];
  SmemMap sm = map_smem(smem_raw, n);
  sm.tr.acc = nullptr;
  const int b = blockIdx.x / team_size();
  const int64_t nn = (int64_t)n * n;
  Ws w;
  w.base = work + (int64_t)b * dec_work_elems(n);
  w.Q = nn;
  w.ncont = 0;
  w.sigp = w.gsp = nullptr;
  team_copy(w.slot(0), Ao + b * nn, (int)nn);
  team_copy(w.slot(2), Bo + b * nn, (int)nn);
  team_copy(w.slot(3), Co + b * nn, (int)nn);
  team_sync();
  int nc = 0;
  double2* gs = nullptr;
  cta_decimation(n, w, tol, max_iter, nc, &gs, wave, sm);
  team_copy(Go + b * nn, gs, (int)nn);
  if (lead() && ncyc) ncyc[b] = nc;
  team_sync();   // no member's shared memory is read any more
}

cudaError_t launch_decimation_batched(int batch, int n, const double2* Ao, const double2* Bo, const double2* Co,
                                      double2* Go, int* ncyc, double tol, int max_iter, double2* work,
                                      cudaStream_t s) {
  const TeamShape t = team_shape(batch, n, 2 * device_sms(), device_sms());
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = team_config(batch, t.team, engine_smem_bytes(n), s, &attr);
  return team_launch(cfg, k_decimation_batched, 0, n, Ao, Bo, Co, Go, ncyc, tol, max_iter, work,
                     2 * device_sms());
}

}  // namespace negf
