// Small-order transmission (small.cuh): the 2-contact Caroli solve of a point
// of block order n <= 32 by one CTA, or by two with a contact each, following
// the reference routine by routine:
//   surface_green + decimation   src/contselfenergy.F90:184-210, 271-340
//   compute_contacts             src/contselfenergy.F90:445-491, 552-566
//   build_ESH (real E)           src/iterative.F90:1956-1982
//   gsmr sweep, Gr(1,1)          src/iterative_cpu.F90:51-170
//   Caroli trace                 src/iterative_cpu.F90:399-470
//
// At these orders a product is 2000 cycles of an SM's FP64 pipe and an
// inversion a chain of 32 dependent steps; what a point costs is latency.
// With every point through one launch per block operation (the form before
// this one: about 280 launches a call, operands through memory each time) a
// launch was 10 to 25 us of mostly fixed latency.  Here a point's blocks
// never leave the SM between operations: one energy of a 20-layer device of
// order 32 takes 0.94 ms (3.10 before), 512 energies 3.34 ms (6.07).
#include <cuda_runtime.h>

#include "../../include/negf_b200.h"
#include "cta_ops.cuh"
#include "small.cuh"

namespace negf {
namespace {

// The kernel for orders up to M (32 or 16).  Blocks lie in shared memory column
// major with M + 2 rows per column: 2 modulo 8 elements, so that the eight lanes
// of a 128-byte phase of a fragment load hit different banks, for the left
// operand with lane (g, t) on row g of column t and for the right one with
// columns taken in the order of ncol().  Orders up to 16 have work for two of
// eight warps in a product and for one row per lane of 16 in a panel, and half
// the threads let four CTAs share an SM instead of two: 9000 energies of a
// 10-layer device of order 1, 8 and 16 take 3.8, 6.6 and 12.5 ms (8.3, 12.9 and
// 20.5 with the shape of order 32; 7.5, 11.9 and 20.6 with one warp per point
// and block operation, every operation a launch).
constexpr int kBlocks = 6;
template <int M>
struct Shape {
  static constexpr int kCta = M == 32 ? kThreads : kThreads / 2;   // threads
  static constexpr int kPerSm = M == 32 ? 2 : 4;                   // CTAs that share an SM
  static constexpr int kLd = M + 2, kBlk = M * kLd;
  static constexpr int kWarps = kCta / 32;
  static constexpr size_t kScratch = 3 * 32 + kWarps * 4 + 4;      // gj_panel<1, 4>
};
constexpr unsigned kFull = 0xffffffffu;

struct SmallShared {
  InvScratch inv;
  int piv[32], perm[32], cperm[32], flag, ncyc, st;
  double red[3][8];
  double2 y[32];
};
template <int M>
constexpr size_t small_smem() {
  return (kBlocks * Shape<M>::kBlk + Shape<M>::kScratch) * sizeof(double2) + sizeof(SmallShared);
}

// The dynamic shared memory, named wherever it is used so that accesses
// compile to shared-memory instructions: blocks, panel scratch, the rest.
extern __shared__ __align__(16) char smem_raw[];
enum Block : int { B_AO = 0, B_BO = 1, B_CO = 2, B_GO = 3, B_X = 4, B_SL = 5 };
template <int M>
__device__ __forceinline__ double2* block(int b) {
  return reinterpret_cast<double2*>(smem_raw) + b * Shape<M>::kBlk;
}
template <int M>
__device__ __forceinline__ SmallShared& shared() {
  return *reinterpret_cast<SmallShared*>(reinterpret_cast<double2*>(smem_raw) + kBlocks * Shape<M>::kBlk +
                                         Shape<M>::kScratch);
}

__device__ __forceinline__ int ncol(int g) { return (g & 4) | ((g & 1) << 1) | ((g & 2) >> 1); }

// A thread's four elements of an M x M product (the fragment layout of
// dmma_16x8x4): element q at (row(q), col(q)); rows and columns from n on
// are not part of the block.
struct Frag {
  double2 v[4];
};
template <int M>
struct Lane {
  static constexpr int kLd = Shape<M>::kLd;
  int n, g, t, m0, n0;
  __device__ __forceinline__ explicit Lane(int order) : n(order) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    g = lane >> 2;
    t = lane & 3;
    m0 = (w >> 2) * 16;
    n0 = (((w & 3) + 2 * (w >> 2)) & 3) * 8;   // tiles of n <= 16 on all four schedulers
  }
  __device__ __forceinline__ int row(int q) const { return m0 + g + ((q >> 1) << 3); }
  __device__ __forceinline__ int col(int q) const { return n0 + ncol(2 * t + (q & 1)); }
  __device__ __forceinline__ bool in(int q) const { return row(q) < n && col(q) < n; }
  __device__ __forceinline__ int at(int q) const { return row(q) + col(q) * kLd; }
};

// A B, on the FP64 tensor pipe; entries of A and B from n on are zero.
template <int M>
__device__ __forceinline__ Frag mm(const Lane<M>& L, const double2* A, const double2* B) {
  double re[4] = {0.0, 0.0, 0.0, 0.0}, im[4] = {0.0, 0.0, 0.0, 0.0};
  constexpr int kLd = Shape<M>::kLd;
  if (L.m0 < L.n && L.n0 < L.n) {
    const double2* pa = A + L.t * kLd + L.m0 + L.g;
    const double2* pb = B + (L.n0 + ncol(L.g)) * kLd + L.t;
#pragma unroll 4
    for (int k = 0; k < L.n; k += 4) {
      const double2 a0 = pa[k * kLd], a1 = pa[k * kLd + 8], b = pb[k];
      dmma_16x8x4(re, a0.x, a1.x, b.x);
      dmma_16x8x4(im, a0.x, a1.x, b.y);
      dmma_16x8x4(re, a0.y, a1.y, -b.y);
      dmma_16x8x4(im, a0.y, a1.y, b.x);
    }
  }
  Frag f;
#pragma unroll
  for (int q = 0; q < 4; ++q) f.v[q] = make_double2(re[q], im[q]);
  return f;
}
template <int M>
__device__ __forceinline__ void put(const Lane<M>& L, double2* D, const Frag& f) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (L.in(q)) D[L.at(q)] = f.v[q];
}
template <int M>
__device__ __forceinline__ Frag get(const Lane<M>& L, const double2* S) {
  Frag f;
#pragma unroll
  for (int q = 0; q < 4; ++q) f.v[q] = L.in(q) ? S[L.at(q)] : make_double2(0.0, 0.0);
  return f;
}
// get() from the shared memory of another CTA of the cluster
template <int M>
__device__ __forceinline__ Frag team_get(const Lane<M>& L, const double2* S, int rank) {
  Frag f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double* e = reinterpret_cast<const double*>(S + L.at(q));
    f.v[q] = L.in(q) ? make_double2(team_ld_double(e, rank), team_ld_double(e + 1, rank)) : make_double2(0.0, 0.0);
  }
  return f;
}
template <int M>
__device__ __forceinline__ void sub_from(const Lane<M>& L, double2* D, const Frag& f) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (L.in(q)) D[L.at(q)] = csub(D[L.at(q)], f.v[q]);
}

// Maximum of v over the CTA (NaN in any thread: NaN); red: 8 doubles.  Ends
// with a barrier before red is next written (the callers' own barriers).
template <int M>
__device__ __forceinline__ double cta_max_nan(double v, double* red) {
  bool bad = !(v <= 1.7976931348623157e308);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(kFull, v, o));
  bad = __any_sync(kFull, bad);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = bad ? __longlong_as_double(0x7ff8000000000000LL) : v;
  __syncthreads();
  double m = red[0];
#pragma unroll
  for (int w = 1; w < Shape<M>::kWarps; ++w) m = (m != m || red[w] != red[w]) ? m + red[w] : fmax(m, red[w]);
  return m;
}

// Go = Ao^-1 (Ao kept), the residual probe and up to two Newton steps
// Go + Go (I - Ao Go) where it exceeds kInvProbeTol (in the X block).
// Returns 1 for an exactly zero pivot, + 2 where the condition estimate of Ao
// exceeds kSensitiveCond.
template <int M>
__device__ __noinline__ int small_inverse(int n) {
  constexpr int kLd = Shape<M>::kLd;
  const Lane<M> L(n);
  const double2* const A = block<M>(B_AO);
  double2* const X = block<M>(B_GO);
  double2* const R = block<M>(B_X);
  SmallShared& sh = shared<M>();
  bool sens = false;
  if (threadIdx.x == 0) sh.flag = 0;
  __syncthreads();
  gj_panel<1, 4, true, Shape<M>::kWarps>(A, kLd, X, kLd, n, 0, n, block<M>(kBlocks), sh.inv);
  const int info = sh.flag != 0 ? 1 : 0;
  // probe: threads (row, group of columns) = (tid / 8, tid mod 8)
  const int r = threadIdx.x >> 3, grp = threadIdx.x & 7;
  for (int round = 0; round < 2; ++round) {
    double2 acc = make_double2(0.0, 0.0);
    if (r < n)
      for (int c = grp; c < n; c += 8) acc = cadd(acc, cmul(X[r + c * kLd], probe_v(c)));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(kFull, acc.x, o);
      acc.y += __shfl_xor_sync(kFull, acc.y, o);
    }
    if (grp == 0 && r < n) sh.y[r] = acc;
    __syncthreads();
    acc = make_double2(0.0, 0.0);
    double sa = 0.0;
    if (r < n)
      for (int c = grp; c < n; c += 8) {
        const double2 a = A[r + c * kLd], y = sh.y[c];
        acc = cadd(acc, cmul(a, y));
        sa += cabs1(a) * cabs1(y);
      }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(kFull, acc.x, o);
      acc.y += __shfl_xor_sync(kFull, acc.y, o);
      sa += __shfl_xor_sync(kFull, sa, o);
    }
    double e = 0.0;
    if (r < n) {
      const double2 d = csub(acc, probe_v(r));
      e = cabs1(d);   // an upper bound of |d| within sqrt 2
      if (!(e <= 1.7976931348623157e308)) e = __longlong_as_double(0x7ff0000000000000LL);
      else if (e > kInvProbeTol) e = cabs(d);
    } else {
      sa = 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      e = fmax(e, __shfl_xor_sync(kFull, e, o));
      sa = fmax(sa, __shfl_xor_sync(kFull, sa, o));
    }
    if ((threadIdx.x & 31) == 0) {
      sh.red[0][threadIdx.x >> 5] = e;
      sh.red[1][threadIdx.x >> 5] = sa;
    }
    __syncthreads();
    double em = 0.0, km = 0.0;
#pragma unroll
    for (int w = 0; w < Shape<M>::kWarps; ++w) {
      em = fmax(em, sh.red[0][w]);
      km = fmax(km, sh.red[1][w]);
    }
    if (round == 0 && km > kSensitiveCond) sens = true;
    if (!(em > kInvProbeTol) || !(em <= 1.7976931348623157e308)) break;
    Frag p = mm(L, A, X);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      p.v[q] = csub(make_double2(L.row(q) == L.col(q) ? 1.0 : 0.0, 0.0), p.v[q]);
    put(L, R, p);
    __syncthreads();
    p = mm(L, X, R);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (L.in(q)) X[L.at(q)] = cadd(X[L.at(q)], p.v[q]);
    __syncthreads();
  }
  return info + (sens ? 2 : 0);
}

// D = z S - H (S null: the identity if diag, else zero) for an n x n block
// in memory; with dag its conjugate transpose.
template <int M>
__device__ __forceinline__ void load_esh(int n, double2* D, const double2* H, const double2* S, double2 z, bool diag,
                                         bool dag) {
  constexpr int kLd = Shape<M>::kLd;
  for (int q = threadIdx.x; q < n * n; q += Shape<M>::kCta) {
    const int i = q % n, j = q / n;
    const double2 s = S ? S[q] : make_double2(diag && i == j ? 1.0 : 0.0, 0.0);
    const double2 v = csub(cmul(z, s), H[q]);
    if (dag) D[j + i * kLd] = cconj(v);
    else D[i + j * kLd] = v;
  }
}

template <int M>
__global__ void __launch_bounds__(Shape<M>::kCta, Shape<M>::kPerSm) k_small_point(MixedArgs a) {
  constexpr int kLd = Shape<M>::kLd;
  double2* const Ao = block<M>(B_AO);
  double2* const Bo = block<M>(B_BO);
  double2* const Co = block<M>(B_CO);
  double2* const Go = block<M>(B_GO);
  double2* const X = block<M>(B_X);
  double2* const SL = block<M>(B_SL);               // the left self-energy
  SmallShared& sh = shared<M>();
  const int pair = team_size() == 2, rank = team_rank();
  const int p = blockIdx.x >> pair, n = a.n;
  const Lane<M> L(n);
  if (threadIdx.x == 0) {
    sh.inv.piv = sh.piv;
    sh.inv.perm = sh.perm;
    sh.inv.cperm = sh.cperm;
    sh.inv.flag = &sh.flag;
    sh.inv.tr.acc = nullptr;
  }
  for (int q = threadIdx.x; q < kBlocks * Shape<M>::kBlk; q += Shape<M>::kCta) Ao[q] = make_double2(0.0, 0.0);
  __syncthreads();
  const DevDesc& d = a.d_descs[a.d_ids[p]];
  const double E = a.d_E[p];
  int st = NEGF_B200_OK, ncyc = 0;
  auto put_st = [&](int code) { if (st == NEGF_B200_OK) st = code; };

#pragma unroll 1
  for (int side = rank; side < (pair ? rank + 1 : 2); ++side) {
    const int c = side == 0 ? a.left : a.right;
    const double2* h00 = d.h00 + d.olead[c];
    const double2* h01 = d.h01 + d.olead[c];
    const double2* s00 = d.has_s00 ? d.s00 + d.olead[c] : nullptr;
    const double2* s01 = d.has_s01 ? d.s01 + d.olead[c] : nullptr;
    int cyc = 0;
    int have = 0;                                // an attempt's gs is kept: 1 one's that converged, 2 any other's
    int kept_cyc = 0;
    Frag kept;
#pragma unroll 1
    for (int att = 0;; ++att) {
      // ---- decimation from the contact energy times 1 + att 2^-50 (see kDecRetries)
      const double scale = 1.0 + att * 0x1p-50;
      const double2 ec = make_double2(E * scale, a.eta * scale);
      load_esh<M>(n, Ao, h00, s00, ec, true, false);
      load_esh<M>(n, Bo, h01, s01, ec, false, false);
      load_esh<M>(n, Co, h01, s01, cconj(ec), false, true);
      __syncthreads();
      Frag Aos = get(L, Ao);
      bool ok = false, done = false, sens = false, diverged = false, off = false;
      cyc = 0;
      int it = 1;
#pragma unroll 1
      for (; it <= a.sgf_max_iter; ++it) {
        const int bad_inv = small_inverse<M>(n);
        if (bad_inv & 1) put_st(NEGF_B200_ERR_SINGULAR);
        sens |= (bad_inv & 2) != 0;
        __syncthreads();
        put(L, X, mm(L, Go, Co));
        __syncthreads();
        const Frag C1 = mm(L, Co, X);
        double mx = 0.0;
        bool bad = false;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (L.in(q)) {
            const double h = hypot(C1.v[q].x, C1.v[q].y);
            mx = fmax(mx, h);
            bad |= !(h <= 1.7976931348623157e308);
          }
        mx = cta_max_nan<M>(bad ? __longlong_as_double(0x7ff8000000000000LL) : mx, sh.red[2]);
        if (!(mx <= 1.7976931348623157e308)) {   // Inf / NaN: will not converge
          diverged = done = true;
        } else if (mx <= a.sgf_tol) {
          done = ok;
          ok = true;
        } else {
          ok = false;
        }
        if (done) {
          cyc = it;
          break;
        }
        Frag f = mm(L, Bo, X);                   // Self
#pragma unroll
        for (int q = 0; q < 4; ++q) Aos.v[q] = csub(Aos.v[q], f.v[q]);
        sub_from(L, Ao, f);
        __syncthreads();                         // X is read; Y takes its place
        put(L, X, mm(L, Go, Bo));
        __syncthreads();
        const Frag B1 = mm(L, Bo, X);
        f = mm(L, Co, X);
        sub_from(L, Ao, f);
        __syncthreads();
        put(L, Bo, B1);
        put(L, Co, C1);
        __syncthreads();
      }
      if (!done) {
        cyc = a.sgf_max_iter + 1;
        put_st(NEGF_B200_ERR_NOT_CONVERGED);
      }
      __syncthreads();
      put(L, Ao, Aos);
      __syncthreads();
      const int bad_gs = small_inverse<M>(n);       // gs in Go
      if (bad_gs & 1) put_st(NEGF_B200_ERR_SINGULAR);
      sens |= (bad_gs & 2) != 0;
      __syncthreads();
      if (a.eta == 0.0) {   // no other branch to try; gs of an iteration broken off means nothing
        if (diverged) {
          cyc = a.sgf_max_iter + 1;
          put_st(NEGF_B200_ERR_NOT_CONVERGED);
        }
        break;
      }
      // the retarded branch (eta > 0) has -Im gs_ii >= 0 up to 1e-6 of the
      // largest |gs_ii|, the advanced one (eta < 0) Im gs_ii >= 0
      const double sgn = a.eta > 0.0 ? -1.0 : 1.0;
      double lo = 1.7976931348623157e308, hi = 0.0;
      for (int i = 0; i < n; ++i) {
        const double2 g = Go[i * (kLd + 1)];
        const double h = cabs(g);
        if (!(h <= 1.7976931348623157e308)) off = true;
        else {
          lo = fmin(lo, sgn * g.y);
          hi = fmax(hi, h);
        }
      }
      if (hi > 0.0 && lo < -1e-6 * hi) off = true;
      if (!diverged && !off && !sens) break;
      // sensitive: accepted once two attempts reach the same gs.  An attempt that
      // ran off with a gs on the right branch is none to accept, but one to
      // agree with a converged attempt's, kept before or still to come
      if (!off) {
        const Frag gs = get(L, Go);
        if (have == 1 || (have == 2 && !diverged)) {
          double df = 0.0, mk = 0.0;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const double h = cabs(csub(gs.v[q], kept.v[q]));
            if (!(h <= df)) df = h > df ? h : __longlong_as_double(0x7ff0000000000000LL);
            mk = fmax(mk, cabs(kept.v[q]));
          }
          df = cta_max_nan<M>(df, sh.red[0]);
          mk = cta_max_nan<M>(mk, sh.red[1]);
          __syncthreads();
          if (df <= 1e-2 * mk) {
            if (diverged) {
              put(L, Go, kept);
              cyc = kept_cyc;
            }
            break;
          }
        }
        if (att < kDecRetries && (!diverged || !have)) {
          kept = gs;
          have = diverged || !done ? 2 : 1;
          kept_cyc = cyc;
        }
      }
      if (att >= kDecRetries) {
        cyc = a.sgf_max_iter + 1;
        put_st(NEGF_B200_ERR_NOT_CONVERGED);
        break;
      }
      __syncthreads();
    }
    ncyc += cyc;
    // ---- Sigma = Tlc gs Tcl
    const double2 ec = make_double2(E, a.eta);
    const double2* hmc = d.hmc + d.omc[c];
    const double2* smc = d.has_smc ? d.smc + d.omc[c] : nullptr;
    load_esh<M>(n, Bo, hmc, smc, ec, false, false);
    load_esh<M>(n, Co, hmc, smc, cconj(ec), false, true);
    __syncthreads();
    put(L, X, mm(L, Bo, Go));
    __syncthreads();
    Frag sig = mm(L, X, Co);
    if (side == rank) put(L, SL, sig);
    if (pair) {
      // one contact per CTA: CTA 0 goes on with both
      if (threadIdx.x == 0) {
        sh.ncyc = ncyc;
        sh.st = st;
      }
      team_sync();
      if (rank == 0) {
        sig = team_get(L, SL, 1);
        ncyc += team_ld_int(&sh.ncyc, 1);
        put_st(team_ld_int(&sh.st, 1));
      }
      team_sync();   // CTA 1's shared memory is read
      if (rank == 1) return;
    }
    if (side == 1 || pair) {
      // W = ESH(nbl, nbl) - Sigma_right
      load_esh<M>(n, Ao, d.hd + d.od[a.nbl - 1], d.has_s ? d.sd + d.od[a.nbl - 1] : nullptr, make_double2(E, 0.0), true,
               false);
      __syncthreads();
      sub_from(L, Ao, sig);
    }
    __syncthreads();
  }
  // ---- gsmr sweep down to Gr(1,1): g in Go
  if (small_inverse<M>(n) & 1) put_st(NEGF_B200_ERR_SINGULAR);
#pragma unroll 1
  for (int i = a.nbl - 2; i >= 0; --i) {
    const double2 e = make_double2(E, 0.0);
    __syncthreads();
    load_esh<M>(n, Bo, d.hu + d.oo[i], d.has_s ? d.su + d.oo[i] : nullptr, e, false, false);
    load_esh<M>(n, Co, d.hl + d.oo[i], d.has_s ? d.sl + d.oo[i] : nullptr, e, false, false);
    load_esh<M>(n, Ao, d.hd + d.od[i], d.has_s ? d.sd + d.od[i] : nullptr, e, true, false);
    __syncthreads();
    put(L, X, mm(L, Bo, Go));
    if (i == 0) sub_from(L, Ao, get(L, SL));
    __syncthreads();
    sub_from(L, Ao, mm(L, X, Co));
    __syncthreads();
    if (small_inverse<M>(n) & 1) put_st(NEGF_B200_ERR_SINGULAR);
  }
  __syncthreads();
  // ---- Gamma = i (Sigma - Sigma^dag) of the left contact, then the trace
  //   T = |Re Tr[Gam i(G - G^dag)] - Re Tr[Gam G Gam G^dag]|,
  //   Tr[Gam G Gam G^dag] = sum (Gam G)_ij conj(G Gam)_ij
  double t1 = 0.0, t2 = 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (L.in(q)) {
      const int i = L.row(q), j = L.col(q);
      const double2 s = SL[i + j * kLd], u = SL[j + i * kLd];
      const double2 gam = make_double2(-(s.y + u.y), s.x - u.x);
      Bo[i + j * kLd] = gam;
      const double2 gji = Go[j + i * kLd], gij = Go[i + j * kLd];
      t1 += gam.x * -(gji.y + gij.y) - gam.y * (gji.x - gij.x);   // Re(Gam_ij i (G_ji - conj G_ij))
    }
  __syncthreads();
  const Frag gg = mm(L, Bo, Go), hh = mm(L, Go, Bo);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (L.in(q)) t2 += gg.v[q].x * hh.v[q].x + gg.v[q].y * hh.v[q].y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t1 += __shfl_xor_sync(kFull, t1, o);
    t2 += __shfl_xor_sync(kFull, t2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sh.red[0][threadIdx.x >> 5] = t1;
    sh.red[1][threadIdx.x >> 5] = t2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    t1 = t2 = 0.0;
    for (int w = 0; w < Shape<M>::kWarps; ++w) {
      t1 += sh.red[0][w];
      t2 += sh.red[1][w];
    }
    const double T = fabs(t1 - t2);
    a.d_T[p] = T;
    if (a.d_ncyc) a.d_ncyc[p] = ncyc;
    // a non-finite T that no step flagged (NaN in the device blocks) is reported as such
    if (a.d_status) a.d_status[p] = (st == NEGF_B200_OK && !isfinite(T)) ? NEGF_B200_ERR_NONFINITE : st;
  }
}

template <int M>
cudaError_t launch(const MixedArgs& a, cudaStream_t s) {
  // Two CTAs per point, a contact each, while they find room at once: order
  // 32, 74 points: 1.34 ms by one CTA, 0.96 by two; 148 points (two CTAs per
  // SM): 1.35 and 1.22; 149: 1.71 and 2.00.
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = team_config(a.npts, a.npts <= device_sms() ? 2 : 1, small_smem<M>(), s, &attr);
  cfg.blockDim = dim3(Shape<M>::kCta);
  const cudaError_t e = team_launch(cfg, k_small_point<M>, small_smem<M>(), a);
  if (e == cudaSuccess && a.launches) ++*a.launches;
  return e;
}

}  // namespace

cudaError_t launch_small_points(const MixedArgs& a, cudaStream_t s) {
  if (a.npts <= 0) return cudaSuccess;
  if (a.n < 1 || a.n > kSmallMax) return cudaErrorInvalidValue;
  return a.n <= 16 ? launch<16>(a, s) : launch<32>(a, s);
}

}  // namespace negf
