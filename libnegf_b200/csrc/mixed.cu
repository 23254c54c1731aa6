// Mixed-precision transmission solve (north-star precision form): the
// 2-contact fast path of calculate_transmissions (src/iterative.F90:1697-1713)
// for a batch of (E, k) points moved through the same steps together, so
// that every block product is one batched product on the integer tensor
// cores (launch_ozaki_zgemm: int8 digits, exact int32 accumulation, FP64
// recombination) and every block inverse one batched FP64 Gauss-Jordan
// inversion (launch_zinv_mapped).  FP64 throughout outside the products: the
// decimation's convergence test on max|C1|, the inverses, and the Caroli
// trace (whose two products are FP64 tensor-core products).
//
// Steps per batch, following the reference routine by routine (the contacts
// of every point are problems of their own in the first two):
//   surface_green + decimation      src/contselfenergy.F90:184-210, 271-340
//     (lock step over the points still iterating; a point leaves the active
//     set on its second consecutive max|C1| <= SGFACC, as the CPU rule)
//   compute_contacts / SelfEnergy   src/contselfenergy.F90:445-491, 552-566
//   build_ESH (ESH at the real E)   src/iterative.F90:1956-1982
//   calculate_gsmr_blocks(nbl, 2)   src/iterative_cpu.F90:51-124
//   Gr(1,1)                         src/iterative_cpu.F90:134-170
//   calculate_single_transmission_2_contacts   src/iterative_cpu.F90:399-470
#include <algorithm>
#include <vector>

#include "../../include/negf_b200.h"
#include "mixed.cuh"
#include "ozaki.cuh"

namespace negf {
namespace {

// n x n complex work blocks per problem (contact of a point); where a point's
// contacts run one after the other the 12th keeps the left self-energy
constexpr int kBlocks = 11, kBlocksMax = 12;

__device__ __forceinline__ double2 cmulm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 conjm(double2 a) { return make_double2(a.x, -a.y); }

// Ao = Ec S00 - H00, Aos = Ao, Bo = Ec S01 - H01, Co = (conj(Ec) S01 - H01)^dag,
// Ec = (E + i eta) scale, for the problems map[b] (map null: b); problem p <
// P is contact `left` of point p, problem P + p contact `right`
__global__ void k_lead_init(int n, int P, int left, int right, const int* ids, const double* E, double eta,
                            double scale, const int* map, const DevDesc* descs, double2* Ao, double2* Aos, double2* Bo,
                            double2* Co, int64_t Q) {
  const int p = map ? map[blockIdx.y] : blockIdx.y;
  const int pt = p < P ? p : p - P, c = p < P ? left : right;
  const DevDesc& d = descs[ids[pt]];
  const double2 ec = make_double2(E[pt] * scale, eta * scale);
  const int64_t ol = d.olead[c], nn = (int64_t)n * n;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % n), j = (int)(q / n);
    const int64_t qt = j + (int64_t)i * n;   // element (j, i)
    const double2 s00 = d.has_s00 ? d.s00[ol + q] : make_double2(i == j ? 1.0 : 0.0, 0.0);
    const double2 h00 = d.h00[ol + q];
    const double2 s01 = d.has_s01 ? d.s01[ol + q] : make_double2(0.0, 0.0);
    const double2 h01 = d.h01[ol + q];
    const double2 s01t = d.has_s01 ? d.s01[ol + qt] : make_double2(0.0, 0.0);
    const double2 h01t = d.h01[ol + qt];
    double2 a = cmulm(ec, s00);
    a.x -= h00.x; a.y -= h00.y;
    double2 b = cmulm(ec, s01);
    b.x -= h01.x; b.y -= h01.y;
    double2 ct = cmulm(conjm(ec), s01t);
    ct.x -= h01t.x; ct.y -= h01t.y;
    Ao[p * Q + q] = a;
    Aos[p * Q + q] = a;
    Bo[p * Q + q] = b;
    Co[p * Q + q] = conjm(ct);
  }
}

// Ao -= Self, Aos -= Self for the points of the list
__global__ void k_sub_self(int64_t nn, const int* list, const double2* Self, double2* Ao,
                           double2* Aos, int64_t Q) {
  const int p = list[blockIdx.y];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const double2 s = Self[p * Q + q];
    double2 a = Ao[p * Q + q], b = Aos[p * Q + q];
    a.x -= s.x; a.y -= s.y;
    b.x -= s.x; b.y -= s.y;
    Ao[p * Q + q] = a;
    Aos[p * Q + q] = b;
  }
}

// The CPU convergence rule (src/contselfenergy.F90:300-310): a point is done
// on its second consecutive max|C1| <= tol.  Builds the list of the points
// that go on (and zeroes their max for the next iteration).  One CTA.
__global__ void k_dec_check(int na, const int* list, double* mx, int* ok, int* ncyc_c, double tol,
                            int it, int* next, int* next_count, int* redo) {
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  for (int b = threadIdx.x; b < na; b += blockDim.x) {
    const int p = list[b];
    const double m = mx[p];
    bool go = true;
    if (!(m <= 1.7976931348623157e308)) {   // Inf / NaN: this decimation will not converge; run it again
      go = false;
      ncyc_c[p] = it;
      redo[p] = 2;
    } else if (m <= tol) {
      if (ok[p]) {
        go = false;
        ncyc_c[p] = it;
      }
      ok[p] = 1;
    } else {
      ok[p] = 0;
    }
    if (go) {
      next[atomicAdd(&cnt, 1)] = p;
      mx[p] = 0.0;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *next_count = cnt;
}

__global__ void k_info_to_status(int nb, const int* list, const int* info, int* status, int code) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
    const int p = list ? list[b] : b;
    if (info[p] != 0 && status[p] == 0) status[p] = code;
  }
}

// Tlc = Ec SMC - HMC (n x L), Tcl = (conj(Ec) SMC - HMC)^dag (L x n); here L =
// n.  Problems as in k_lead_init.
__global__ void k_tlc(int n, int P, int left, int right, const int* ids, const double* E, double eta,
                      const DevDesc* descs, double2* Tlc, double2* Tcl, int64_t Q) {
  const int p = blockIdx.y;
  const int pt = p < P ? p : p - P, c = p < P ? left : right;
  const DevDesc& d = descs[ids[pt]];
  const double2 ec = make_double2(E[pt], eta);
  const int64_t om = d.omc[c], nn = (int64_t)n * n;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % n), j = (int)(q / n);
    const int64_t qt = j + (int64_t)i * n;
    const double2 smc = d.has_smc ? d.smc[om + q] : make_double2(0.0, 0.0);
    const double2 hmc = d.hmc[om + q];
    double2 t = cmulm(ec, smc);
    t.x -= hmc.x; t.y -= hmc.y;
    const double2 smct = d.has_smc ? d.smc[om + qt] : make_double2(0.0, 0.0);
    const double2 hmct = d.hmc[om + qt];
    double2 u = cmulm(conjm(ec), smct);
    u.x -= hmct.x; u.y -= hmct.y;
    Tlc[p * Q + q] = t;
    Tcl[p * Q + q] = conjm(u);
  }
}

// ESH blocks at the real energy: which 0 = (i,i) minus sig (if given),
// 1 = (i,i+1), 2 = (i+1,i); i 0-based
__global__ void k_esh(int n, int which, int i, const int* ids, const double* E, const DevDesc* descs,
                      const double2* sig, double2* out, int64_t Q) {
  const int p = blockIdx.y;
  const DevDesc& d = descs[ids[p]];
  const double e = E[p];
  const int64_t nn = (int64_t)n * n;
  const int64_t off = (which == 0) ? d.od[i] : d.oo[i];
  const double2* H = (which == 0) ? d.hd : (which == 1 ? d.hu : d.hl);
  const double2* S = (which == 0) ? d.sd : (which == 1 ? d.su : d.sl);
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const double2 h = H[off + q];
    double2 v;
    if (d.has_s) {
      const double2 sv = S[off + q];
      v = make_double2(e * sv.x - h.x, e * sv.y - h.y);
    } else {
      v = make_double2(-h.x, -h.y);
      if (which == 0 && (q % n) == (q / n)) v.x += e;
    }
    if (sig) {
      const double2 sg = sig[p * Q + q];
      v.x -= sg.x; v.y -= sg.y;
    }
    out[p * Q + q] = v;
  }
}

// The three ESH blocks of one sweep step in one pass: U = ESH(i,i+1),
// L = ESH(i+1,i), W = ESH(i,i) - sig (sig may be null)
__global__ void k_esh_step(int n, int i, const int* ids, const double* E, const DevDesc* descs, const double2* sig,
                           double2* U, double2* Lo, double2* W, int64_t Q) {
  const int p = blockIdx.y;
  const DevDesc& d = descs[ids[p]];
  const double e = E[p];
  const int64_t nn = (int64_t)n * n;
  const int64_t od = d.od[i], oo = d.oo[i];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const double2 hu = d.hu[oo + q], hl = d.hl[oo + q], hd = d.hd[od + q];
    double2 u, l, w;
    if (d.has_s) {
      const double2 su = d.su[oo + q], sl = d.sl[oo + q], sd = d.sd[od + q];
      u = make_double2(e * su.x - hu.x, e * su.y - hu.y);
      l = make_double2(e * sl.x - hl.x, e * sl.y - hl.y);
      w = make_double2(e * sd.x - hd.x, e * sd.y - hd.y);
    } else {
      u = make_double2(-hu.x, -hu.y);
      l = make_double2(-hl.x, -hl.y);
      w = make_double2(-hd.x, -hd.y);
      if ((q % n) == (q / n)) w.x += e;
    }
    if (sig) {
      const double2 sg = sig[p * Q + q];
      w.x -= sg.x; w.y -= sg.y;
    }
    U[p * Q + q] = u;
    Lo[p * Q + q] = l;
    W[p * Q + q] = w;
  }
}

// Gamma = i (Sigma - Sigma^dag)   (zspectral_dns, src/sparsekit_drv.F90:2870-2890)
__global__ void k_gamma(int n, const double2* Sig, double2* Gam, int64_t Q) {
  const int p = blockIdx.y;
  const int64_t nn = (int64_t)n * n;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % n), j = (int)(q / n);
    const double2 a = Sig[p * Q + q], b = Sig[p * Q + j + (int64_t)i * n];
    // i * (a - conj(b))
    Gam[p * Q + q] = make_double2(-(a.y + b.y), a.x - b.x);
  }
}

// T = |Re Tr[Gam i(G - G^dag)] - Re Tr[Gam G Gam G^dag]|
//   Tr[Gam A]            = sum_ij Gam_ij i (G_ji - conj(G_ij))
//   Tr[Gam G Gam G^dag]  = sum_ij M_ij conj(N_ij),  M = Gam G, N = G Gam
// (calculate_single_transmission_2_contacts, src/iterative_cpu.F90:424-464).
// One CTA per point; FP64.
__global__ void k_trace(int n, const double2* Gam, const double2* G, const double2* M, const double2* N, double* T,
                        int64_t Q) {
  const int p = blockIdx.x;
  const int64_t nn = (int64_t)n * n;
  double t1 = 0.0, t2 = 0.0;
  for (int64_t q = threadIdx.x; q < nn; q += blockDim.x) {
    const int i = (int)(q % n), j = (int)(q / n);
    const double2 g = Gam[p * Q + q];
    const double2 gji = G[p * Q + j + (int64_t)i * n], gij = G[p * Q + q];
    // A_ji = i (G_ji - conj(G_ij))
    const double2 aji = make_double2(-(gji.y + gij.y), gji.x - gij.x);
    t1 += g.x * aji.x - g.y * aji.y;
    const double2 m = M[p * Q + q], nq = N[p * Q + q];
    t2 += m.x * nq.x + m.y * nq.y;   // Re(m conj(n))
  }
  __shared__ double r1[32], r2[32];
  for (int o = 16; o > 0; o >>= 1) {
    t1 += __shfl_xor_sync(0xffffffffu, t1, o);
    t2 += __shfl_xor_sync(0xffffffffu, t2, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { r1[w] = t1; r2[w] = t2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s1 = 0.0, s2 = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { s1 += r1[k]; s2 += r2[k]; }
    T[p] = fabs(s1 - s2);
  }
}

// Points whose surface Green's function left the retarded solution (eta > 0,
// sgn = -1; the advanced one for eta < 0, sgn = 1): the diagonal of sgn Im gs
// must be >= 0 (up to 1e-6 of the largest |gs_ii|); a
// converged fixed point of the wrong kind, or one that is not finite, marks
// the point for the engine (redo[p] = 1).  One CTA per point.
__global__ void k_retarded_check(int n, const double2* gs, int64_t Q, double sgn, const int* map, int* redo) {
  const int p = map ? map[blockIdx.x] : blockIdx.x;
  double lo = 1.7976931348623157e308, hi = 0.0;
  int bad = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double2 g = gs[p * Q + (int64_t)i * (n + 1)];
    const double v = sgn * g.y, h = sqrt(g.x * g.x + g.y * g.y);
    if (!(h <= 1.7976931348623157e308)) bad = 1;
    else {
      lo = fmin(lo, v);
      hi = fmax(hi, h);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  bad = __any_sync(0xffffffffu, bad);
  __shared__ double slo[32], shi[32];
  __shared__ int sbad[32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { slo[w] = lo; shi[w] = hi; sbad[w] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
      lo = fmin(lo, slo[q]);
      hi = fmax(hi, shi[q]);
      bad |= sbad[q];
    }
    if (bad || (hi > 0.0 && lo < -1e-6 * hi)) redo[p] = 1;
  }
}

// Start of a decimation for the points map[b], b < nsub (map null: b):
// ok = 0, max = 0, ncyc = 0, sensitivity 0, the active list = the points.
__global__ void k_dec_start(int nsub, const int* map, int* ok, double* mx, int* ncyc_c, int* list, int* sens) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nsub; b += gridDim.x * blockDim.x) {
    const int p = map ? map[b] : b;
    ok[p] = 0;
    sens[p] = 0;
    mx[p] = 0.0;
    ncyc_c[p] = 0;
    list[b] = p;
  }
}

// kept_p = gs_p (or back) for the points map[b], b < nsub; one CTA per point.
__global__ void k_keep(int64_t nn, const int* map, const double2* gs, double2* kept, int64_t Q) {
  const int p = map[blockIdx.x];
  for (int64_t q = threadIdx.x; q < nn; q += blockDim.x) kept[p * Q + q] = gs[p * Q + q];
}

// agree[p] = max |gs_p - kept_p| <= tol max |kept_p| for the points map[b]; one CTA per point.
__global__ void k_agree(int64_t nn, const int* map, const double2* gs, const double2* kept, int64_t Q, double tol,
                        int* agree) {
  const int p = map[blockIdx.x];
  double d = 0.0, m = 0.0;
  for (int64_t q = threadIdx.x; q < nn; q += blockDim.x) {
    const double2 a = gs[p * Q + q], b = kept[p * Q + q];
    const double h = hypot(a.x - b.x, a.y - b.y);
    if (!(h <= d)) d = h > d ? h : __longlong_as_double(0x7ff0000000000000LL);   // NaN agrees with nothing
    m = fmax(m, hypot(b.x, b.y));
  }
  for (int o = 16; o > 0; o >>= 1) {
    d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  __shared__ double sd[32], sm[32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { sd[w] = d; sm[w] = m; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) { d = fmax(d, sd[q]); m = fmax(m, sm[q]); }
    agree[p] = (d <= tol * m) ? 1 : 0;
  }
}

// Problems still flagged after the last attempt: NOT_CONVERGED, ncyc = cap + 1.
__global__ void k_flag_unresolved(int P, const int* redo, int* ncyc_c, int* status, int max_iter) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x)
    if (redo[p]) {
      ncyc_c[p] = max_iter + 1;
      if (status[p] == 0) status[p] = NEGF_B200_ERR_NOT_CONVERGED;
    }
}


size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Carver {
  char* p;
  size_t off = 0;
  template <typename T>
  T* take(size_t n) {
    T* r = p ? reinterpret_cast<T*>(p + off) : nullptr;
    off = align256(off + n * sizeof(T));
    return r;
  }
};

struct Ws {
  double2* blk[kBlocksMax];
  double* mx;
  int *ok, *nc, *list0, *list1, *count, *info, *pst, *pst2, *redo, *sub, *sens, *agree;
  double* tb;
  double2* zwork;
  OzakiSet rows[3], cols;      // digits of three left operands (one after the other in the same place
                               // where the contacts run one by one) and a right one
  double* t0;
};

Ws carve(void* base, int P, int n, int slices, bool one_contact, size_t* total) {
  Carver c{static_cast<char*>(base)};
  Ws w;
  // problems at a time: the contacts of every point, or one contact of it
  const size_t Q = (size_t)n * n, N = (one_contact ? 1 : 2) * (size_t)P;
  for (int b = 0; b < (one_contact ? kBlocksMax : kBlocks); ++b) w.blk[b] = c.take<double2>(N * Q);
  w.mx = c.take<double>(N);
  w.ok = c.take<int>(N);
  w.nc = c.take<int>(2 * (size_t)P);
  w.list0 = c.take<int>(N);
  w.list1 = c.take<int>(N);
  w.count = c.take<int>(4);
  w.info = c.take<int>(N);
  w.pst = c.take<int>(P);
  w.pst2 = c.take<int>(2 * (size_t)P);
  w.tb = c.take<double>(P);
  w.redo = c.take<int>(N);
  w.sub = c.take<int>(N);
  w.sens = c.take<int>(N);
  w.agree = c.take<int>(N);
  w.zwork = c.take<double2>(N * zinv_batched_work_elems(n) + 1);
  uint8_t* q = nullptr;
  for (int i = 0; i < 3; ++i) {
    if (i == 0 || !one_contact) q = c.take<uint8_t>(ozaki_rows_bytes((int)N, n, n, slices));
    if (base) w.rows[i] = ozaki_rows_at(q, (int)N, n, n, slices);
  }
  q = c.take<uint8_t>(ozaki_cols_bytes((int)N, n, n, slices));
  if (base) w.cols = ozaki_cols_at(q, (int)N, n, n, slices);
  w.t0 = c.take<double>(N * Q);
  *total = c.off + 256;
  return w;
}

// The status of a point after its two decimations: a product's code (3, 7) of
// the right one, else the left one's, else the right one's.
__global__ void k_merge_status(int P, const int* both, int* pst) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const int l = both[p], r = both[P + p];
    pst[p] = (r == NEGF_B200_ERR_NONFINITE || r == NEGF_B200_ERR_TIMEOUT || l == 0) ? r : l;
  }
}

__global__ void k_finish(int P, const int* ncl, const int* ncr, const int* pst, const double* Tb, double* T,
                         int* ncyc, int* status) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    T[p] = Tb[p];
    if (ncyc) ncyc[p] = ncl[p] + ncr[p];
    // a non-finite T that no step flagged (NaN in the device blocks) is reported as such
    if (status) status[p] = (pst[p] == 0 && !isfinite(Tb[p])) ? NEGF_B200_ERR_NONFINITE : pst[p];
  }
}

__global__ void k_not_converged(int na, const int* list, int* ncyc_c, int* pst, int max_iter) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < na; b += gridDim.x * blockDim.x) {
    const int p = list[b];
    ncyc_c[p] = max_iter + 1;
    if (pst[p] == 0) pst[p] = NEGF_B200_ERR_NOT_CONVERGED;
  }
}

}  // namespace

size_t mixed_ws_bytes(int batch, int n, int slices, bool one_contact) {
  size_t t = 0;
  carve(nullptr, batch, n, slices, one_contact, &t);
  return t;
}

int mixed_batch_for(size_t bytes, int n, int slices) {
  int lo = 0, hi = 1 << 14;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (mixed_ws_bytes(mid, n, slices, false) <= bytes) lo = mid; else hi = mid - 1;
  }
  return lo;
}

int mixed_run(const MixedArgs& a, void* ws, int batch, bool one_contact, cudaStream_t s, std::string* err) {
  const int n = a.n;
  const int64_t Q = (int64_t)n * n;
  const double2 one = make_double2(1, 0), zero = make_double2(0, 0), mone = make_double2(-1, 0);
  size_t tot = 0;
  Ws w = carve(ws, batch, n, a.slices, one_contact, &tot);
  double2** B = w.blk;
  const dim3 eb(256);
  const int gx = (int)std::min<int64_t>(64, (Q + 255) / 256);
  auto ck = [&](cudaError_t e, const char* what) -> int {
    if (e == cudaSuccess) return 0;
    if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
    return NEGF_B200_ERR_CUDA;
  };
#define MCK(x, what)             \
  do {                           \
    int r_ = ck((x), what);      \
    if (r_) return r_;           \
  } while (0)
  // Products and inverses of the problems map[b], b < nb.  An operand is split
  // into digits once for all the products it takes part in: of a decimation
  // iteration's six products, three left and four right operands.
  uint64_t nl = 0;                 // kernels launched (reported through a.launches)
  // Where the contacts run one by one the left operands share one place and are
  // split when a product needs another one than the place holds.
  const double2* left_of[3] = {nullptr, nullptr, nullptr};
  int held = -1;
  auto rows = [&](int nb, const int* map, const double2* A, int set) -> cudaError_t {
    if (one_contact) {
      left_of[set] = A;
      if (held == set) held = -1;
      return cudaSuccess;
    }
    ++nl;
    return launch_ozaki_rows(nb, n, n, A, Q, a.slices, w.rows[set], s, map);
  };
  auto cols = [&](int nb, const int* map, const double2* Bm) -> cudaError_t {
    ++nl;
    return launch_ozaki_cols(nb, n, n, Bm, Q, a.slices, w.cols, s, map);
  };
  auto prod = [&](int nb, const int* map, double2 alpha, int set, double2 beta, double2* C, double* maxabs,
                  int* status) -> cudaError_t {
    if (one_contact && held != set) {
      ++nl;
      const cudaError_t e = launch_ozaki_rows(nb, n, n, left_of[set], Q, a.slices, w.rows[set], s, map);
      if (e != cudaSuccess) return e;
      held = set;
    }
    ++nl;
    return launch_ozaki_product(nb, n, n, n, alpha, w.rows[set], w.cols, beta, C, Q, a.slices, w.t0, maxabs, status,
                                s, map);
  };
  auto inv = [&](int nb, const int* map, const double2* A, double2* X) -> cudaError_t {
    ++nl;
    return launch_zinv_mapped(nb, n, A, Q, X, Q, map, w.info, w.zwork, s, w.sens);   // probe and refinement inside
  };
  // FP64 products of the trace
  auto prod64 = [&](int nb, const double2* A, const double2* Bm, double2* C) -> cudaError_t {
    ++nl;
    return launch_zgemm_batched(nb, n, n, n, one, A, Q, Bm, Q, zero, C, Q, 0, s);
  };

  for (int p0 = 0; p0 < a.npts; p0 += batch) {
    const int P = std::min(batch, a.npts - p0), N = one_contact ? P : 2 * P;
    const int* ids = a.d_ids + p0;
    const double* E = a.d_E + p0;
    MCK(cudaMemsetAsync(w.pst2, 0, sizeof(int) * 2 * P, s), "memset status");
    for (int side = 0; side < (one_contact ? 2 : 1); ++side) {
      const int cl = side == 0 ? a.left : a.right, cr = one_contact ? cl : a.right;
      int *nc = w.nc + (int64_t)side * P, *pst2 = w.pst2 + (int64_t)side * P;
      double2 *gs = B[9], *sig = B[10], *kept_gs = B[10];   // (a kept gs is done with before the self-energies)
      // ---- surface Green's functions of both contacts of every point (problem
      // p: left contact of point p, P + p: right; or those of one contact), all
      // in lock step.
      // Decimation of the problems sub[b], b < nsub (sub null: all N), the
      // contact energy scaled by `scale`; then gs = Aos^-1 and the
      // retarded-branch check (redo[p] = 1 where it fails, 2 where only the
      // iteration ran off)
      auto decimate = [&](const int* sub, int nsub, double scale) -> int {
        double2 *Ao = B[0], *Aos = B[1], *Bo = B[2], *Co = B[3], *Go = B[4], *X = B[5], *C1 = B[6], *Y = B[7],
                *B1 = B[8];
        k_lead_init<<<dim3(gx, nsub), eb, 0, s>>>(n, P, cl, cr, ids, E, a.eta, scale, sub, a.d_descs, Ao, Aos,
                                                  Bo, Co, Q);
        ++nl;
        MCK(cudaGetLastError(), "lead init");
        k_dec_start<<<(nsub + 255) / 256, 256, 0, s>>>(nsub, sub, w.ok, w.mx, nc, w.list0, w.sens);
        ++nl;
        int na = nsub;                                   // host bound of the active list
        int* cur = w.list0;
        int* nxt = w.list1;
        int it = 1;
        for (; it <= a.sgf_max_iter && na > 0; ++it) {
          // one batched product per step, the active list compacted on the host
          MCK(inv(na, cur, Ao, Go), "zinv");
          k_info_to_status<<<(na + 255) / 256, 256, 0, s>>>(na, cur, w.info, pst2, NEGF_B200_ERR_SINGULAR);
          ++nl;
          MCK(rows(na, cur, Go, 0), "split Go");
          MCK(cols(na, cur, Co), "split Co");
          MCK(prod(na, cur, one, 0, zero, X, nullptr, pst2), "GoXCo");
          MCK(rows(na, cur, Co, 1), "split Co");
          MCK(cols(na, cur, X), "split X");
          MCK(prod(na, cur, one, 1, zero, C1, w.mx, pst2), "C1");
          k_dec_check<<<1, 1024, 0, s>>>(na, cur, w.mx, w.ok, nc, a.sgf_tol, it, nxt, w.count, w.redo);
          ++nl;
          MCK(cudaGetLastError(), "check");
          std::swap(cur, nxt);
          {
            int h_count = 0;
            MCK(cudaMemcpyAsync(&h_count, w.count, sizeof(int), cudaMemcpyDeviceToHost, s), "count");
            MCK(cudaStreamSynchronize(s), "sync");
            na = h_count;
            if (na == 0) break;
          }
          MCK(rows(na, cur, Bo, 2), "split Bo");
          MCK(prod(na, cur, one, 2, zero, B1, nullptr, pst2), "Self");
          k_sub_self<<<dim3(gx, na), eb, 0, s>>>(Q, cur, B1, Ao, Aos, Q); ++nl;
          MCK(cols(na, cur, Bo), "split Bo");
          MCK(prod(na, cur, one, 0, zero, Y, nullptr, pst2), "GoXBo");
          MCK(cols(na, cur, Y), "split Y");
          MCK(prod(na, cur, one, 2, zero, B1, nullptr, pst2), "B1");
          MCK(prod(na, cur, mone, 1, one, Ao, nullptr, pst2), "Ao update");
          // Bo = B1, Co = C1 for every problem still iterating (the others are done with them)
          std::swap(B[2], B[8]);
          std::swap(B[3], B[6]);
          Bo = B[2]; Co = B[3]; B1 = B[8]; C1 = B[6];
        }
        if (na > 0) {
          k_not_converged<<<(na + 255) / 256, 256, 0, s>>>(na, cur, nc, pst2, a.sgf_max_iter);
          ++nl;
        }
        MCK(inv(nsub, sub, Aos, gs), "gs");
        k_info_to_status<<<(nsub + 255) / 256, 256, 0, s>>>(nsub, sub, w.info, pst2, NEGF_B200_ERR_SINGULAR);
        ++nl;
        if (a.eta != 0.0) {
          k_retarded_check<<<nsub, 128, 0, s>>>(n, gs, Q, a.eta > 0.0 ? -1.0 : 1.0, sub, w.redo);
          ++nl;
        }
        return 0;
      };
      MCK(cudaMemsetAsync(w.redo, 0, sizeof(int) * N, s), "memset redo");
      if (int r = decimate(nullptr, N, 1.0)) return r;
      if (a.eta != 0.0) {
        // Decimations that reached another fixed point (or ran off to Inf / NaN) run
        // again, in lock step over just those problems, from the contact energy times
        // 1 + k 2^-50.  A sensitive decimation (one of its inverses needed a Newton
        // step: a nearly singular Ao) is accepted once two attempts reach the same gs.
        // An attempt that ran off (redo 2) with a gs on the right branch is none to
        // accept, but one to agree with a converged attempt's, kept before or still
        // to come.  kept: 1 a converged attempt's gs, of kept_nc iterations, 2 any
        // other's.
        std::vector<int> hredo(N), hsens(N), hagree(N), hnc(N), kept(N, 0), kept_nc(N), cur_sub, again, cmp, keep, take;
        cur_sub.resize(N);
        for (int p = 0; p < N; ++p) cur_sub[p] = p;
        for (int att = 1;; ++att) {
          MCK(cudaMemcpyAsync(hredo.data(), w.redo, sizeof(int) * N, cudaMemcpyDeviceToHost, s), "redo");
          MCK(cudaMemcpyAsync(hsens.data(), w.sens, sizeof(int) * N, cudaMemcpyDeviceToHost, s), "sens");
          MCK(cudaMemcpyAsync(hnc.data(), nc, sizeof(int) * N, cudaMemcpyDeviceToHost, s), "ncyc");
          MCK(cudaStreamSynchronize(s), "sync");
          cmp.clear();
          for (int p : cur_sub)
            if (kept[p] && ((!hredo[p] && hsens[p]) || (hredo[p] == 2 && kept[p] == 1))) cmp.push_back(p);
          if (!cmp.empty()) {
            MCK(cudaMemcpyAsync(w.sub, cmp.data(), sizeof(int) * cmp.size(), cudaMemcpyHostToDevice, s), "cmp");
            k_agree<<<(int)cmp.size(), 256, 0, s>>>(Q, w.sub, gs, kept_gs, Q, 1e-2, w.agree); ++nl;
            MCK(cudaMemcpyAsync(hagree.data(), w.agree, sizeof(int) * N, cudaMemcpyDeviceToHost, s), "agree");
            MCK(cudaStreamSynchronize(s), "sync");
          }
          again.clear();
          keep.clear();
          take.clear();
          for (int p : cur_sub) {
            if (hredo[p] == 2 && kept[p] == 1 && hagree[p]) {                 // the kept gs is accepted
              take.push_back(p);
              hredo[p] = 0;
              hnc[p] = kept_nc[p];
              continue;
            }
            if (hredo[p]) {                                                   // wrong fixed point: run again
              again.push_back(p);
              if (hredo[p] == 2 && !kept[p]) keep.push_back(p);
              continue;
            }
            if (!hsens[p]) continue;                                          // settled
            if (kept[p] && hagree[p]) continue;                               // two attempts agree
            keep.push_back(p);                                                // keep this gs, run again
            again.push_back(p);
          }
          if (!take.empty()) {
            MCK(cudaMemcpyAsync(w.sub, take.data(), sizeof(int) * take.size(), cudaMemcpyHostToDevice, s), "take");
            k_keep<<<(int)take.size(), 256, 0, s>>>(Q, w.sub, kept_gs, gs, Q); ++nl;
            MCK(cudaMemcpyAsync(nc, hnc.data(), sizeof(int) * N, cudaMemcpyHostToDevice, s), "ncyc");
            MCK(cudaStreamSynchronize(s), "sync");
          }
          if (again.empty()) break;
          if (att > kDecRetries) {
            for (int p : again) hredo[p] = 1;
            MCK(cudaMemcpyAsync(w.redo, hredo.data(), sizeof(int) * N, cudaMemcpyHostToDevice, s), "redo");
            k_flag_unresolved<<<(N + 255) / 256, 256, 0, s>>>(N, w.redo, nc, pst2, a.sgf_max_iter);
            ++nl;
            MCK(cudaStreamSynchronize(s), "sync");
            break;
          }
          if (!keep.empty()) {
            MCK(cudaMemcpyAsync(w.sub, keep.data(), sizeof(int) * keep.size(), cudaMemcpyHostToDevice, s), "keep");
            k_keep<<<(int)keep.size(), 256, 0, s>>>(Q, w.sub, gs, kept_gs, Q); ++nl;
            for (int p : keep) {
              kept[p] = hredo[p] == 2 || hnc[p] > a.sgf_max_iter ? 2 : 1;
              kept_nc[p] = hnc[p];
            }
          }
          MCK(cudaMemcpyAsync(w.sub, again.data(), sizeof(int) * again.size(), cudaMemcpyHostToDevice, s), "sub");
          MCK(cudaMemsetAsync(w.redo, 0, sizeof(int) * N, s), "memset redo");
          if (int r = decimate(w.sub, (int)again.size(), 1.0 + att * 0x1p-50)) return r;
          cur_sub = again;
          MCK(cudaStreamSynchronize(s), "sync");   // the host vectors above are reused next round
        }
      } else {   // no other branch to try; gs of an iteration broken off (Inf / NaN) means nothing
        k_flag_unresolved<<<(N + 255) / 256, 256, 0, s>>>(N, w.redo, nc, pst2, a.sgf_max_iter);
        ++nl;
      }
      // ---- self-energies Sigma_c = Tlc gs Tcl of both contacts
      k_tlc<<<dim3(gx, N), eb, 0, s>>>(n, P, cl, cr, ids, E, a.eta, a.d_descs, B[0], B[1], Q); ++nl;
      MCK(cudaGetLastError(), "tlc");
      MCK(rows(N, nullptr, B[0], 0), "split Tlc");
      MCK(cols(N, nullptr, gs), "split gs");
      MCK(prod(N, nullptr, one, 0, zero, B[2], nullptr, pst2), "Tlc gs");
      MCK(rows(N, nullptr, B[2], 0), "split Tlc gs");
      MCK(cols(N, nullptr, B[1]), "split Tcl");
      MCK(prod(N, nullptr, one, 0, zero, sig, nullptr, pst2), "Sigma");
      if (one_contact && side == 0) std::swap(B[10], B[11]);
    }
    k_merge_status<<<(P + 255) / 256, 256, 0, s>>>(P, w.pst2, w.pst); ++nl;
    const double2 *sig_l = one_contact ? B[11] : B[10], *sig_r = one_contact ? B[10] : B[10] + (int64_t)P * Q;
    // ---- gsmr sweep from block nbl down to 2, then Gr(1,1)
    double2 *g = B[4], *X = B[5], *W = B[6], *U = B[7], *Lb = B[8];
    k_esh<<<dim3(gx, P), eb, 0, s>>>(n, 0, a.nbl - 1, ids, E, a.d_descs, sig_r, W, Q); ++nl;
    MCK(inv(P, nullptr, W, g), "gsmr N");
    k_info_to_status<<<(P + 255) / 256, 256, 0, s>>>(P, nullptr, w.info, w.pst, NEGF_B200_ERR_SINGULAR);
    ++nl;
    for (int i = a.nbl - 2; i >= 0; --i) {
      // W = ESH(i,i) - ESH(i,i+1) gsmr(i+1) ESH(i+1,i)  (block i 0-based; Sigma_left on block 0)
      k_esh_step<<<dim3(gx, P), eb, 0, s>>>(n, i, ids, E, a.d_descs, i == 0 ? sig_l : nullptr, U, Lb, W, Q); ++nl;
      MCK(cudaGetLastError(), "esh");
      MCK(rows(P, nullptr, U, 0), "split U");
      MCK(cols(P, nullptr, g), "split g");
      MCK(prod(P, nullptr, one, 0, zero, X, nullptr, w.pst), "U g");
      MCK(rows(P, nullptr, X, 0), "split U g");
      MCK(cols(P, nullptr, Lb), "split L");
      MCK(prod(P, nullptr, mone, 0, one, W, nullptr, w.pst), "W");
      MCK(inv(P, nullptr, W, g), "gsmr");
      k_info_to_status<<<(P + 255) / 256, 256, 0, s>>>(P, nullptr, w.info, w.pst, NEGF_B200_ERR_SINGULAR);
      ++nl;
    }
    // g = Gr(1,1).  Trace with Gamma of the contact on block 1 (FP64 products)
    k_gamma<<<dim3(gx, P), eb, 0, s>>>(n, sig_l, B[0], Q); ++nl;
    MCK(prod64(P, B[0], g, B[1]), "Gam G");
    MCK(prod64(P, g, B[0], B[2]), "G Gam");
    k_trace<<<P, 512, 0, s>>>(n, B[0], g, B[1], B[2], w.tb, Q); ++nl;
    MCK(cudaGetLastError(), "trace");
    k_finish<<<(P + 255) / 256, 256, 0, s>>>(P, w.nc, w.nc + P, w.pst, w.tb, a.d_T + p0,
                                             a.d_ncyc ? a.d_ncyc + p0 : nullptr,
                                             a.d_status ? a.d_status + p0 : nullptr); ++nl;
    MCK(cudaGetLastError(), "finish");
  }
#undef MCK
  if (a.launches) *a.launches += nl;
  return NEGF_B200_OK;
}

}  // namespace negf
