// Gauss-Jordan panels (gj_panel, gj_leaf4) and row-owner node updates
// (gj_rows_update), compiled in a translation
// unit of their own (see gemm_run in cta_ops.cuh).
#include "cta_ops.cuh"

namespace negf {

__device__ void panel_run_w32(const double2* A, double2* X, int n, int c0, int w, InvScratch& s) {
  extern __shared__ __align__(16) char smem_raw[];
  gj_panel<1, 4, true>(A, n, X, n, n, c0, w, reinterpret_cast<double2*>(smem_raw), s);
}
__device__ void panel_run_w64(const double2* A, double2* X, int n, int c0, int w, InvScratch& s) {
  extern __shared__ __align__(16) char smem_raw[];
  gj_panel<2, 8, true>(A, n, X, n, n, c0, w, reinterpret_cast<double2*>(smem_raw), s);
}
__device__ void panel_run_4(const double2* src, double2* dst, int n, int c0, int w, InvScratch& s) {
  extern __shared__ __align__(16) char smem_raw[];
  gj_panel<4, 4, false>(src + (size_t)c0 * n, n, dst + (size_t)c0 * n, n, n, c0, w,
                        reinterpret_cast<double2*>(smem_raw), s);
}
__device__ void panel_run_8(const double2* src, double2* dst, int n, int c0, int w, InvScratch& s) {
  extern __shared__ __align__(16) char smem_raw[];
  gj_panel<8, 2, false>(src + (size_t)c0 * n, n, dst + (size_t)c0 * n, n, n, c0, w,
                        reinterpret_cast<double2*>(smem_raw), s);
}
__device__ void leaf_run_r2(double2* X, int n, int c0, int w, double2* sh, InvScratch& s) {
  gj_leaf4<2, 4>(X, n, c0, w, sh, s);
}
__device__ void leaf_run_r4(double2* X, int n, int c0, int w, double2* sh, InvScratch& s) {
  gj_leaf4<4, 2>(X, n, c0, w, sh, s);
}

__device__ void rows_run_t2(const double2* X, double2* Y, const double2* Wm, int n, int N, int k0, int K,
                            const int* perm, double2* stage) {
  gj_rows_update<1, 2, 8>(X, Y, Wm, n, N, k0, K, perm, stage);
}
__device__ void rows_run_r1(const double2* X, double2* Y, const double2* Wm, int n, int N, int k0, int K,
                            const int* perm, double2* stage) {
  gj_rows_update<1, 1, 16>(X, Y, Wm, n, N, k0, K, perm, stage);
}
__device__ void rows_run_r2(const double2* X, double2* Y, const double2* Wm, int n, int N, int k0, int K,
                            const int* perm, double2* stage) {
  gj_rows_update<2, 1, 16>(X, Y, Wm, n, N, k0, K, perm, stage);
}
__device__ void rows_run_r4(const double2* X, double2* Y, const double2* Wm, int n, int N, int k0, int K,
                            const int* perm, double2* stage) {
  gj_rows_update<4, 1, 8>(X, Y, Wm, n, N, k0, K, perm, stage);
}
__device__ void rows_run_team(const double2* X, double2* Y, const double2* Wm, int n, int N, int k0, int K,
                              const int* perm, double2* stage) {
  gj_rows_update_team(X, Y, Wm, n, N, k0, K, perm, stage);
}

}  // namespace negf
