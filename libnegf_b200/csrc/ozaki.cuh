// Complex128 block products on the integer tensor cores (sm_100a tcgen05,
// kind::i8) by an exact-splitting (Ozaki) scheme.
//
// Every real part and imaginary part of a row of A (a column of B) is scaled
// by the same power of two 2^-e so that it lies in (-1, 1), then cut into S
// digits rounded to nearest: x = sum_t d_t 2^(-6-7t) + r, |d_t| <= 64,
// |r| <= 2^(-7S).  The digit matrices are int8; their products accumulate
// exactly in int32 (|sum| <= 8 * 2K * 64^2 < 2^31 for K <= 1024).  The digit
// pairs (t, u), 0-based, with t + u < min(S + 1, 8) are kept, one TMEM
// accumulator per level t + u, and the epilogue rebuilds
// C = 2^(eA_r + eB_c) sum_levels 2^(-12-7 level) acc in FP64.  The result
// carries about 7S bits relative to the row / column scales (S = 7: a few
// units of the rounding of an FP64 product).
//
// Complex: C_re = [Ar | -Ai] [Br ; Bi] and C_im = [Ai | Ar] [Br ; Bi], two
// real products over the concatenated K (the digits of Ar, Ai and -Ai are
// all stored, so the B tiles are shared).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace negf {

constexpr int kOzTileM = 128;       // UMMA M (one CTA)
constexpr int kOzTileN = 128;       // UMMA N (the full-rate width); 4 levels x 128 columns of TMEM
constexpr int kOzKChunk = 32;       // bytes of K per pipeline stage (one 32-byte swizzle row, one MMA K step)
constexpr int kOzStages = 3;
constexpr int kOzMinSlices = 4, kOzMaxSlices = 8;

// The digits of one operand of a batch of problems: planes, an exponent per
// row (column) and a non-finite flag per problem, all at the problem's index,
// so that an operand split once serves every product it takes part in, also
// after problems have left the batch.
struct OzakiSet {
  int8_t* q;
  int* e;
  int* flag;
  int problems;
};
size_t ozaki_rows_bytes(int problems, int m, int k, int slices);   // of left operands (m x k)
size_t ozaki_cols_bytes(int problems, int k, int n, int slices);   // of right operands (k x n)
OzakiSet ozaki_rows_at(void* base, int problems, int m, int k, int slices);   // base: 256-byte aligned
OzakiSet ozaki_cols_at(void* base, int problems, int k, int n, int slices);

// Split the operands A_p (B_p) of the problems p = map[b], b < batch (map
// null: p = b); complex128, column major, sA / sB complex elements apart.
cudaError_t launch_ozaki_rows(int batch, int m, int k, const double2* A, int64_t sA, int slices, const OzakiSet& d,
                              cudaStream_t s, const int* map);
cudaError_t launch_ozaki_cols(int batch, int k, int n, const double2* B, int64_t sB, int slices, const OzakiSet& d,
                              cudaStream_t s, const int* map);
// C_p = alpha * A_p * B_p + beta * C_p from split operands, the same problem
// selection.  beta == 0: C is not read.  t0: m x n doubles per launch item.
// maxabs (optional, one double per problem, non-negative, updated with
// atomicMax on its bit pattern): max |C_p| over the stored elements, NaN when
// one of them is NaN or Inf.  status (optional, one int per problem): 3 on a
// non-finite operand (C is NaN), 7 when a pipeline wait ran out (C is not
// written).
cudaError_t launch_ozaki_product(int batch, int m, int n, int k, double2 alpha, const OzakiSet& A, const OzakiSet& B,
                                 double2 beta, double2* C, int64_t sC, int slices, double* t0, double* maxabs,
                                 int* status, cudaStream_t s, const int* map);

// Both splits and the product of a whole batch, in a workspace of
// ozaki_work_bytes() (256-byte aligned).  C may alias A or B (the operands are
// split into the workspace first).
size_t ozaki_work_bytes(int batch, int m, int n, int k, int slices);
cudaError_t launch_ozaki_zgemm(int batch, int m, int n, int k, double2 alpha, const double2* A, int64_t sA,
                               const double2* B, int64_t sB, double2 beta, double2* C, int64_t sC, int slices,
                               void* work, double* maxabs, int* status, cudaStream_t s);

}  // namespace negf
