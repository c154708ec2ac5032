// Dense complex double products of the ring-block LU (dense.cu): the library's own strided-batched
// GEMM on the FP64 tensor cores and matrix-vector products, in place of a BLAS library.
#pragma once

#include <cuComplex.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace eb {
namespace dense {

// GEMM kernel variants (identical results): register-staged double buffer, cp.async ring of
// three slices on 64 x 64 tiles, cp.async ring of two slices on 64 x 32 tiles (four CTAs per SM).
constexpr int kStaged = 0, kAsync = 1, kAsyncNarrow = 2;
constexpr int kDefaultVariant = kAsyncNarrow;  // 32.5 against 26.3 TFLOP/s on 512^3 x 16

// C_z = alpha A_z B_z + beta C_z for z < batch, column-major, A_z = A + z stride_a (elements)
// etc.; alpha, beta real; beta == 0 does not read C. variant < 0 takes the default (or the one
// EB_ZGEMM=v<k> names). Returns an EB_* status.
int zgemm_nn_batched(int M, int N, int K, double alpha, const cuDoubleComplex* A, int lda,
                     int64_t stride_a, const cuDoubleComplex* B, int ldb, int64_t stride_b,
                     double beta, cuDoubleComplex* C, int ldc, int64_t stride_c, int batch,
                     cudaStream_t st, int variant = -1);

// Products inside a set of workspaces: entry e < n of workspace s multiplies the matrices at
// byte offsets a[e], b[e], c[e] of base + stride s.
struct Products {
  int n = 0;
  int64_t a[4], b[4], c[4];
  void add(int64_t pa, int64_t pb, int64_t pc) {
    a[n] = pa;
    b[n] = pb;
    c[n++] = pc;
  }
};
// C = alpha A B + beta C for every entry of every workspace (complex); the columns [gap0, gap1) of
// C, gap0 a multiple of 64, are left out.
int zgemm_set(int M, int N, int K, double alpha, double beta, char* base, int64_t stride,
              int workspaces, const Products& set, int lda, int ldb, int ldc, cudaStream_t st,
              int gap0 = 0, int gap1 = 0);

// The same with real matrices; the dimensions and leading dimensions are multiples of 4.
int dgemm_set(int M, int N, int K, double alpha, double beta, char* base, int64_t stride,
              int workspaces, const Products& set, int lda, int ldb, int ldc, cudaStream_t st);

// One matrix-vector product of a triangular sweep, as byte offsets into a workspace:
// y = [y +] alpha op(A) x - Bd v - op(A2) (Bd2 v2), with op(A) = A and Bd, Bd2 as they are, or
// op(A) = A^H and Bd, Bd2 transposed. A, A2: n x n complex, column-major; Bd, Bd2: n / 4 real
// column-major 4 x 4 blocks (negative offset: term absent).
struct SweepTerm {
  int64_t a = -1, x = -1, y = -1;
  int64_t bd = -1, v = -1;
  int64_t a2 = -1, bd2 = -1, v2 = -1;
  double alpha = 0.0;
  int add = 0;
};
struct SweepTerms {
  int n = 0;
  SweepTerm t[4];
  void add(const SweepTerm& s) { t[n++] = s; }
};
// The products of one sweep step for every workspace (they may run in any order).
int sweep_product(int conj_trans, int n, char* base, int64_t stride, int workspaces,
                  const SweepTerms& terms, cudaStream_t st);

// The same step over nr <= 8 right-hand sides per workspace (op(A) = A; no second matrix): x, y
// and v are byte offsets into vectors + vstride z, blocks of n x nr columns; workspaces
// z = zmap[0 .. *n_active - 1] only (device arrays).
int sweep_product_multi(int n, int nr, char* base, int64_t stride, char* vectors, int64_t vstride,
                        int workspaces, const int* zmap, const int* n_active,
                        const SweepTerms& terms, cudaStream_t st);

}  // namespace dense
}  // namespace eb
