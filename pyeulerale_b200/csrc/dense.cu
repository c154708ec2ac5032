// Dense double products of the ring-block LU (ringlu.cu): strided-batched C = alpha A B + beta C
// (column-major, no transposes; complex, or real where every shift is real) on the FP64
// tensor-core instruction mma.sync.m8n8k4.f64, and the matrix-vector products of its sweeps.
// alpha and beta are real (the LU uses +-1 and 0 / 1).
//
// GEMM: a CTA computes a tile of C for one batch entry with four warps, each a sub-tile of 8 x 8
// products (m8n8k4 fragments; complex: real and imaginary parts in separate accumulators, re +=
// Ar Br - Ai Bi, im += Ar Bi + Ai Br, four real MMAs per complex product). The kBK-deep slices of A
// and B go through shared memory, two slices in flight (the next slice's loads are issued before
// the current slice's MMAs). Edges (sizes not multiples of the tile) load zeros and store under
// bounds checks. The default moves the slices with cp.async into a ring of shared buffers that keep
// each complex element's two parts together (one 16-byte fragment load gives both) on 64 x 32
// tiles, or 32 x 16 where those would leave SMs idle; a register-staged variant and one on 64 x 64
// tiles issue the same MMAs in the same order, so all give identical results.
//
// Sweep products: y (+)= -sum of blocks times vectors for one right-hand side (k_sweep_n, and
// k_sweep_h for the adjoint's A^H), or for several that share the block (k_sweep_multi). A ring's
// terms go in one launch, and the launches of a sweep start early (programmatic dependent
// launches): each loads its matrix while the one before it finishes.

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>

#include "../../include/euler_b200.h"
#include "dense.cuh"

namespace eb {

int check_launch(const char* what);
int fail(int code, const char* msg);

namespace dense {
namespace {

constexpr int kBM = 64, kBN = 64, kBK = 16;
constexpr int kGemmThreads = 128;
// Shared-memory pitches (doubles) of the A planes [k][m] and B planes [n][k], 4 modulo 16, so
// that a warp's fragment loads (4 k x 8 m, and 8 n x 4 k) fall on distinct banks within each
// half-warp.
constexpr int kPadM = kBM + 4;
constexpr int kPadK = kBK + 4;

// Operands of batch entry z: strided from three bases, or entry z % n of workspace z / n.
struct Operands {
  const char *a, *b;
  char* c;
  int64_t sa, sb, sc;  // bytes
  Products set;        // set.n == 0: strided
  int gap0 = 0, gap1 = 0;  // columns of C left out (whole tiles)
  __device__ __forceinline__ int column(int n0) const { return n0 < gap0 ? n0 : n0 + gap1 - gap0; }
  template <class T>
  __device__ __forceinline__ void of(int64_t z, const T*& A, const T*& B, T*& C) const {
    int64_t oa = sa * z, ob = sb * z, oc = sc * z;
    if (set.n > 0) {
      const int64_t s = z / set.n;
      const int e = (int)(z % set.n);
      oa = sa * s + set.a[e];
      ob = sb * s + set.b[e];
      oc = sc * s + set.c[e];
    }
    A = reinterpret_cast<const T*>(a + oa);
    B = reinterpret_cast<const T*>(b + ob);
    C = reinterpret_cast<T*>(c + oc);
  }
};

struct GemmSmem {
  double ar[2][kBK][kPadM], ai[2][kBK][kPadM];
  double br[2][kBN][kPadK], bi[2][kBN][kPadK];
};

// D = A B + C for one 8 x 8 x 4 FP64 tile (a: A[lane / 4][lane % 4], b: B[lane % 4][lane / 4],
// c / d: C[lane / 4][2 (lane % 4) + {0, 1}]).
// (Not volatile: the instruction has no effect beyond its outputs, so the compiler may
// interleave independent MMAs to cover their latency.)
__device__ __forceinline__ void mma884(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// A 16-byte read-only load that the compiler keeps in program order with the other such loads,
// so that a thread's unrolled loads of a matrix are all in flight before the first is used (left
// to itself the compiler may sink each load next to its use, one DRAM latency per column).
__device__ __forceinline__ double2 ldg_inflight(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// Global -> registers for one kBK slice: each thread holds kBM * kBK / kGemmThreads complex
// elements of A and kBK * kBN / kGemmThreads of B (zero outside the matrices).
constexpr int kAPer = kBM * kBK / kGemmThreads;  // 8
constexpr int kBPer = kBK * kBN / kGemmThreads;  // 8

__device__ __forceinline__ void load_slice(const double2* A, int lda, const double2* B, int ldb,
                                           int M, int N, int K, int m0, int n0, int k0,
                                           double2 (&ra)[kAPer], double2 (&rb)[kBPer]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int q = 0; q < kAPer; ++q) {  // A: consecutive threads along m (columns are contiguous)
    const int e = tid + kGemmThreads * q, m = e % kBM, k = e / kBM;
    const int gm = m0 + m, gk = k0 + k;
    ra[q] = (gm < M && gk < K) ? A[gm + (int64_t)lda * gk] : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int q = 0; q < kBPer; ++q) {  // B: consecutive threads along k
    const int e = tid + kGemmThreads * q, k = e % kBK, n = e / kBK;
    const int gk = k0 + k, gn = n0 + n;
    rb[q] = (gk < K && gn < N) ? B[gk + (int64_t)ldb * gn] : make_double2(0.0, 0.0);
  }
}

__device__ __forceinline__ void store_slice(GemmSmem& S, int buf, const double2 (&ra)[kAPer],
                                            const double2 (&rb)[kBPer]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int q = 0; q < kAPer; ++q) {
    const int e = tid + kGemmThreads * q, m = e % kBM, k = e / kBM;
    S.ar[buf][k][m] = ra[q].x;
    S.ai[buf][k][m] = ra[q].y;
  }
#pragma unroll
  for (int q = 0; q < kBPer; ++q) {
    const int e = tid + kGemmThreads * q, k = e % kBK, n = e / kBK;
    S.br[buf][n][k] = rb[q].x;
    S.bi[buf][n][k] = rb[q].y;
  }
}

__global__ void __launch_bounds__(kGemmThreads)
    k_zgemm_nn(int M, int N, int K, double alpha, Operands ops, int lda, int ldb, double beta,
               int ldc) {
  extern __shared__ __align__(16) unsigned char zg_smem[];
  GemmSmem& S = *reinterpret_cast<GemmSmem*>(zg_smem);
  const double2 *A, *B;
  double2* C;
  ops.of(blockIdx.z, A, B, C);
  const int m0 = blockIdx.x * kBM, n0 = ops.column(blockIdx.y * kBN);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;  // the warp's 32 x 32 sub-tile
  const int fr = lane >> 2, fc = lane & 3;                 // fragment row / column indices
  double re[4][4][2], im[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  double2 ra[kAPer], rb[kBPer];
  load_slice(A, lda, B, ldb, M, N, K, m0, n0, 0, ra, rb);
  store_slice(S, 0, ra, rb);
  __syncthreads();
  const int slices = (K + kBK - 1) / kBK;
  for (int s = 0; s < slices; ++s) {
    const int buf = s & 1;
    if (s + 1 < slices) load_slice(A, lda, B, ldb, M, N, K, m0, n0, (s + 1) * kBK, ra, rb);
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a_r[4], a_i[4], a_n[4], b_r[4], b_i[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a_r[i] = S.ar[buf][kk + fc][wm + 8 * i + fr];
        a_i[i] = S.ai[buf][kk + fc][wm + 8 * i + fr];
        a_n[i] = -a_i[i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b_r[j] = S.br[buf][wn + 8 * j + fr][kk + fc];
        b_i[j] = S.bi[buf][wn + 8 * j + fr][kk + fc];
      }
      // two rounds over the 4 x 4 tiles, so that an accumulator's two MMAs of a k-step are
      // 32 independent MMAs apart (same order of the terms per accumulator)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          mma884(re[i][j], a_r[i], b_r[j]);
          mma884(im[i][j], a_r[i], b_i[j]);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          mma884(re[i][j], a_n[i], b_i[j]);
          mma884(im[i][j], a_i[i], b_r[j]);
        }
    }
    if (s + 1 < slices) {
      store_slice(S, buf ^ 1, ra, rb);
      __syncthreads();
    }
  }
  // epilogue: C = alpha acc + beta C (beta == 0: C is not read)
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + 8 * i + fr, gn = n0 + wn + 8 * j + 2 * fc + h;
        if (gm < M && gn < N) {
          double2* c = C + gm + (int64_t)ldc * gn;
          double2 v = make_double2(alpha * re[i][j][h], alpha * im[i][j][h]);
          if (beta != 0.0) {
            const double2 o = *c;
            v.x = fma(beta, o.x, v.x);
            v.y = fma(beta, o.y, v.y);
          }
          *c = v;
        }
      }
}

// ---- cp.async variants --------------------------------------------------------------------
// pitches in complex elements: A rows [k][m] 2 modulo 8, B rows [n][k] 4 modulo 8, so that the
// 16-byte fragment loads of each quarter-warp fall on distinct banks
constexpr int kPitchB = kBK + 4;

// BN: tile columns (64: warps of 32 x 32; 32: warps of 32 x 16, half the registers and shared
// memory, four CTAs per SM, twice the tiles); Stages: slices in flight.
template <int BN, int Stages, int BM = kBM>
struct AsyncSmem {
  double2 a[Stages][kBK][BM + 2];
  double2 b[Stages][BN][kPitchB];
};

// 16-byte global -> shared copy; valid == false fills zeros (src is then not read).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int Pending>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(Pending) : "memory");
}

template <int BN, int Stages, int BM = kBM>
__global__ void __launch_bounds__(kGemmThreads)
    k_zgemm_nn_async(int M, int N, int K, double alpha, Operands ops, int lda, int ldb,
                     double beta, int ldc) {
  constexpr int NI = BM / 16, NJ = BN / 16;          // 8-row and 8-column fragments per warp
  constexpr int kAPerT = BM * kBK / kGemmThreads;   // A elements per thread and slice
  constexpr int kBPerT = kBK * BN / kGemmThreads;   // B elements per thread and slice
  extern __shared__ __align__(16) unsigned char zg_smem[];
  AsyncSmem<BN, Stages, BM>& S = *reinterpret_cast<AsyncSmem<BN, Stages, BM>*>(zg_smem);
  const double2 *A, *B;
  double2* C;
  ops.of(blockIdx.z, A, B, C);
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * BM, n0 = ops.column(blockIdx.y * BN);
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp & 1) * (BM / 2), wn = (warp >> 1) * (BN / 2);
  const int fr = lane >> 2, fc = lane & 3;
  double re[NI][NJ][2], im[NI][NJ][2];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  const int slices = (K + kBK - 1) / kBK;
  // slice s into buffer s % Stages (one commit group per call, empty past the last slice)
  auto issue = [&](int s) {
    if (s < slices) {
      const int buf = s % Stages, k0 = s * kBK;
#pragma unroll
      for (int q = 0; q < kAPerT; ++q) {  // A: consecutive threads along m
        const int e = tid + kGemmThreads * q, m = e % BM, k = e / BM;
        const int gm = m0 + m, gk = k0 + k;
        const bool ok = gm < M && gk < K;
        cp_async16(&S.a[buf][k][m], ok ? A + gm + (int64_t)lda * gk : A, ok);
      }
#pragma unroll
      for (int q = 0; q < kBPerT; ++q) {  // B: consecutive threads along k
        const int e = tid + kGemmThreads * q, k = e % kBK, n = e / kBK;
        const int gk = k0 + k, gn = n0 + n;
        const bool ok = gk < K && gn < N;
        cp_async16(&S.b[buf][n][k], ok ? B + gk + (int64_t)ldb * gn : B, ok);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < Stages - 1; ++s) issue(s);
  for (int s = 0; s < slices; ++s) {
    cp_async_wait<Stages - 2>();  // slice s has landed (this thread's copies)
    __syncthreads();              // ... everyone's; and slice s - 1's buffer is free
    issue(s + Stages - 1);
    const int buf = s % Stages;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double2 a[NI], b[NJ];
      double a_n[NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        a[i] = S.a[buf][kk + fc][wm + 8 * i + fr];
        a_n[i] = -a[i].y;
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = S.b[buf][wn + 8 * j + fr][kk + fc];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          mma884(re[i][j], a[i].x, b[j].x);
          mma884(im[i][j], a[i].x, b[j].y);
        }
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          mma884(re[i][j], a_n[i], b[j].y);
          mma884(im[i][j], a[i].y, b[j].x);
        }
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + 8 * i + fr, gn = n0 + wn + 8 * j + 2 * fc + h;
        if (gm < M && gn < N) {
          double2* c = C + gm + (int64_t)ldc * gn;
          double2 v = make_double2(alpha * re[i][j][h], alpha * im[i][j][h]);
          if (beta != 0.0) {
            const double2 o = *c;
            v.x = fma(beta, o.x, v.x);
            v.y = fma(beta, o.y, v.y);
          }
          *c = v;
        }
      }
}

// Fewer 64 x 32 tiles than SMs: the products go in 32 x 16 tiles (the same sums in the same order),
// four times as many CTAs with a quarter of the work per slice (a pair of real 256^3 products:
// 6.6 us, 11.5 in 64 x 32 tiles).
inline bool few_tiles(int M, int N, int batch) {
  return (int64_t)((M + 63) / 64) * ((N + 31) / 32) * batch < 148;
}

// ---- real matrices ----------------------------------------------------------------------------
// The cp.async ring on 64 x 32 tiles with real elements: a copy moves two (the dimensions are
// multiples of 4, so a pair never straddles an edge), pitches 4 modulo 16 doubles keep the
// fragment loads of each half-warp on distinct banks. K = 512: 128 tiles per product, two
// products (or shifts) fill the SMs.
constexpr int kRealBN = 32, kRealStages = 3;
template <int BM, int BN>
struct RealSmem {
  double a[kRealStages][kBK][BM + 4];
  double b[kRealStages][BN][kPadK];
};

template <int BM, int BN>
__global__ void __launch_bounds__(kGemmThreads)
    k_dgemm_nn(int M, int N, int K, double alpha, Operands ops, int lda, int ldb, double beta,
               int ldc) {
  constexpr int Stages = kRealStages, NI = BM / 16, NJ = BN / 16;
  extern __shared__ __align__(16) unsigned char dg_smem[];
  RealSmem<BM, BN>& S = *reinterpret_cast<RealSmem<BM, BN>*>(dg_smem);
  const double *A, *B;
  double* C;
  ops.of(blockIdx.z, A, B, C);
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * BM, n0 = ops.column(blockIdx.y * BN);
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp & 1) * (BM / 2), wn = (warp >> 1) * (BN / 2);
  const int fr = lane >> 2, fc = lane & 3;
  double acc[NI][NJ][2];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int slices = (K + kBK - 1) / kBK;
  auto issue = [&](int s) {  // slice s into buffer s % Stages (one commit group per call)
    if (s < slices) {
      const int buf = s % Stages, k0 = s * kBK;
#pragma unroll
      for (int q = 0; q < BM * kBK / 2 / kGemmThreads; ++q) {
        const int e = tid + kGemmThreads * q, m = 2 * (e % (BM / 2)), k = e / (BM / 2);
        const int gm = m0 + m, gk = k0 + k;
        const bool ok = gm < M && gk < K;
        cp_async16(&S.a[buf][k][m], ok ? A + gm + (int64_t)lda * gk : A, ok);
      }
#pragma unroll
      for (int q = 0; q < kBK * BN / 2 / kGemmThreads; ++q) {
        const int e = tid + kGemmThreads * q, k = 2 * (e % (kBK / 2)), n = e / (kBK / 2);
        const int gk = k0 + k, gn = n0 + n;
        const bool ok = gk < K && gn < N;
        cp_async16(&S.b[buf][n][k], ok ? B + gk + (int64_t)ldb * gn : B, ok);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < Stages - 1; ++s) issue(s);
  for (int s = 0; s < slices; ++s) {
    cp_async_wait<Stages - 2>();
    __syncthreads();
    issue(s + Stages - 1);
    const int buf = s % Stages;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 4) {
      double a[NI], b[NJ];
#pragma unroll
      for (int i = 0; i < NI; ++i) a[i] = S.a[buf][kk + fc][wm + 8 * i + fr];
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = S.b[buf][wn + 8 * j + fr][kk + fc];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma884(acc[i][j], a[i], b[j]);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gm = m0 + wm + 8 * i + fr, gn = n0 + wn + 8 * j + 2 * fc + h;
        if (gm < M && gn < N) {
          double* c = C + gm + (int64_t)ldc * gn;
          const double v = alpha * acc[i][j][h];
          *c = beta != 0.0 ? fma(beta, *c, v) : v;
        }
      }
}

int launch_zgemm(int M, int N, int K, double alpha, double beta, const Operands& ops, int lda,
                 int ldb, int ldc, int batch, int variant, cudaStream_t st) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (variant < 0) {  // the default, or EB_ZGEMM=v<k> (measurements of the variants in place)
    const char* e = std::getenv("EB_ZGEMM");
    variant = (e && e[0] == 'v' && e[1] >= '0' && e[1] <= '2') ? e[1] - '0' : kDefaultVariant;
  }
  const bool small = variant == kAsyncNarrow && few_tiles(M, N - (ops.gap1 - ops.gap0), batch);
  auto kernel = variant == kAsync ? k_zgemm_nn_async<64, 3>
                : small           ? k_zgemm_nn_async<16, 3, 32>
                : variant == kAsyncNarrow ? k_zgemm_nn_async<32, 2>
                                          : k_zgemm_nn;
  const int smem = variant == kAsync ? (int)sizeof(AsyncSmem<64, 3>)
                   : small           ? (int)sizeof(AsyncSmem<16, 3, 32>)
                   : variant == kAsyncNarrow ? (int)sizeof(AsyncSmem<32, 2>)
                                             : (int)sizeof(GemmSmem);
  const int bm = small ? 32 : kBM, bn = small ? 16 : variant == kAsyncNarrow ? 32 : kBN;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
      cudaSuccess)
    return check_launch("zgemm attribute");
  const dim3 grid((M + bm - 1) / bm, (N - (ops.gap1 - ops.gap0) + bn - 1) / bn, batch);
  kernel<<<grid, kGemmThreads, smem, st>>>(M, N, K, alpha, ops, lda, ldb, beta, ldc);
  return check_launch("zgemm");
}

}  // namespace

int zgemm_nn_batched(int M, int N, int K, double alpha, const cuDoubleComplex* A, int lda,
                     int64_t stride_a, const cuDoubleComplex* B, int ldb, int64_t stride_b,
                     double beta, cuDoubleComplex* C, int ldc, int64_t stride_c, int batch,
                     cudaStream_t st, int variant) {
  constexpr int64_t kB = sizeof(cuDoubleComplex);
  const Operands ops{reinterpret_cast<const char*>(A), reinterpret_cast<const char*>(B),
                     reinterpret_cast<char*>(C), kB * stride_a, kB * stride_b, kB * stride_c, {}};
  return launch_zgemm(M, N, K, alpha, beta, ops, lda, ldb, ldc, batch, variant, st);
}

int zgemm_set(int M, int N, int K, double alpha, double beta, char* base, int64_t stride,
              int workspaces, const Products& set, int lda, int ldb, int ldc, cudaStream_t st,
              int gap0, int gap1) {
  if (gap0 % kBN != 0 || gap1 < gap0 || gap1 > N)
    return fail(EB_ERR_ARG, "zgemm: bad gap");
  if (gap1 - gap0 == N) return 0;
  const Operands ops{base, base, base, stride, stride, stride, set, gap0, gap1};
  return launch_zgemm(M, N, K, alpha, beta, ops, lda, ldb, ldc, workspaces * set.n, -1, st);
}

int dgemm_set(int M, int N, int K, double alpha, double beta, char* base, int64_t stride,
              int workspaces, const Products& set, int lda, int ldb, int ldc, cudaStream_t st) {
  if (M <= 0 || N <= 0 || workspaces * set.n <= 0) return 0;
  if ((M | N | K | lda | ldb | ldc) % 4 != 0)
    return fail(EB_ERR_ARG, "dgemm: sizes must be multiples of 4");
  const Operands ops{base, base, base, stride, stride, stride, set};
  auto run = [&](auto kernel, int bm, int bn, size_t smem) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return check_launch("dgemm attribute");
    const dim3 grid((M + bm - 1) / bm, (N + bn - 1) / bn, workspaces * set.n);
    kernel<<<grid, kGemmThreads, smem, st>>>(M, N, K, alpha, ops, lda, ldb, beta, ldc);
    return check_launch("dgemm");
  };
  if (few_tiles(M, N, workspaces * set.n))
    return run(k_dgemm_nn<32, 16>, 32, 16, sizeof(RealSmem<32, 16>));
  return run(k_dgemm_nn<kBM, kRealBN>, kBM, kRealBN, sizeof(RealSmem<kBM, kRealBN>));
}

namespace {

// (Bd v)[i] or (Bd^T v)[i] for one entry i of a block diagonal of real 4 x 4 blocks.
__device__ __forceinline__ double2 bd_entry(const double* bd, const double2* v, int i, bool trans) {
  const double* b = bd + 16 * (i >> 2);
  const double2* u = v + (i & ~3);
  const int r = i & 3;
  double2 o = make_double2(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double w = trans ? b[k + 4 * r] : b[r + 4 * k];
    o.x = fma(w, u[k].x, o.x);
    o.y = fma(w, u[k].y, o.y);
  }
  return o;
}

// Programmatic dependent launch: a step's kernel starts while the step before it still runs, issues
// its loads of the factors (which no step writes) and only then waits for that step's results. (The
// sweeps over several right-hand sides let the next step start first thing: the 64-shift sweep of
// the 129x129 grid takes 876 ms so, 892 with the next step let in after the wait, 924 without.)
__device__ __forceinline__ void let_next_start() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
template <class... Params, class... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, int threads, size_t smem,
                             cudaStream_t st, Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class T>
__device__ __forceinline__ T* place(char* ws, int64_t off) {
  return reinterpret_cast<T*>(ws + off);
}

// y[i] of one row: the sum of the products, the block-diagonal term and the previous y.
__device__ __forceinline__ void finish_row(const SweepTerm& t, char* ws, int i, double sr,
                                           double si, bool trans) {
  double2* y = place<double2>(ws, t.y) + i;
  double2 o = make_double2(sr, si);
  if (t.add) {
    o.x += y->x;
    o.y += y->y;
  }
  if (t.bd >= 0) {
    const double2 b = bd_entry(place<const double>(ws, t.bd), place<const double2>(ws, t.v), i, trans);
    o.x -= b.x;
    o.y -= b.y;
  }
  *y = o;
}

// Sweep step, op(A) = A. For few workspaces what bounds a step is latency, a few dependent loads and
// one launch, so a product is spread thin, eight rows per CTA (K = 512: 64 CTAs of 64 KB each; with
// 32 rows per CTA each of 16 SMs streamed 256 KB); many are bound by reading their matrices, 32 rows
// per CTA, whose warps read 512 bytes at a time. Thread (r, g) sums the columns j = g (mod
// kSweepThreads / Rows) of row r, eight loads in flight, four CTAs per SM, so that the next step's
// CTAs find room beside this one's (sixteen loads at three CTAs per SM: a solve at K = 512 with 12
// rings took 328 us, 273 so; 32 shifts 3391, 2553 with 32 rows, 2783 with eight). The partial sums are
// added in a fixed order. Grid: (row groups x terms, workspaces).
constexpr int kSweepThreads = 256;
template <int Rows>
__global__ void __launch_bounds__(kSweepThreads, 4) k_sweep_n(int n, char* base, int64_t stride,
                                                              SweepTerms terms) {
  constexpr int kGroups = kSweepThreads / Rows;  // columns taken at a time
  __shared__ double2 part[8][Rows];
  const SweepTerm t = terms.t[blockIdx.x % terms.n];
  const int group = blockIdx.x / terms.n;
  char* ws = base + stride * blockIdx.y;
  const int r = threadIdx.x % Rows, g = threadIdx.x / Rows, lane = threadIdx.x & 31;
  const int i = group * Rows + r;
  double sr = 0.0, si = 0.0;
  const bool active = i < n && t.a >= 0;
  const double2* A = place<const double2>(ws, t.a) + i;
  const double2* x = place<const double2>(ws, t.x);
  constexpr int kUnroll = 8;  // column loads in flight per thread (ldg_inflight)
  bool waited = false;
  for (int j = g; j < n || !waited; j += kGroups * kUnroll) {
    double2 a[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      a[u] = make_double2(0.0, 0.0);
      if (active && j + kGroups * u < n) a[u] = ldg_inflight(A + (int64_t)n * (j + kGroups * u));
    }
    if (!waited) {
      wait_previous();
      let_next_start();
    }
    waited = true;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (active && j + kGroups * u < n) {
        const double2 v = x[j + kGroups * u];
        sr = fma(a[u].x, v.x, fma(-a[u].y, v.y, sr));
        si = fma(a[u].x, v.y, fma(a[u].y, v.x, si));
      }
  }
#pragma unroll
  for (int o = Rows; o < 32; o <<= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    si += __shfl_xor_sync(0xffffffffu, si, o);
  }
  if (lane < Rows) part[threadIdx.x >> 5][lane] = make_double2(sr, si);
  __syncthreads();
  if (threadIdx.x < Rows && i < n) {
    double tr = 0.0, ti = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      tr += part[k][threadIdx.x].x;
      ti += part[k][threadIdx.x].y;
    }
    finish_row(t, ws, i, t.alpha * tr, t.alpha * ti, false);
  }
}

// Sweep step, op(A) = A^H: one warp per output (a column of A), the vectors in shared memory; a
// fixed shuffle tree adds the lanes' partial sums. Grid: (groups of eight outputs x terms,
// workspaces).
__global__ void __launch_bounds__(256) k_sweep_h(int n, char* base, int64_t stride,
                                                 SweepTerms terms) {
  extern __shared__ __align__(16) unsigned char sw_smem[];
  double2* xs = reinterpret_cast<double2*>(sw_smem);  // x, then Bd2^T v2
  const SweepTerm t = terms.t[blockIdx.x % terms.n];
  const int group = blockIdx.x / terms.n;
  char* ws = base + stride * blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int j = group * 8 + (threadIdx.x >> 5);
  // the first rows of the first matrix before the wait (512 rows: all of a column at K = 512)
  constexpr int kAhead = 16;
  double2 ahead[kAhead];
  const double2* first = place<const double2>(ws, t.a) + (int64_t)n * j;
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    ahead[u] = make_double2(0.0, 0.0);
    if (t.a >= 0 && j < n && lane + 32 * u < n) ahead[u] = ldg_inflight(first + lane + 32 * u);
  }
  wait_previous();
  let_next_start();
  for (int i = threadIdx.x; i < n; i += 256) {
    if (t.a >= 0) xs[i] = place<const double2>(ws, t.x)[i];
    if (t.a2 >= 0)
      xs[n + i] = bd_entry(place<const double>(ws, t.bd2), place<const double2>(ws, t.v2), i, true);
  }
  __syncthreads();
  if (j >= n) return;
  double sr = 0.0, si = 0.0;
  auto add = [&](const double2 a, const double2 w, double& tr, double& ti) {  // conj(a) w
    tr = fma(a.x, w.x, fma(a.y, w.y, tr));
    ti = fma(a.x, w.y, fma(-a.y, w.x, ti));
  };
  auto dot = [&](const double2* col, const double2* v, int from, double& tr, double& ti) {
    constexpr int kUnroll = 8;  // row loads in flight per lane (ldg_inflight)
    for (int i = from + lane; i < n; i += 32 * kUnroll) {
      double2 a[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        a[u] = make_double2(0.0, 0.0);
        if (i + 32 * u < n) a[u] = ldg_inflight(col + i + 32 * u);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (i + 32 * u < n) add(a[u], v[i + 32 * u], tr, ti);
    }
  };
  if (t.a >= 0) {
    double tr = 0.0, ti = 0.0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (lane + 32 * u < n) add(ahead[u], xs[lane + 32 * u], tr, ti);
    dot(first, xs, 32 * kAhead, tr, ti);
    sr = fma(t.alpha, tr, sr);
    si = fma(t.alpha, ti, si);
  }
  if (t.a2 >= 0) {
    double tr = 0.0, ti = 0.0;
    dot(place<const double2>(ws, t.a2) + (int64_t)n * j, xs + n, 0, tr, ti);
    sr -= tr;
    si -= ti;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    si += __shfl_xor_sync(0xffffffffu, si, o);
  }
  if (lane == 0) finish_row(t, ws, j, sr, si, true);
}

// The sweep step over NR right-hand sides, one read of A for all of them. Bound by reading A once
// (K = 512: 4.2 MB per workspace and term): eight rows per CTA, thread (r, g) takes the columns
// j = g (mod 32), 16 of them in flight at a time, issued before the right-hand sides are staged in
// shared memory; two CTAs keep 128 KB in flight per SM. The partial sums are added in a fixed order.
// A cluster of eight CTAs per 32 rows, which had each SM wait for its cluster's barriers and remote
// sums, read at 2.4 TB/s with 22 workspaces active.
// Grid: (row groups x terms, workspaces); workspaces from *n_active on exit.
constexpr int kMaxRhs = 8;
constexpr int kChunk = 512;  // columns per round: 16 per thread

template <int NR>
__global__ void __launch_bounds__(256, 2)
    k_sweep_multi(int n, const char* base, int64_t stride, char* vectors, int64_t vstride,
                  const int* zmap, const int* n_active, SweepTerms terms) {
  extern __shared__ __align__(16) unsigned char sk_smem[];
  __shared__ double2 part[8][NR][8];
  double2* xs = reinterpret_cast<double2*>(sk_smem);  // NR x min(n, kChunk)
  const int64_t z = zmap[blockIdx.y];
  if ((int)blockIdx.y >= *n_active) return;
  const SweepTerm t = terms.t[blockIdx.x % terms.n];
  const int group = blockIdx.x / terms.n;
  char* ws = const_cast<char*>(base) + stride * z;
  char* vs = vectors + vstride * z;
  const int tid = threadIdx.x, r = tid & 7, g = tid >> 3, lane = tid & 31;
  const int i = group * 8 + r;
  const int pitch = min(n, kChunk);
  let_next_start();
  double sr[NR], si[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) sr[q] = si[q] = 0.0;
  const double2* A = place<const double2>(ws, t.a) + i;
  const double2* x = place<const double2>(vs, t.x);
  for (int c0 = 0; c0 < n; c0 += kChunk) {
    const int cols = min(kChunk, n - c0);
    double2 a[kChunk / 32];
#pragma unroll
    for (int u = 0; u < kChunk / 32; ++u) {
      a[u] = make_double2(0.0, 0.0);
      if (i < n && g + 32 * u < cols) a[u] = ldg_inflight(A + (int64_t)n * (c0 + g + 32 * u));
    }
    if (c0 == 0) {
      wait_previous();
    } else {
      __syncthreads();  // the previous columns' right-hand sides have been used
    }
#pragma unroll
    for (int q = 0; q < NR; ++q)
      for (int j = tid; j < cols; j += 256) xs[pitch * q + j] = x[c0 + j + (int64_t)n * q];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kChunk / 32; ++u)
      if (g + 32 * u < cols) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          const double2 v = xs[pitch * q + g + 32 * u];
          sr[q] = fma(a[u].x, v.x, fma(-a[u].y, v.y, sr[q]));
          si[q] = fma(a[u].x, v.y, fma(a[u].y, v.x, si[q]));
        }
      }
  }
#pragma unroll
  for (int q = 0; q < NR; ++q) {
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      sr[q] += __shfl_xor_sync(0xffffffffu, sr[q], o);
      si[q] += __shfl_xor_sync(0xffffffffu, si[q], o);
    }
    if (lane < 8) part[tid >> 5][q][lane] = make_double2(sr[q], si[q]);
  }
  __syncthreads();
  const int row = group * 8 + (tid & 7), q = tid >> 3;
  if (q < NR && row < n) {
    double tr = 0.0, ti = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      tr += part[k][q][tid & 7].x;
      ti += part[k][q][tid & 7].y;
    }
    double2* out = place<double2>(vs, t.y) + row + (int64_t)n * q;
    double2 o = make_double2(t.alpha * tr, t.alpha * ti);
    if (t.add) {
      o.x += out->x;
      o.y += out->y;
    }
    if (t.bd >= 0) {
      const double2 b = bd_entry(place<const double>(ws, t.bd),
                                 place<const double2>(vs, t.v) + (int64_t)n * q, row, false);
      o.x -= b.x;
      o.y -= b.y;
    }
    *out = o;
  }
}

template <int NR>
int launch_sweep_multi(int n, char* base, int64_t stride, char* vectors, int64_t vstride,
                       int workspaces, const int* zmap, const int* n_active,
                       const SweepTerms& terms, cudaStream_t st) {
  const int smem = (int)sizeof(double2) * NR * (n < kChunk ? n : kChunk);
  // the limit is the kernel's, not the launch's: always the most it can need, so that another
  // thread's smaller sweep does not lower it under this launch
  if (cudaFuncSetAttribute(k_sweep_multi<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(double2) * NR * kChunk) != cudaSuccess)
    return check_launch("sweep attribute");
  if (launch_dependent(k_sweep_multi<NR>, dim3((n + 7) / 8 * terms.n, workspaces), 256, smem, st, n,
                       (const char*)base, stride, vectors, vstride, zmap, n_active, terms) !=
      cudaSuccess)
    return check_launch("sweep product");
  return EB_OK;
}

// Rows per CTA of a forward step: eight until their CTAs for one term fill the 592 places (four per
// SM) one and a half times. Solves over 12 rings in us, eight rows against 32: K = 320, 12 shifts 872,
// 967, 24 shifts 1675, 1596; K = 512, 8 shifts 760, 979, 16 shifts 1452, 1454, 24 shifts 2130, 2059;
// K = 1024, 4 shifts 836, 1300, 8 shifts 1598, 1657.
inline int sweep_rows(int n, int workspaces) {
  return (int64_t)((n + 7) / 8) * workspaces > 6 * 148 ? 32 : 8;
}

}  // namespace

int sweep_product(int conj_trans, int n, char* base, int64_t stride, int workspaces,
                  const SweepTerms& terms, cudaStream_t st) {
  if (n <= 0 || workspaces <= 0 || terms.n <= 0) return 0;
  const int rows = conj_trans ? 8 : sweep_rows(n, workspaces);
  const dim3 grid((n + rows - 1) / rows * terms.n, workspaces);
  auto launch = [&](auto kernel, size_t smem) {
    return launch_dependent(kernel, grid, kSweepThreads, smem, st, n, base, stride, terms);
  };
  const cudaError_t e = conj_trans   ? launch(k_sweep_h, 2 * sizeof(double2) * (size_t)n)
                        : rows == 32 ? launch(k_sweep_n<32>, 0)
                                     : launch(k_sweep_n<8>, 0);
  return e == cudaSuccess ? EB_OK : check_launch("sweep product");
}

int sweep_product_multi(int n, int nr, char* base, int64_t stride, char* vectors, int64_t vstride,
                        int workspaces, const int* zmap, const int* n_active,
                        const SweepTerms& terms, cudaStream_t st) {
  if (n % 4 != 0) return fail(EB_ERR_ARG, "sweep: block diagonals need n % 4 == 0");
  if (n <= 0 || workspaces <= 0 || nr <= 0 || terms.n <= 0) return 0;
  for (int k = 0; k < terms.n; ++k)
    if (terms.t[k].a < 0 || terms.t[k].a2 >= 0) return fail(EB_ERR_ARG, "sweep: one matrix per term");
  auto run = [&](auto launch) {
    return launch(n, base, stride, vectors, vstride, workspaces, zmap, n_active, terms, st);
  };
  switch (nr) {
    case 1: return run(launch_sweep_multi<1>);
    case 2: return run(launch_sweep_multi<2>);
    case 3: return run(launch_sweep_multi<3>);
    case 4: return run(launch_sweep_multi<4>);
    case 5: return run(launch_sweep_multi<5>);
    case 6: return run(launch_sweep_multi<6>);
    case 7: return run(launch_sweep_multi<7>);
    case kMaxRhs: return run(launch_sweep_multi<kMaxRhs>);
    default: return fail(EB_ERR_ARG, "sweep: too many right-hand sides");
  }
}

}  // namespace dense
}  // namespace eb

extern "C" int eb_zgemm_strided_batched(int M, int N, int K, double alpha, const double* A,
                                        int lda, int64_t stride_a, const double* B, int ldb,
                                        int64_t stride_b, double beta, double* C, int ldc,
                                        int64_t stride_c, int batch, int variant, void* stream) {
  if (M < 0 || N < 0 || K < 0 || batch < 0 || lda < (M > 1 ? M : 1) ||
      ldb < (K > 1 ? K : 1) || ldc < (M > 1 ? M : 1) || variant < -1 || variant > 2 ||
      (M > 0 && N > 0 && batch > 0 && (!A || !B || !C)))
    return eb::fail(EB_ERR_ARG, "zgemm: bad sizes, leading dimensions, variant or pointers");
  return eb::dense::zgemm_nn_batched(
      M, N, K, alpha, reinterpret_cast<const cuDoubleComplex*>(A), lda, stride_a,
      reinterpret_cast<const cuDoubleComplex*>(B), ldb, stride_b, beta,
      reinterpret_cast<cuDoubleComplex*>(C), ldc, stride_c, batch,
      reinterpret_cast<cudaStream_t>(stream), variant);
}
