// The pivot steps of the ring LU's Gauss-Jordan inversions: elimination of a panel of columns held
// in the registers of one CTA (ring_invert.cu, and the panels of the blocked form in ringlu.cu),
// with the scalar operations for real and complex elements.
#pragma once

#include <cuComplex.h>
#include <cuda_runtime.h>

namespace eb {
namespace rl {

constexpr int kMaxRows = 1024;

__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ cuDoubleComplex mul(cuDoubleComplex a, cuDoubleComplex b) {
  return make_cuDoubleComplex(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double neg(double a) { return -a; }
__device__ __forceinline__ cuDoubleComplex neg(cuDoubleComplex a) {
  return make_cuDoubleComplex(-a.x, -a.y);
}
// c + a b
__device__ __forceinline__ double fmadd(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ cuDoubleComplex fmadd(cuDoubleComplex a, cuDoubleComplex b,
                                                 cuDoubleComplex c) {
  return make_cuDoubleComplex(fma(a.x, b.x, fma(-a.y, b.y, c.x)),
                              fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// c - a b
__device__ __forceinline__ double fmsub(double a, double b, double c) { return fma(-a, b, c); }
__device__ __forceinline__ cuDoubleComplex fmsub(cuDoubleComplex a, cuDoubleComplex b,
                                                 cuDoubleComplex c) {
  return make_cuDoubleComplex(fma(-a.x, b.x, fma(a.y, b.y, c.x)),
                              fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}
// 1 / a of a normal number below 2^1022: two Newton-Raphson steps y <- y + y (1 - a y), each of which
// squares the relative error, from the hardware's approximation (2^-19 or better), without the
// branches of a division, so that it runs in the shadow of the pivot search. (Bringing the other
// numbers into that range by a power of two, or dividing by them where a row is staged, took 3 %
// of a ring's time.)
__device__ __forceinline__ double recip(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;\n" : "=d"(y) : "d"(a));
  y = fma(y, fma(-a, y, 1.0), y);
  return fma(y, fma(-a, y, 1.0), y);
}
__device__ __forceinline__ cuDoubleComplex recip(cuDoubleComplex a) {
  const double d = recip(a.x * a.x + a.y * a.y);
  return make_cuDoubleComplex(a.x * d, -a.y * d);
}
// a non-negative number ordered like the modulus
__device__ __forceinline__ double size_of(double a) { return fabs(a); }
__device__ __forceinline__ double size_of(cuDoubleComplex a) { return a.x * a.x + a.y * a.y; }
template <class T>
__device__ __forceinline__ T zero_of();
template <>
__device__ __forceinline__ double zero_of<double>() {
  return 0.0;
}
template <>
__device__ __forceinline__ cuDoubleComplex zero_of<cuDoubleComplex>() {
  return make_cuDoubleComplex(0.0, 0.0);
}

// Barrier `id` of `n` threads (a multiple of 32): wait, or arrive without waiting.
__device__ __forceinline__ void bar_sync(int id, int n) {
  asm volatile("barrier.cta.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("barrier.cta.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}

constexpr int kSub = 4;      // steps handed over together
constexpr int kStepBar = 1;  // the steps' barrier

template <class T, int NC, int Warps>
struct StepShared {
  T cand[2][Warps][NC];     // each warp's best row of a step
  T cand_inv[2][Warps];     // the reciprocal of its pivot entry
  unsigned cand_key[2][Warps];
  int own[NC];              // the pivot rows
};

// `width` elimination steps (a multiple of kSub, at most NC) on the columns a: thread tid of the 32
// Warps that call it holds rows tid + 32 Warps r (r < ROWS, rows from K on are zero), left[r] tells
// the rows not chosen yet. A step takes the largest modulus among those (to one part in 2^10; ties
// go to the smaller row) as the pivot: every warp stages its best row, one barrier, every thread
// finds the winner and eliminates the column from its rows, the next step's column first, so that
// its search runs under the other columns' updates. S.own[jj] and pos[r] = c0 + jj record step jj's
// row. Calls done(jj) after each group of kSub steps (their columns are then a[.][NC - kSub ..]),
// failed(jj) and returns false at a zero or non-finite pivot or one outside recip's range (alike in
// all threads). The columns rotate by one per step: the step's column is a[.][0], its result goes
// to the last place, so after NC steps they are in order, after fewer column k is at NC - width +
// k. (The loop stays rolled: each CTA runs it once, and unrolled steps, all fetched cold, took 950
// cycles each; 512 to 930 cycles by rows per thread in this form.)
template <class T, int NC, int ROWS, int Warps, class Done, class Failed>
__device__ __forceinline__ bool eliminate(StepShared<T, NC, Warps>& S, T (&a)[ROWS][NC],
                                          bool (&left)[ROWS], int (&pos)[ROWS], int width, int c0,
                                          int K, int tid, Done done, Failed failed) {
  constexpr int nt = 32 * Warps;
  const int warp = tid >> 5;
  // this thread's best remaining entry of column a[.][0]: its key (ordered like the modulus to
  // one part in 2^10, the row in the low ten bits; 0: none) and its reciprocal
  unsigned mine = 0u;
  T inv_mine = zero_of<T>();
  auto candidate = [&]() {
    T pivot = a[0][0];
    mine = 0u;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const unsigned key = left[r] ? ((unsigned)__double2hiint(size_of(a[r][0])) & ~0x3FFu) |
                                         (unsigned)(kMaxRows - 1 - (tid + r * nt))
                                   : 0u;
      if (r == 0 || key > mine) {
        mine = key;
        pivot = a[r][0];
      }
    }
    inv_mine = recip(pivot);
  };
  candidate();
#pragma unroll 1
  for (int jj = 0; jj < width; ++jj) {
    const int par = jj & 1;
    const unsigned best = __reduce_max_sync(0xffffffffu, mine);
    if (mine == best) {  // this thread's row is the warp's best: stage it
      // (best = 0, no row left: every lane stages, and the step fails if all warps say so)
      const int brow = kMaxRows - 1 - (int)(best & 0x3FFu);
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (brow == tid + r * nt) {
#pragma unroll
          for (int k = 0; k < NC; ++k) S.cand[par][warp][k] = a[r][k];
        }
      S.cand_inv[par][warp] = inv_mine;
      S.cand_key[par][warp] = best;
    }
    bar_sync(kStepBar, nt);
    unsigned kb = 0u;
#pragma unroll
    for (int q = 0; q < Warps; ++q) kb = max(kb, S.cand_key[par][q]);
    const int prow = kMaxRows - 1 - (int)(kb & 0x3FFu);
    const unsigned size = kb & ~0x3FFu;
    // the same in every thread: zero, not finite, or out of recip's range (size_of: the modulus of
    // a real number, its square of a complex one)
    if (size - 0x00100000u >= 0x7FC00000u || prow >= K) {
      failed(jj);
      return false;
    }
    const int w = (prow % nt) >> 5;  // the warp that holds row prow
    const T inv = S.cand_inv[par][w];
    const T* row = S.cand[par][w];
    if (tid == 0) S.own[jj] = prow;
    T f[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) f[r] = mul(a[r][0], inv);
    if (warp == w) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (tid + r * nt == prow) {  // the pivot row becomes inv times itself
          left[r] = false;
          pos[r] = c0 + jj;
          f[r] = neg(inv);
#pragma unroll
          for (int k = 1; k < NC; ++k) a[r][k] = zero_of<T>();
        }
    }
    // the next step's column first: its search runs under the other columns' updates
#pragma unroll
    for (int r = 0; r < ROWS; ++r) a[r][0] = fmsub(f[r], row[1], a[r][1]);
    candidate();
#pragma unroll
    for (int k = 2; k < NC; ++k) {
      const T b = row[k];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) a[r][k - 1] = fmsub(f[r], b, a[r][k]);
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) a[r][NC - 1] = neg(f[r]);
    if (jj % kSub == kSub - 1) done(jj);
  }
  return true;
}

}  // namespace rl
}  // namespace eb
