// Inversion of the ring LU's diagonal super-blocks by one cooperative launch (ring_invert.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace eb {
namespace rl {

// A block of every system of a launch: system z = chains * s + t at byte
// base + stride * s + off + chain * t.
struct At {
  int64_t off = 0;    // of chain 0
  int64_t chain = 0;  // from chain 0 to chain 1
};

// Byte offsets of the blocks a launch works on (see k_ring_invert).
struct InvertAt {
  At in;     // the K x K block (elements of the scalar type)
  At pub;    // K x K scratch: the finished panels on their way to the other CTAs
  At out;    // the inverse, complex (may be `in`)
  At real;   // the inverse again as real numbers (real scalar type only)
  At flags;  // uint64[kInvertFlags], zero before the first launch of a factorisation
  At info;   // int: 0, or non-zero once a pivot was zero or not finite
};
constexpr int kInvertFlags = 256;  // K / 4 groups of steps at most

// Inverts the blocks of n_shifts * chains systems of order K (at most 1024, a multiple of 4).
// epoch: a positive number that grows from launch to launch on the same flags. real: the blocks
// hold real numbers. Returns an EB_* status.
int ring_invert(int K, int n_shifts, int chains, char* base, int64_t stride, const InvertAt& at,
                int epoch, bool real, cudaStream_t st);

}  // namespace rl
}  // namespace eb
