// Inversion of the ring LU's diagonal super-blocks by one cooperative launch (ring_invert.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace eb {
namespace rl {

// Byte offsets in a system's workspace of the blocks an inversion works on.
struct InvertAt {
  size_t in;     // the K x K block (elements of the scalar type)
  size_t pub;    // K x K scratch: the finished columns on their way to the other CTAs
  size_t out;    // the inverse, complex (may be `in`)
  size_t real;   // the inverse again as real numbers (real scalar type only)
  size_t flags;  // uint64[kInvertFlags], zero before the first launch of a factorisation
  size_t info;   // int: 0, or the first of the states below
};
constexpr int kSingular = 1;  // a pivot was zero or not finite
constexpr int kRanOut = 2;    // a wait for another CTA's pivots ran out
// The EB_* status of an info value, with its error text.
int info_status(int info);
constexpr int kInvertFlags = 256;  // K / 4 groups of steps at most

// Inverts the block of every system (workspaces at base + stride s), of order K (at most 1024, a
// multiple of 4). epoch: a positive number that grows from launch to launch on the same flags.
// real: the blocks hold real numbers. Returns an EB_* status.
int ring_invert(int K, int systems, char* base, int64_t stride, const InvertAt& at, int epoch,
                bool real, cudaStream_t st);
// The number of systems that one launch of it holds (later ones wait), or a negative EB_* status.
int ring_invert_resident(int K, bool real);

}  // namespace rl
}  // namespace eb
