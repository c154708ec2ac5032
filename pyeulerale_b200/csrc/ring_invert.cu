// Gauss-Jordan inversion of a ring's K x K diagonal block (ringlu.cu) with partial pivoting, as
// one cooperative launch: the block's columns are spread over CTAs, NC columns per CTA, each
// thread keeping its rows of them in registers from the first pivot to the last.
//
// What bounds it is the chain of K pivot steps, not arithmetic: a panel on one SM and its update
// on all of them, as two launches per panel, spent 27 us per 16 steps on the panel and as much
// again on loading it, the update and two launch gaps. Here a panel never leaves its CTA's
// registers: CTA p eliminates its columns (search for the largest remaining entry, one barrier
// per step), hands each group of four finished steps to a publishing warp, which copies them to
// global memory and raises a flag with the pivot rows in it, and every other CTA applies the
// group to its own columns as a rank-4 update, so that CTA p + 1 begins its pivots about 2.5 us
// after CTA p's last one. NC = 16 real or 8 complex columns: a block of K = 512 occupies 32 (64)
// SMs. Measured per block (one or two blocks at a time): K = 128 complex 88 us, real 67; 256: 205
// and 145; 512: 562 and 360; 1024: 2250 and 1170. With the two launches per panel a ring of
// K = 512 took 1150 us, of K = 128 about 300 us, complex.
//
// The waits are polls of a flag in global memory by CTAs of one cooperative launch (all are
// resident); each gives up after kPollLimit polls, records it in info (kRanOut) and ends the
// launch's work on that system.

#include "gj_step.cuh"
#include "ring_invert.cuh"

#include <cuComplex.h>

#include <algorithm>
#include <string>

#include "../../include/euler_b200.h"

namespace eb {

int fail(int code, const char* msg);
int check_launch(const char* what);

namespace rl {
namespace {

constexpr int kPollLimit = 1 << 22;  // about three seconds

// Loads past L1: the panels are written by other SMs during the launch.
__device__ __forceinline__ double load_l2(const double* p) { return __ldcg(p); }
__device__ __forceinline__ cuDoubleComplex load_l2(const cuDoubleComplex* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return make_cuDoubleComplex(v.x, v.y);
}

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_release(unsigned long long* p, unsigned long long v) {
  asm volatile("fence.acq_rel.gpu;\n st.release.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v)
               : "memory");
}
// The word published for a group of kSub steps: the launch's epoch, whether the steps found
// their pivots, and the pivot rows (ten bits each).
__device__ __forceinline__ unsigned long long pack(int epoch, bool ok, const int* piv) {
  unsigned long long w = ((unsigned long long)epoch << 1) | (ok ? 1ull : 0ull);
#pragma unroll
  for (int k = 0; k < kSub; ++k) w = (w << 10) | (unsigned long long)(ok ? piv[k] : 0);
  return w;
}
__device__ __forceinline__ bool is_epoch(unsigned long long w, int epoch) {
  return (w >> (10 * kSub + 1)) == (unsigned long long)epoch;
}
__device__ __forceinline__ bool is_ok(unsigned long long w) { return (w >> (10 * kSub)) & 1ull; }
__device__ __forceinline__ int row_of(unsigned long long w, int k) {
  return (int)((w >> (10 * (kSub - 1 - k))) & 0x3FFull);
}

// Polls until the flag holds a word of this launch; false once `limit` polls have not seen one.
__device__ __forceinline__ bool wait_word(const unsigned long long* flag, int epoch, int limit,
                                          unsigned long long& w) {
  for (int n = 0; n < limit; ++n) {
    w = load_acquire(flag);
    if (is_epoch(w, epoch)) return true;
  }
  return false;
}

// Waits on a flag that nothing sets.
__global__ void k_wait_probe(const unsigned long long* flag, int* info, int polls) {
  unsigned long long w;
  if (!wait_word(flag, 1, polls, w)) atomicCAS(info, 0, kRanOut);
}

template <class T, int NC, int Warps>
struct alignas(16) Shared {  // (the staged columns behind it are copied in pairs of doubles)
  StepShared<T, NC, Warps> step;
  T rows[kSub][NC];              // the pivot rows of a group of steps in this CTA's columns
  unsigned long long word;       // the group's published word (0: the wait gave up)
  int bad;                       // the group of its own steps that met no pivot (else kGroups)
  int failed;                    // info at the start: an earlier block of the system failed
  int ended;                     // the work ended before its own steps
};

// Grid: (ceil(K / NC), systems); block: the compute threads, ceil(K / ROWS) rounded up to whole
// warps, and one warp that publishes. Compute thread t holds rows t + r nt (r < ROWS) of the
// CTA's columns j NC .. j NC + NC - 1. Steps follow the in-place Gauss-Jordan elimination with
// implicit row pivoting: a group of steps with pivot rows P turns every other column c into
// A[:, c] (rows P zeroed) + A'[:, group] A[P, c], and after the last step the working array W
// holds Dinv[pos(i), perm[k]] = W[i, k] with pos(i) the step that chose row i.
template <class T, int NC, int ROWS, int Threads>
__global__ void __launch_bounds__(Threads + 32, 1)
    k_ring_invert(int K, int z0, char* base, int64_t stride, InvertAt at, int epoch) {
  constexpr bool kReal = sizeof(T) == sizeof(double);
  constexpr int nt = Threads, kWarps = Threads / 32;  // compute threads and warps
  constexpr int kGroupBar = 2;  // kGroupBar + q: group q of this CTA's steps
  constexpr int kGroups = NC / kSub;
  extern __shared__ __align__(16) unsigned char ri_smem[];
  using Sh = Shared<T, NC, Threads / 32>;
  Sh& S = *reinterpret_cast<Sh*>(ri_smem);
  T* stage = reinterpret_cast<T*>(ri_smem + sizeof(Sh));  // NC columns of K
  char* ws = base + stride * (z0 + blockIdx.y);
  auto place = [&](size_t off) { return ws + off; };
  const T* in = reinterpret_cast<const T*>(place(at.in));
  T* pub = reinterpret_cast<T*>(place(at.pub));
  unsigned long long* flags = reinterpret_cast<unsigned long long*>(place(at.flags));
  int* info = reinterpret_cast<int*>(place(at.info));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j = blockIdx.x, panels = gridDim.x, c0 = j * NC, width = min(NC, K - c0);
  if (tid == 0) {  // info may be set during this launch: one thread's view is the CTA's
    S.failed = *info;
    S.bad = kGroups;
    S.ended = 0;
  }
  __syncthreads();
  if (S.failed != 0) return;
  if (warp == kWarps) {  // the publishing warp: copies the groups from shared memory
    const int words = kSub * K * (int)sizeof(T) / 16;
    for (int q = 0; q < width / kSub; ++q) {
      bar_sync(kGroupBar + q, nt + 32);
      if (S.ended != 0) return;
      const double2* from = reinterpret_cast<const double2*>(stage + (size_t)K * kSub * q);
      double2* to = reinterpret_cast<double2*>(pub + (size_t)K * (c0 + kSub * q));
#pragma unroll 8
      for (int i = lane; i < words; i += 32) __stcg(to + i, from[i]);
      __syncwarp();
      // the compute threads may be in a later group by now: its failure leaves q < bad as it is
      const bool ok = q < *(volatile int*)&S.bad;
      if (lane == 0) store_release(flags + c0 / kSub + q, pack(epoch, ok, S.step.own + kSub * q));
      if (!ok) return;
    }
    bar_arrive(kGroupBar + kGroups, nt + 32);
    return;
  }
  T a[ROWS][NC];
  bool left[ROWS];  // rows not chosen yet
  int pos[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int i = tid + r * nt;
    left[r] = i < K;
    pos[r] = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k)
      a[r][k] = i < K && k < width ? in[(size_t)K * (c0 + k) + i] : zero_of<T>();
  }
  for (int p = 0; p < panels; ++p) {
    if (p == j) {
      const bool ok = eliminate(
          S.step, a, left, pos, width, c0, K, tid,
          [&](int jj) {  // hand the finished group's columns to the other CTAs
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
              const int i = tid + r * nt;
              if (i < K) {
#pragma unroll
                for (int k = 0; k < kSub; ++k)
                  stage[K * (jj - (kSub - 1) + k) + i] = a[r][NC - kSub + k];
              }
            }
            bar_arrive(kGroupBar + jj / kSub, nt + 32);
          },
          [&](int jj) {
            if (tid == 0) {
              S.bad = jj / kSub;
              atomicCAS(info, 0, kSingular);
            }
            bar_arrive(kGroupBar + jj / kSub, nt + 32);
          });
      if (!ok) return;
      continue;
    }
    const int groups = min(NC, K - p * NC) / kSub;
    for (int q = 0; q < groups; ++q) {
      const int g0 = p * NC + q * kSub;  // the group's first step
      if (warp == 0) {
        unsigned long long w;
        const bool came = wait_word(flags + g0 / kSub, epoch, kPollLimit, w);
        if (lane == 0) {
          if (!came) atomicCAS(info, 0, kRanOut);
          S.word = came && is_ok(w) ? w : 0ull;
        }
      }
      bar_sync(kStepBar, nt);
      const unsigned long long word = S.word;
      if (word == 0ull) {
        if (p < j) {  // the publishing warp waits for this CTA's first group: it ends as well
          if (tid == 0) S.ended = 1;
          bar_arrive(kGroupBar, nt + 32);
        }
        return;
      }
      T g[ROWS][kSub];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int i = tid + r * nt;
#pragma unroll
        for (int k = 0; k < kSub; ++k)
          g[r][k] = i < K ? load_l2(pub + (size_t)K * (g0 + k) + i) : zero_of<T>();
      }
#pragma unroll
      for (int k = 0; k < kSub; ++k) {
        const int piv = row_of(word, k);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (tid + r * nt == piv) {
            left[r] = false;
            pos[r] = g0 + k;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              S.rows[k][c] = a[r][c];
              a[r][c] = zero_of<T>();
            }
          }
      }
      bar_sync(kStepBar, nt);
#pragma unroll
      for (int k = 0; k < kSub; ++k)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const T b = S.rows[k][c];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) a[r][c] = fmadd(g[r][k], b, a[r][c]);
        }
    }
  }
  bar_sync(kGroupBar + kGroups, nt + 32);  // the publishing warp has read stage
  // the inverse's columns: rows in the order of their steps, through shared memory. (Only the
  // last panel can be narrow; its rotation leaves column k at place NC - width + k.)
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
    if (tid + r * nt < K) {
#pragma unroll
      for (int k = 0; k < NC; ++k)
        if (k >= NC - width) stage[(size_t)K * (k - (NC - width)) + pos[r]] = a[r][k];
    }
  bar_sync(kStepBar, nt);
  cuDoubleComplex* out = reinterpret_cast<cuDoubleComplex*>(place(at.out));
  for (int k = 0; k < width; ++k) {
    const size_t col = (size_t)K * S.step.own[k];
    for (int i = tid; i < K; i += nt) {
      const T v = stage[(size_t)K * k + i];
      if constexpr (kReal) {
        out[col + i] = make_cuDoubleComplex(v, 0.0);
        reinterpret_cast<double*>(place(at.real))[col + i] = v;
      } else {
        out[col + i] = v;
      }
    }
  }
}

// The kernel variant of a block order, and the launches with it.
template <class T, int NC, int ROWS, int Threads>
struct Variant {
  static constexpr int kThreads = Threads + 32;
  static int bytes(int K) {
    return (int)(sizeof(Shared<T, NC, Threads / 32>) + sizeof(T) * NC * (size_t)K);
  }
  // The number of systems whose CTAs are resident together, or a negative EB_* status.
  static int resident(int K) {
    auto kernel = k_ring_invert<T, NC, ROWS, Threads>;
    // the limit is the kernel's, not the launch's: always the most this variant can need, so that
    // another thread's smaller block does not lower it under this launch
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             bytes(ROWS * Threads)) != cudaSuccess)
      return check_launch("ring_invert attribute");
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, bytes(K)) !=
            cudaSuccess)
      return check_launch("ring_invert occupancy");
    const int fit = sms * per_sm / ((K + NC - 1) / NC);
    return fit < 1 ? fail(EB_ERR_CUDA, "ring_invert: the device cannot hold one block's CTAs") : fit;
  }
  static int launch(int K, int systems, char* base, int64_t stride, const InvertAt& at, int epoch,
                    cudaStream_t st) {
    auto kernel = k_ring_invert<T, NC, ROWS, Threads>;
    const int fit = resident(K);
    if (fit < 0) return fit;
    for (int z0 = 0; z0 < systems; z0 += fit) {
      const dim3 grid((K + NC - 1) / NC, std::min(fit, systems - z0));
      void* args[] = {(void*)&K,      (void*)&z0, (void*)&base,
                      (void*)&stride, (void*)&at, (void*)&epoch};
      if (cudaLaunchCooperativeKernel((const void*)kernel, grid, dim3(kThreads), args, bytes(K),
                                      st) != cudaSuccess)
        return check_launch("ring_invert");
    }
    return EB_OK;
  }
};

// Calls run with the variant for blocks of order K. Rows per thread: 128 compute threads (one warp per
// scheduler: the step's latency grows with the warps that share one) as long as a thread's rows
// fit its registers; above K = 512 more threads, which caps them (K = 1024 real: 1174 us at four
// rows, 1262 at two; complex: 2246 us at two rows and 512 threads, 2453 at four and 256).
template <class Run>
int with_variant(int K, bool real, Run run) {
  using Z = cuDoubleComplex;
  if (real)
    return K <= 128   ? run(Variant<double, 16, 1, 128>())
           : K <= 256 ? run(Variant<double, 16, 2, 128>())
           : K <= 512 ? run(Variant<double, 16, 4, 128>())
           : K <= 768 ? run(Variant<double, 16, 3, 256>())
                      : run(Variant<double, 16, 4, 256>());
  return K <= 128   ? run(Variant<Z, 8, 1, 128>())
         : K <= 256 ? run(Variant<Z, 8, 2, 128>())
         : K <= 512 ? run(Variant<Z, 8, 4, 128>())
         : K <= 768 ? run(Variant<Z, 8, 3, 256>())
                    : run(Variant<Z, 8, 2, 512>());
}

}  // namespace

int ring_invert(int K, int systems, char* base, int64_t stride, const InvertAt& at, int epoch,
                bool real, cudaStream_t st) {
  if (K < 4 || K > kMaxRows || K % 4 != 0 || systems < 1 || epoch < 1)
    return fail(EB_ERR_ARG, "ring_invert: bad sizes");
  return with_variant(K, real, [&](auto variant) {
    return variant.launch(K, systems, base, stride, at, epoch, st);
  });
}

int ring_invert_resident(int K, bool real) {
  return with_variant(K, real, [&](auto variant) { return variant.resident(K); });
}

int info_status(int info) {
  if (info == kRanOut)
    return fail(EB_ERR_CUDA, "ringlu: an inversion's wait for another CTA's pivots ran out");
  return info ? fail(EB_ERR_NAN, "ringlu: singular or non-finite ring block") : EB_OK;
}

}  // namespace rl
}  // namespace eb

extern "C" int eb_ringlu_wait_probe(int polls, void* scratch, void* stream) {
  using namespace eb;
  if (polls < 1 || polls > rl::kPollLimit || !scratch || (reinterpret_cast<uintptr_t>(scratch) & 15))
    return fail(EB_ERR_ARG, "wait probe: bad arguments");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto* flag = static_cast<unsigned long long*>(scratch);
  int* info = reinterpret_cast<int*>(flag + 1);
  int seen = 0;
  if (cudaMemsetAsync(scratch, 0, 16, st) != cudaSuccess) return check_launch("wait probe");
  rl::k_wait_probe<<<1, 32, 0, st>>>(flag, info, polls);
  if (cudaMemcpyAsync(&seen, info, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return check_launch("wait probe");
  return rl::info_status(seen);
}
