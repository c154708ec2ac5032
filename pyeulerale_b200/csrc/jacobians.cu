// C ABI of the first-order Jacobians, replacing the complex-step procedures of
// src/spatial_discretization.f90: the residual's by the closed-form kernels of jac_cells.cu, the
// forces' by the dual-number kernels of jacobian_kernels.cuh with B = double; and the residual's by
// the states in dual numbers, for comparison.

#include "jacobian_kernels.cuh"

using namespace eb;

namespace eb {
// The Jacobians of the residual in closed form (jac_cells.cu).
int launch_jac_states(const eb_batch* b, const double* X, const double* V, const double* U,
                      double* J, cudaStream_t st);
int launch_jac_corners(const eb_batch* b, bool velocities, const double* X, const double* V,
                       const double* U, double* J, cudaStream_t st);
int launch_jac_mach(const eb_batch* b, const double* X, const double* V, const double* U,
                    double* J, cudaStream_t st);

namespace {

// Face flux kept out of line: the dual-number states Jacobian evaluates it in a loop with a wide
// type, and inlining every case makes the kernel very large.
template <class R, class SP, class TX, class TV, class TM>
__device__ __noinline__ S4<R> face_call(int q, int flag, const SP& u, const Geometry<TX, TV>& g,
                                        const TM& mach, const Instance& in) {
  return face<R>(q, flag, u, g, mach, in);
}

// State provider for the states Jacobian: the states of slot `seed_slot` carry the identity
// tangent, every other state a zero tangent.
struct SeededStates {
  const Plain* p;
  int seed_slot;
  EB_HD S4<Dual<double, 4>> operator()(int s) const {
    S4<Dual<double, 4>> r;
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = seed<double, 4>(p->u[s].v[k], s == seed_slot ? k : -1);
    return r;
  }
};

// d(odes)/d(states) blocks (compute_odes_wrt_states, f90:666-750) by dual numbers. Each slot's
// block sums only the faces that read that slot (others contribute exactly zero). Grid z: slots.
__global__ void __launch_bounds__(128) k_jac_states(Table t, const double* X, const double* V,
                                                    const double* U, double* J) {
  using R = Dual<double, 4>;
  const Instance in = t.dev ? t.dev[blockIdx.y] : t.single;  // grid y = instance
  const int64_t cells = (int64_t)in.M * in.N;
  for (int64_t local = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; local < cells;
       local += (int64_t)gridDim.x * blockDim.x) {
    Plain p;
    load_plain(in, local, X, V, U, p);
    const Geometry<double, double> geo = geometry(p.x, p.w);
    const int s = blockIdx.z;
    double* out = J + 144 * in.cell_offset + 16 * local + 16 * cells * s;
    double acc[4][4] = {};
    const bool active = slot_active(s, p.m, in.M);
    const SeededStates prov{&p, s};
    for (int q = 0; q < 4; ++q) {
      if (!active || !face_uses_slot(q, p.flag, s)) continue;
      const S4<R> f = face_call<R>(q, p.flag, prov, geo, in.mach, in);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[r][i] = acc[r][i] + f.v[r].d[i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int r = 0; r < 4; ++r) out[r + 4 * i] = active ? -acc[r][i] / geo.area : 0.0;
  }
}

}  // namespace
}  // namespace eb

extern "C" {

int eb_compute_odes_wrt_mach(const eb_batch* b, const double* X, const double* V,
                             const double* U, double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  return launch_jac_mach(b, X, V, U, J, EB_STREAM(stream));
}

int eb_compute_odes_wrt_states(const eb_batch* b, const double* X, const double* V,
                               const double* U, double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  return launch_jac_states(b, X, V, U, J, EB_STREAM(stream));
}

// The per-cell states Jacobian (one thread per cell, each block from its own face evaluations).
// Kept as the plain variant for comparison; the closed-form kernel serves eb_compute_odes_wrt_states.
int eb_compute_odes_wrt_states_untiled(const eb_batch* b, const double* X, const double* V,
                                       const double* U, double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  dim3 jgrid;
  if (int rc = per_instance_grid(b, false, 1, 128, jgrid)) return rc;
  jgrid.z = 9;
  k_jac_states<<<jgrid, 128, 0, EB_STREAM(stream)>>>(t, X, V, U, J);
  return check_launch("compute_odes_wrt_states_untiled");
}

int eb_compute_odes_wrt_vertices(const eb_batch* b, const double* X, const double* V,
                                 const double* U, double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  return launch_jac_corners(b, false, X, V, U, J, EB_STREAM(stream));
}

int eb_compute_odes_wrt_velocities(const eb_batch* b, const double* X, const double* V,
                                   const double* U, double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  return launch_jac_corners(b, true, X, V, U, J, EB_STREAM(stream));
}

int eb_compute_forces_wrt_states(const eb_batch* b, const double* X, const double* U,
                                 double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  k_jac_forces_states<double, kDirNone><<<grid_for(b->n_wall, 128), 128, 0, EB_STREAM(stream)>>>(
      t, b->n_wall, X, U, nullptr, J, nullptr, nullptr);
  return check_launch("compute_forces_wrt_states");
}

int eb_compute_forces_wrt_vertices(const eb_batch* b, const double* X, const double* U,
                                   double* J, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, U, J);
  if (!X || !U || !J) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  k_jac_forces_vertices<double, kDirNone>
      <<<grid_for(b->n_wall, 128), 128, 0, EB_STREAM(stream)>>>(t, b->n_wall, X, U, nullptr, J,
                                                                 nullptr, nullptr);
  return check_launch("compute_forces_wrt_vertices");
}

}  // extern "C"
