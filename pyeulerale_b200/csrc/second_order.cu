// C ABI of the second-order building blocks: directional derivatives of the Jacobians, the real and
// imaginary parts of a complex direction as a dual's two tangents (B = Dual<double, 2>). They
// replace the four complex-step Jacobian rebuilds per call of the reference's finite-difference
// second-order routines (src/py_euler_ale/core.py:718-1275).
//
// The residual's state and vertex Jacobians are the closed forms of jac_faces.cuh evaluated in
// duals, one thread per cell and block: three numbers per scalar, where duals nested in duals
// carried fifteen. What bounds them is FP64 arithmetic in few threads (a block of one cell
// evaluates one to four faces of about 1,000 operations); the grid's z is the slot or the corner, since a
// 128 x 128 grid with a thread per cell alone would leave an SM four warps.
// Measured on a 128 x 128 grid, directions of the states, inputs not in L2: states Jacobian 382 us
// nested, 61 us now (1240 us before each slot had its threads); vertices Jacobian 208 us nested, 53 us
// now (427 us).

#include "jac_faces.cuh"
#include "jacobian_kernels.cuh"

using namespace eb;

namespace eb {
namespace {

// Both parts of a warp's blocks.
template <int D>
__device__ __forceinline__ void write_parts(WarpRows<D>& S, const D2 (&a)[D], int lane, int valid,
                                            double* re, double* im) {
  double part[D];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int e = 0; e < D; ++e) part[e] = a[e].d[i];
    write_rows(S, part, lane, valid, i ? im : re);
  }
}

// Directional derivatives of d(odes)/d(states); grid z: slots. A face contributes to the blocks of
// its own four states, a ghost's block to the cell's through the ghost's derivative.
template <int Kind>
__global__ void __launch_bounds__(128)
    k_states_dir(Table t, const double* X, const double* V, const double* U, const double* D,
                 double* Jre, double* Jim) {
  __shared__ WarpRows<16> rows[4];
  const Instance in = t.dev ? t.dev[blockIdx.y] : t.single;
  WarpRows<16>& S = rows[threadIdx.x >> 5];
  const int slot = blockIdx.z, sm = slot_dm(slot), sn = slot_dn(slot);
  const int64_t base = 144 * in.cell_offset + 16 * (int64_t)in.M * in.N * slot;
  for_cells(in, [&](int64_t first, int64_t local, int lane, int valid) {
    const CellAt<D2, Kind> at(in, local, X, V, U, D);
    const bool active = at.m + sm >= 0 && at.m + sm < in.M;
    const State<D2> c = at.state(0, 0);
    D2 a[16];
    clear(a);
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const int dm = q < 2 ? 0 : q == 2 ? -1 : 1, dn = q > 1 ? 0 : q == 0 ? -1 : 1;
      const bool own = slot == kC, is_r = sm == dm && sn == dn, is_ll = sm == -dm && sn == -dn;
      const bool is_rr = sm == 2 * dm && sn == 2 * dn;
      if (!(own || is_r || is_ll || is_rr) || !active) continue;
      const NumberedFace<D2, Kind> n(at, c, q, in);
      const FaceDerivatives<D2> d(n.ll, c, n.r, n.rr, n.f, n.diss, in);
      if (own) add_block(a, d.template of<true>(c), c, d.nx, d.nz, d.vl);
      if (is_rr) add_outer(a, d.Q, d.g_rr, d.c4, n.rr);
      if (is_r || (own && n.r_ghost) || is_ll || (own && n.ll_ghost)) {
        D2 e[16];
        clear(e);
        if (is_r || (own && n.r_ghost))
          add_block(e, d.template of<false>(n.r), n.r, d.nx, d.nz, d.vr);
        else
          add_outer(e, d.Q, d.g_ll, -d.c4, n.ll);
        if (own && at.m == 0) {
          through_wall(a, e, NumberedFace<D2, Kind>::wall(at));
        } else {
          const double sign = own ? -1.0 : 1.0;  // the far-field ghost: minus its block
#pragma unroll
          for (int k = 0; k < 16; ++k) a[k] = mad(sign, e[k], a[k]);
        }
      }
    }
    const D2 s = -recip_(abs_c(cross_of(at)) * 0.5);
#pragma unroll
    for (int e = 0; e < 16; ++e) a[e] = active ? s * a[e] : lift<D2>(0.0);
    write_parts(S, a, lane, valid, Jre + base + 16 * first, Jim + base + 16 * first);
  });
}

// Directional derivatives of d(odes)/d(vertices); grid z: corners. A corner moves the normals of the
// two faces that meet at it, the area, and at the wall the ghost's state.
template <int Kind>
__global__ void __launch_bounds__(128)
    k_vertices_dir(Table t, const double* X, const double* V, const double* U, const double* D,
                   double* Jre, double* Jim) {
  __shared__ WarpRows<8> rows[4];
  const Instance in = t.dev ? t.dev[blockIdx.y] : t.single;
  WarpRows<8>& S = rows[threadIdx.x >> 5];
  const int corner = blockIdx.z;
  // corner k ends face `into` and begins face `from` (corners 0-1: i, 1-2: f, 2-3: o, 3-0: b)
  const int from = corner == 0 ? 2 : corner == 1 ? 1 : corner == 2 ? 3 : 0;
  const int into = corner == 0 ? 0 : corner == 1 ? 2 : corner == 2 ? 1 : 3;
  const int64_t base = 32 * in.cell_offset + 8 * (int64_t)in.M * in.N * corner;
  for_cells(in, [&](int64_t first, int64_t local, int lane, int valid) {
    const CellAt<D2, Kind> at(in, local, X, V, U, D);
    const State<D2> c = at.state(0, 0);
    D2 a[8], sum[4];  // a: by x, then by z
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = a[k + 4] = sum[k] = lift<D2>(0.0);
    const bool by_ghost = at.m == 0 && (from == 2 || into == 2);
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const NumberedFace<D2, Kind> n(at, c, q, in);
      const FaceDerivatives<D2> d(n.ll, c, n.r, n.rr, n.f, n.diss, in);
      // the normal of the face p -> q is (z_q - z_p, x_p - x_q): `into` moves z_q by +, x_q by -
      const double sign = q == into ? 1.0 : -1.0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        sum[k] = sum[k] + d.flux(n.ll, c, n.r, n.rr, k);
        if (q == into || q == from) {
          a[k] = mad(-sign, d.template by_normal<false>(c, n.r, n.f, k), a[k]);
          a[k + 4] = mad(sign, d.template by_normal<true>(c, n.r, n.f, k), a[k + 4]);
        }
      }
      if (by_ghost && q > 1) {  // the wall ghost is on both radial lines
        const Wall<D2> w = NumberedFace<D2, Kind>::wall(at);
        D2 e[16];
        clear(e);
        if (q == 2) add_block(e, d.template of<false>(n.r), n.r, d.nx, d.nz, d.vr);
        else add_outer(e, d.Q, d.g_ll, -d.c4, n.ll);
        const double si = into == 2 ? 1.0 : -1.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const P2<D2> g = ghost_by_normal(w, c, e[k + 4], e[k + 8]);
          a[k] = mad(-si, g.z, a[k]);
          a[k + 4] = mad(si, g.x, a[k + 4]);
        }
      }
    }
    const D2 cross = cross_of(at), s = -recip_(abs_c(cross) * 0.5);
    const double sa = value(cross) < 0.0 ? -0.5 : 0.5;  // the area by the cross product
    // cross = (x2 - x0) (z3 - z1) - (z2 - z0) (x3 - x1), by this corner's coordinates
    const P2<D2> p = at.template corner<false>((corner + 1) & 3);
    const P2<D2> q = at.template corner<false>((corner + 3) & 3);
    const D2 ax = sa * (p.z - q.z), az = sa * (q.x - p.x);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const D2 R = sum[k] * s;
      a[k] = s * mad(R, ax, a[k]);
      a[k + 4] = s * mad(R, az, a[k + 4]);
    }
    write_parts(S, a, lane, valid, Jre + base + 8 * first, Jim + base + 8 * first);
  });
}

}  // namespace
}  // namespace eb

extern "C" {

#define EB_DIR_DISPATCH(LAUNCH)                                                               \
  switch (dir_kind) {                                                                       \
    case kDirStates: LAUNCH(kDirStates); break;                                             \
    case kDirVertices: LAUNCH(kDirVertices); break;                                         \
    case kDirVelocities: LAUNCH(kDirVelocities); break;                                     \
    default:                                                                                \
      return fail(EB_ERR_ARG, "dir_kind must be 0 (states), 1 (vertices) or 2 (velocities)"); \
  }

int eb_odes_wrt_mach_dir(const eb_batch* b, const double* X, const double* V, const double* U,
                         int dir_kind, const double* d, double* J_re, double* J_im,
                         void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, d, J_re, J_im);
  if (!X || !U || !d || !J_re || !J_im) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  dim3 jgrid;
  if (int rc = per_instance_grid(b, false, 1, 128, jgrid)) return rc;
#define EB_LAUNCH(K)                                                                        \
  k_jac_mach<D2, K>                                                                         \
      <<<jgrid, 128, 0, EB_STREAM(stream)>>>(t, b->n_cells, X, V, U, d, nullptr, J_re, J_im)
  EB_DIR_DISPATCH(EB_LAUNCH)
#undef EB_LAUNCH
  return check_launch("odes_wrt_mach_dir");
}

int eb_odes_wrt_states_dir(const eb_batch* b, const double* X, const double* V,
                           const double* U, int dir_kind, const double* d, double* J_re,
                           double* J_im, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, d, J_re, J_im);
  if (!X || !U || !d || !J_re || !J_im) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  dim3 jgrid;
  if (int rc = per_instance_grid(b, false, 1, 128, jgrid)) return rc;
  jgrid.z = 9;
#define EB_LAUNCH(K) \
  k_states_dir<K><<<jgrid, 128, 0, EB_STREAM(stream)>>>(t, X, V, U, d, J_re, J_im)
  EB_DIR_DISPATCH(EB_LAUNCH)
#undef EB_LAUNCH
  return check_launch("odes_wrt_states_dir");
}

int eb_odes_wrt_vertices_dir(const eb_batch* b, const double* X, const double* V,
                             const double* U, int dir_kind, const double* d, double* J_re,
                             double* J_im, void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, V, U, d, J_re, J_im);
  if (!X || !U || !d || !J_re || !J_im) return fail(EB_ERR_ARG, "null array");
  const Table t = make_table(b);
  dim3 jgrid;
  if (int rc = per_instance_grid(b, false, 1, 128, jgrid)) return rc;
  jgrid.z = 4;
#define EB_LAUNCH(K) \
  k_vertices_dir<K><<<jgrid, 128, 0, EB_STREAM(stream)>>>(t, X, V, U, d, J_re, J_im)
  EB_DIR_DISPATCH(EB_LAUNCH)
#undef EB_LAUNCH
  return check_launch("odes_wrt_vertices_dir");
}

int eb_forces_wrt_states_dir(const eb_batch* b, const double* X, const double* U,
                             int dir_kind, const double* d, double* J_re, double* J_im,
                             void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, U, d, J_re, J_im);
  if (!X || !U || !d || !J_re || !J_im) return fail(EB_ERR_ARG, "null array");
  if (dir_kind != kDirStates && dir_kind != kDirVertices)
    return fail(EB_ERR_ARG, "forces depend on states and vertices only");
  const Table t = make_table(b);
  const int g = grid_for(b->n_wall, 128);
  cudaStream_t s = EB_STREAM(stream);
  if (dir_kind == kDirStates)
    k_jac_forces_states<D2, kDirStates><<<g, 128, 0, s>>>(t, b->n_wall, X, U, d, nullptr, J_re, J_im);
  else
    k_jac_forces_states<D2, kDirVertices><<<g, 128, 0, s>>>(t, b->n_wall, X, U, d, nullptr, J_re, J_im);
  return check_launch("forces_wrt_states_dir");
}

int eb_forces_wrt_vertices_dir(const eb_batch* b, const double* X, const double* U,
                               int dir_kind, const double* d, double* J_re, double* J_im,
                               void* stream) {
  EB_VALIDATE(b);
  EB_ALIGNED(X, U, d, J_re, J_im);
  if (!X || !U || !d || !J_re || !J_im) return fail(EB_ERR_ARG, "null array");
  if (dir_kind != kDirStates && dir_kind != kDirVertices)
    return fail(EB_ERR_ARG, "forces depend on states and vertices only");
  const Table t = make_table(b);
  const int g = grid_for(b->n_wall, 128);
  cudaStream_t s = EB_STREAM(stream);
  if (dir_kind == kDirStates)
    k_jac_forces_vertices<D2, kDirStates><<<g, 128, 0, s>>>(t, b->n_wall, X, U, d, nullptr, J_re, J_im);
  else
    k_jac_forces_vertices<D2, kDirVertices><<<g, 128, 0, s>>>(t, b->n_wall, X, U, d, nullptr, J_re, J_im);
  return check_launch("forces_wrt_vertices_dir");
}

}  // extern "C"
