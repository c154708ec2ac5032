// d(odes)/d(states), d(odes)/d(vertices), d(odes)/d(velocities) and d(odes)/d(mach)
// (eb_compute_odes_wrt_*, replacing the complex-step procedures of
// src/spatial_discretization.f90:552-593, 666-750, 933-993, 1087-1143): one thread per cell, each
// of its four faces differentiated in closed form (jac_faces.cuh).
//
// A cell's outputs (nine 4 x 4 blocks, or four corners' 4 x 2 blocks) are what bounds these
// kernels: 1152 or 256 bytes per cell against about 1200 FP64 operations. Threads are the cells in
// their order in memory (radial index fastest), so a warp's 32 blocks of one slot are contiguous
// whatever the grid's sizes; each warp passes them through shared memory and writes them in
// whole 512-byte rows (written by the threads themselves, a store touched 32 lines for 16 bytes
// each). A block sum keeps the reference's face order, ((F_b + F_f) + F_i) + F_o.
//
// Measured on 282,000 cells of uneven grids against dual numbers (tiles staged in shared memory, at
// one CTA per SM): states 567 -> 80 us (4.1 TB/s of 6.5 copied), vertices 594 -> 45 us, velocities
// 263 -> 26 us, mach 34 -> 7.5 us. What is left is latency: the registers of a face's derivatives
// leave eight to twelve warps per SM.

#include "autotune.cuh"
#include "common.cuh"
#include "jac_faces.cuh"

#include <algorithm>

namespace eb {
namespace {

using Cell_ = CellAt<double, kDirNone>;
using Geometry_ = CellGeometry<double>;
using Line_ = RadialLine<double>;
using Face_ = FaceDerivatives<double>;

// Calls body(instance, warp's first cell, thread's cell, lane, valid cells of the warp) for a batch's
// cells, 32 to a warp. Grid y = instance, or one row for all: then the warps' cells of all
// instances, each rounded up to whole warps, are one range, and a warp finds its instance by the
// sums of the table's sizes. Whole warps stay in the loop together; the thread's cell is clamped to
// the instance.
template <class Body>
__device__ __forceinline__ void for_batch_cells(const Table& t, Body body) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool flat = t.dev != nullptr && (int)gridDim.y < t.n;
  for (int64_t w = blockIdx.x * (int64_t)warps + (threadIdx.x >> 5);;
       w += (int64_t)gridDim.x * warps) {
    int64_t part = w;  // the warp's place among its instance's
    int at = blockIdx.y;
    if (flat) {
      int base = 0;
      for (; base < t.n; base += 32) {
        int64_t sum = 0;
        if (base + lane < t.n)
          sum = ((int64_t)t.dev[base + lane].M * t.dev[base + lane].N + 31) / 32;
        const int64_t own = sum;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
          const int64_t before = __shfl_up_sync(0xffffffffu, sum, d);
          if (lane >= d) sum += before;
        }
        const unsigned past = __ballot_sync(0xffffffffu, sum > part);
        if (past != 0u) {
          const int k = __ffs(past) - 1;
          part -= __shfl_sync(0xffffffffu, sum - own, k);
          at = base + k;
          break;
        }
        part -= __shfl_sync(0xffffffffu, sum, 31);
      }
      if (base >= t.n) return;
    }
    const Instance in = t.dev ? t.dev[at] : t.single;
    const int64_t cells = (int64_t)in.M * in.N, first = 32 * part;
    if (first >= cells) return;
    body(in, first, min(first + lane, cells - 1), lane, (int)min((int64_t)32, cells - first));
  }
}

template <int Warps>
__global__ void __launch_bounds__(32 * Warps, Warps == 4 ? 3 : 4)
    k_jac_states_cells(Table t, const double* X, const double* V, const double* U, double* J) {
  __shared__ WarpRows<16> rows[Warps];
  WarpRows<16>& S = rows[threadIdx.x >> 5];
  for_batch_cells(t, [&](const Instance& in, int64_t first, int64_t local, int lane, int valid) {
    const int64_t slot = 16 * (int64_t)in.M * in.N;
    const Cell_ at(in, local, X, V, U, nullptr);
    const int m = at.m, M = in.M;
    const Geometry_ geo(at);
    const double s = -geo.inv_area();
    double* out = J + 144 * in.cell_offset + 16 * first;
    auto store = [&](int k, double (&a)[16], bool active) {
#pragma unroll
      for (int e = 0; e < 16; ++e) a[e] = active ? s * a[e] : 0.0;
      write_rows(S, a, lane, valid, out + slot * k);
    };
    double centre[16], a[16];
    clear(centre);
    const State<double> c = at.state(0, 0);
    {  // angular faces: b (line f, c, b, bb), then f (line b, c, f, ff)
      const State<double> fw = at.state(0, 1), bw = at.state(0, -1);
      double Qb[4], gb, c4b;  // face b's block of its outer state f
      {
        const State<double> bb = at.state(0, -2);
        const Face_ d(fw, c, bw, bb, geo.b, true, in);
        add_block(centre, d.of<true>(c), c, d.nx, d.nz, d.vl);
        clear(a);
        add_outer(a, d.Q, d.g_rr, d.c4, bb);
        store(kBB, a, true);
        clear(a);
        add_block(a, d.of<false>(bw), bw, d.nx, d.nz, d.vr);
#pragma unroll
        for (int k = 0; k < 4; ++k) Qb[k] = d.Q[k];
        gb = d.g_ll;
        c4b = d.c4;
      }
      const State<double> ff = at.state(0, 2);
      const Face_ d(bw, c, fw, ff, geo.f, true, in);
      add_block(centre, d.of<true>(c), c, d.nx, d.nz, d.vl);
      add_outer(a, d.Q, d.g_ll, -d.c4, bw);
      store(kB, a, true);
      clear(a);
      add_outer(a, Qb, gb, -c4b, fw);
      add_block(a, d.of<false>(fw), fw, d.nx, d.nz, d.vr);
      store(kF, a, true);
      clear(a);
      add_outer(a, d.Q, d.g_rr, d.c4, ff);
      store(kFF, a, true);
    }
    // radial faces: i (line o, c, i, ii), then o (line i, c, o, oo); a ghost's block goes to the
    // cell itself, through the ghost's derivative
    const Line_ line(at, c, geo, in);
    double Qi[4], gi, c4i;  // face i's block of its outer state o
    {
      const Face_ d(line.o, c, line.i, line.ii, geo.i, line.diss_i, in);
      add_block(centre, d.of<true>(c), c, d.nx, d.nz, d.vl);
      clear(a);
      add_outer(a, d.Q, d.g_rr, d.c4, line.ii);
      store(kII, a, m > 1);
      clear(a);
      add_block(a, d.of<false>(line.i), line.i, d.nx, d.nz, d.vr);
#pragma unroll
      for (int k = 0; k < 4; ++k) Qi[k] = d.Q[k];
      gi = d.g_ll;
      c4i = d.c4;
    }
    const Face_ d(line.i, c, line.o, line.oo, geo.o, line.diss_o, in);
    if (m == 0) through_wall(centre, a, geo.wall());
    if (m == M - 1) {  // face i's outer state is the far-field ghost: minus its block
      double e[16];
      clear(e);
      add_outer(e, Qi, gi, -c4i, line.o);
#pragma unroll
      for (int k = 0; k < 16; ++k) centre[k] -= e[k];
    }
    add_block(centre, d.of<true>(c), c, d.nx, d.nz, d.vl);
    if (m == 0) {
      double e[16];
      clear(e);
      add_outer(e, d.Q, d.g_ll, -d.c4, line.i);
      through_wall(centre, e, geo.wall());
    }
    add_outer(a, d.Q, d.g_ll, -d.c4, line.i);
    store(kI, a, m > 0);
    clear(a);
    add_outer(a, d.Q, d.g_rr, d.c4, line.oo);
    store(kOO, a, m < M - 2);
    clear(a);
    add_block(a, d.of<false>(line.o), line.o, d.nx, d.nz, d.vr);
    if (m == M - 1) {
#pragma unroll
      for (int k = 0; k < 16; ++k) centre[k] -= a[k];
    }
    add_outer(a, Qi, gi, -c4i, line.o);
    store(kO, a, m < M - 1);
    store(kC, centre, true);
  });
}

// The same by the wall's grid velocity (see ghost_by_normal).
__device__ __forceinline__ P2<double> ghost_by_velocity(const Wall<double>& w,
                                                        const State<double>& c, double e1,
                                                        double e2) {
  const double a = quot_(2.0 * c.u[0] * fma(e1, w.nx, e2 * w.nz), fma(w.nx, w.nx, w.nz * w.nz));
  return P2<double>{a * w.nx, a * w.nz};
}

// d(odes)/d(vertices) (Velo = false) or d(odes)/d(velocities): four corners' 4 x 2 blocks. The
// vertices' kernel holds four faces' derivatives by their normals at once: at two CTAs per SM (252
// registers) it took 58 us, at three (168, 900 bytes spilled) 67 us (a grid row per instance); the
// velocities' fits three.
template <bool Velo>
__global__ void __launch_bounds__(128, Velo ? 3 : 2)
    k_jac_corners_cells(Table t, const double* X, const double* V, const double* U, double* J) {
  __shared__ WarpRows<8> rows[4];
  WarpRows<8>& S = rows[threadIdx.x >> 5];
  for_batch_cells(t, [&](const Instance& in, int64_t first, int64_t local, int lane, int valid) {
    const int64_t slot = 8 * (int64_t)in.M * in.N;
    const Cell_ at(in, local, X, V, U, nullptr);
    const int m = at.m;
    const Geometry_ geo(at);
    const double ia = geo.inv_area();
    const State<double> c = at.state(0, 0);
    // per face (b, f, i, o): dF_k by its normal; or by its grid velocity, mean[k] times the normal,
    // and what the wall face's moves through the ghost
    double gx[4][4], gz[4][4], sum[4], mean[4][4], wx[4], wz[4];
    auto face = [&](int q, const State<double>& ll, const State<double>& r,
                    const State<double>& rr, const FaceGeometry<double>& f, bool diss) {
      if constexpr (Velo) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mean[q][k] = -0.5 * (c.u[k] + r.u[k]);
      } else {
        const Face_ d(ll, c, r, rr, f, diss, in);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          gx[q][k] = d.by_normal<true>(c, r, f, k);
          gz[q][k] = d.by_normal<false>(c, r, f, k);
          const double v = d.flux(ll, c, r, rr, k);
          sum[k] = q == 0 ? v : sum[k] + v;
        }
      }
    };
    {
      const State<double> fw = at.state(0, 1), bw = at.state(0, -1);
      if constexpr (Velo) {
        face(0, c, bw, c, geo.b, true);
        face(1, c, fw, c, geo.f, true);
      } else {
        face(0, fw, bw, at.state(0, -2), geo.b, true);
        face(1, bw, fw, at.state(0, 2), geo.f, true);
      }
    }
    const Line_ line(at, c, geo, in);
    face(2, line.o, line.i, line.ii, geo.i, line.diss_i);
    face(3, line.i, line.o, line.oo, geo.o, line.diss_o);
#pragma unroll
    for (int k = 0; k < 4; ++k) wx[k] = wz[k] = 0.0;
    if (m == 0) {  // the wall ghost is on both radial lines and moves with the inner face
      const Wall<double> w = geo.wall();
      double e[16], dp[4];
      clear(e);
      const Face_ di(line.o, c, line.i, line.ii, geo.i, line.diss_i, in);
      add_block(e, di.of<false>(line.i), line.i, di.nx, di.nz, di.vr);
      const Face_ dO(line.i, c, line.o, line.oo, geo.o, line.diss_o, in);
      grad_p(line.i, dp);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // face o's outer block: Q g_ll (x) dp - c4 I
        const double q = dO.Q[k] * dO.g_ll;
        const double e1 = e[k + 4] + fma(q, dp[1], k == 1 ? -dO.c4 : 0.0);
        const double e2 = e[k + 8] + fma(q, dp[2], k == 2 ? -dO.c4 : 0.0);
        const P2<double> a = Velo ? ghost_by_velocity(w, c, e1, e2) : ghost_by_normal(w, c, e1, e2);
        if constexpr (Velo) {
          wx[k] = a.x;
          wz[k] = a.z;
        } else {
          gx[2][k] += a.x;
          gz[2][k] += a.z;
        }
      }
    }
    double* out = J + 32 * in.cell_offset + 8 * first;
    const double sa = geo.cross < 0.0 ? -0.5 : 0.5;  // the area by the cross product
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      // corner k ends face `into` and begins face `from` (corners 0-1: i, 1-2: f, 2-3: o, 3-0: b)
      const int from = k == 0 ? 2 : k == 1 ? 1 : k == 2 ? 3 : 0;
      const int into = k == 0 ? 0 : k == 1 ? 2 : k == 2 ? 1 : 3;
      double a[8];
      if constexpr (Velo) {
        const FaceGeometry<double> faces[4] = {geo.b, geo.f, geo.i, geo.o};
        const FaceGeometry<double>&p = faces[from], &q = faces[into];
        const bool wall = from == 2 || into == 2;
        // -v / (2 area), corrected by its remainder: an entry has so few roundings of its own that the
        // inverse area's shows (error 1.83e-16 of the entries, root mean squares, 1.75 so)
        const double twice = fabs(geo.cross), half = 0.5 * ia;
        auto by_area = [&](double v) {
          const double t = v * half;
          return -fma(fma(-twice, t, v), half, t);
        };
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double x = fma(mean[from][r], p.nx, mean[into][r] * q.nx);
          const double z = fma(mean[from][r], p.nz, mean[into][r] * q.nz);
          a[r] = by_area(wall ? x + wx[r] : x);
          a[r + 4] = by_area(wall ? z + wz[r] : z);
        }
      } else {
        // cross = (x2 - x0) (z3 - z1) - (z2 - z0) (x3 - x1), by corner k's coordinates
        const P2<double> p = geo.x[(k + 1) & 3], q = geo.x[(k + 3) & 3];
        double ax = p.z - q.z, az = q.x - p.x;
        ax *= sa;
        az *= sa;
#pragma unroll
        for (int r = 0; r < 4; ++r) {  // the normal of the face p -> q is (z_q - z_p, x_p - x_q)
          const double R = -sum[r] * ia;
          a[r] = -ia * fma(R, ax, gz[from][r] - gz[into][r]);
          a[r + 4] = -ia * fma(R, az, gx[into][r] - gx[from][r]);
        }
      }
      write_rows(S, a, lane, valid, out + slot * k);
    }
  });
}

// d(odes)/d(mach): zero but for the far-field row, whose ghost 2 U_inf - U depends on the Mach
// number. Blocks of the grid's first part write the zeros (rows of whole warps), the rest take the
// far-field cells, one thread each (with a thread per cell, every warp that held a far-field cell
// ran its four faces for one lane).
__global__ void __launch_bounds__(128)
    k_jac_mach_cells(Table t, int zero_blocks, const double* X, const double* V, const double* U,
                     double* J) {
  const Instance in = t.dev ? t.dev[blockIdx.y] : t.single;
  const int64_t cells = (int64_t)in.M * in.N;
  double* Ji = J + 4 * in.cell_offset;
  if ((int)blockIdx.x < zero_blocks) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 2 * cells;
         e += (int64_t)zero_blocks * blockDim.x)
      if ((e >> 1) % in.M != in.M - 1) reinterpret_cast<double2*>(Ji)[e] = make_double2(0.0, 0.0);
    return;
  }
  for (int n = (blockIdx.x - zero_blocks) * blockDim.x + threadIdx.x; n < in.N;
       n += (gridDim.x - zero_blocks) * blockDim.x) {
    const int64_t local = in.M - 1 + (int64_t)in.M * n;
    const Cell_ at(in, local, X, V, U, nullptr);
    const Geometry_ geo(at);
    const State<double> c = at.state(0, 0);
    const Line_ line(at, c, geo, in);
    const Face_ di(line.o, c, line.i, line.ii, geo.i, line.diss_i, in);
    const Face_ dO(line.i, c, line.o, line.oo, geo.o, line.diss_o, in);
    double e[16];
    clear(e);
    add_outer(e, di.Q, di.g_ll, -di.c4, line.o);
    add_block(e, dO.of<false>(line.o), line.o, dO.nx, dO.nz, dO.vr);
    double d[4];
    ghost_by_mach(in, d);
    const double s = -geo.inv_area();
#pragma unroll
    for (int k = 0; k < 4; ++k)
      Ji[4 * local + k] = s * fma(e[k + 4], d[1], fma(e[k + 8], d[2], e[k + 12] * d[3]));
  }
}

// Grid of a kernel that goes through for_batch_cells. One grid row per instance, sized by the table's
// largest dimension squared, leaves an uneven batch most of its blocks without cells, and each
// still takes registers until it has read its instance's entry: 21 grids of 282,000 cells, 512 x 21
// blocks for 2,200 with cells, 207 us for the six Jacobians, 170 us as one flat range. The search
// reads the table in rounds of 32, so the flat range is for batches of up to four rounds that fill
// less than three quarters of the rows.
int cells_grid(const eb_batch* b, int threads, dim3& grid) {
  if (int rc = per_instance_grid(b, false, 1, threads, grid)) return rc;
  const int64_t square = (int64_t)b->max_dim * b->max_dim;
  if (b->n_inst > 1 && b->n_inst <= 128 && 4 * b->n_cells <= 3 * square * b->n_inst) {
    const int64_t blocks = b->n_cells / threads + b->n_inst;
    grid = dim3((unsigned)std::min<int64_t>(blocks, 148 * 64 * 8), 1);
  }
  return EB_OK;
}

template <int Warps>
int launch_states(const eb_batch* b, const Table& t, const double* X, const double* V,
                  const double* U, double* J, cudaStream_t st) {
  dim3 grid;
  if (int rc = cells_grid(b, 32 * Warps, grid)) return rc;
  k_jac_states_cells<Warps><<<grid, 32 * Warps, 0, st>>>(t, X, V, U, J);
  return check_launch("compute_odes_wrt_states");
}

}  // namespace

int launch_jac_states(const eb_batch* b, const double* X, const double* V, const double* U,
                      double* J, cudaStream_t st) {
  const Table t = make_table(b);
  static const char* const kNames[2] = {"width 4 (warps per CTA)", "width 2 (warps per CTA)"};
  return tune::launch_tuned("jac_states_tiled", b->n_cells, b->max_dim, 2, 0, kNames, st,
                            [&](int v) {
                              return v == 0 ? launch_states<4>(b, t, X, V, U, J, st)
                                            : launch_states<2>(b, t, X, V, U, J, st);
                            });
}

int launch_jac_corners(const eb_batch* b, bool velocities, const double* X, const double* V,
                       const double* U, double* J, cudaStream_t st) {
  const Table t = make_table(b);
  dim3 grid;
  if (int rc = cells_grid(b, 128, grid)) return rc;
  if (velocities) k_jac_corners_cells<true><<<grid, 128, 0, st>>>(t, X, V, U, J);
  else k_jac_corners_cells<false><<<grid, 128, 0, st>>>(t, X, V, U, J);
  return check_launch(velocities ? "compute_odes_wrt_velocities" : "compute_odes_wrt_vertices");
}

int launch_jac_mach(const eb_batch* b, const double* X, const double* V, const double* U,
                    double* J, cudaStream_t st) {
  const Table t = make_table(b);
  dim3 grid;
  if (int rc = per_instance_grid(b, false, 1, 512, grid)) return rc;
  const int N = b->n_inst > 1 || b->d_table ? b->max_dim : b->single.N;
  const int zero_blocks = (int)grid.x;
  grid.x += (N + 127) / 128;
  k_jac_mach_cells<<<grid, 128, 0, st>>>(t, zero_blocks, X, V, U, J);
  return check_launch("compute_odes_wrt_mach");
}

}  // namespace eb
