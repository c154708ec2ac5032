// Closed-form derivatives of one face's flux (make_face_flux, src/spatial_discretization.f90:
// 189-274), for the Jacobian kernels (jac_cells.cu).
//
// A JST face flux in the orientation of its cell l, with the stencil line ll, l, r, rr, is
//   F = central(l, r, n) - (l + r)/2 vn - c2 (r - l) + c4 (rr - 3 r + 3 l - ll),
//   c2 = k2 S lambda,  c4 = max_c(0, k4 lambda - c4c c2),
// S the larger (max_c) of the two pressure sensors and lambda of the two spectral radii. Its
// derivative with respect to a state is therefore the central flux's own Jacobian, a multiple of
// the identity, and two rank-one terms: the derivative of the flux by S (the vector Q) times the
// sensor's derivative, which reaches a state only through its pressure, and the derivative by
// lambda (the vector h) times lambda's, which reaches the state whose spectral radius was taken.
// So each 4 x 4 block is  alpha (x) dp + beta (x) dv + extra (x) e_0 + diag I  with dp and dv the
// gradients of the state's pressure and normal velocity: about two multiply-adds per entry,
// where dual numbers carried four derivative components through every operation of the flux and
// repeated it for each seeded state.
//
// The values that decide branches (abs_c's sign, max_c's choice, f90:97-120) are formed as the
// reference forms them, in plain operations (this code is compiled without contraction), so ties
// at degenerate states, e.g. an exact free stream, fall as in the reference; the derivatives,
// which decide nothing, use explicit fused multiply-adds.
#pragma once

#include "physics.cuh"

namespace eb {

struct State {  // a conserved state with what its faces need
  double u[4];  // rho, j1, j2, e
  double p, ir, vx, vz;  // pressure, 1 / rho, velocity
};

__device__ __forceinline__ State make_state(double rho, double j1, double j2, double e) {
  State s;
  s.u[0] = rho;
  s.u[1] = j1;
  s.u[2] = j2;
  s.u[3] = e;
  s.ir = recip_(rho);
  s.p = kGm1 * (e - (j1 * j1 + j2 * j2) * s.ir * 0.5);
  s.vx = j1 * s.ir;
  s.vz = j2 * s.ir;
  return s;
}

// Gradient of the pressure by the conserved variables.
__device__ __forceinline__ void grad_p(const State& s, double (&g)[4]) {
  g[0] = kGm1 * 0.5 * fma(s.vx, s.vx, s.vz * s.vz);
  g[1] = -kGm1 * s.vx;
  g[2] = -kGm1 * s.vz;
  g[3] = kGm1;
}

struct Wall {  // a wall face: normal, grid velocity, n.g and 1 / |n|^2
  double nx, nz, gx, gz, gn, inn;
};
__device__ __forceinline__ Wall make_wall(double nx, double nz, double gx, double gz) {
  return Wall{nx, nz, gx, gz, nx * gx + nz * gz, recip_(nx * nx + nz * nz)};
}
// make_wall_ghost_state, f90:231-240.
__device__ __forceinline__ State wall_ghost_of(const State& s, const Wall& w) {
  const double proj = w.nx * (s.u[1] - w.gx * s.u[0]) + w.nz * (s.u[2] - w.gz * s.u[0]);
  const double nn = w.nx * w.nx + w.nz * w.nz;
  return make_state(s.u[0], s.u[1] - quot_(2.0 * w.nx * proj, nn),
                    s.u[2] - quot_(2.0 * w.nz * proj, nn), s.u[3]);
}
// make_farfield_ghost_state, f90:269-274: 2 U_inf - U.
__device__ __forceinline__ State farfield_ghost_of(const State& s, const Instance& in) {
  const double speed = in.mach * sqrt_(kGamma);
  const double f1 = speed * in.cos_aoa, f2 = speed * in.sin_aoa;
  const double fe = 1.0 / kGm1 + speed * speed / 2.0;
  return make_state(2.0 - s.u[0], 2.0 * f1 - s.u[1], 2.0 * f2 - s.u[2], 2.0 * fe - s.u[3]);
}

struct FaceGeometry {  // normal, grid velocity
  double nx, nz, gx, gz;
};

// The derivative of a face flux by one of its states, factored (see above).
struct Block {
  double alpha[4], beta[4], extra[4], diag;
};

// A face's flux in its cell's orientation, differentiated. diss = false: the central flux of the
// faces next to the boundaries (f90:197, 219); ll and rr need then only be finite.
struct FaceDerivatives {
  double nx, nz, vn, vl, vr;
  double Q[4], h[4];            // dF/dS, dF/dlambda (zero without dissipation)
  double g_ll, g_l, g_r, g_rr;  // dS/dp of the four states
  double c2, c4;
  bool lam_l;                   // lambda is l's (else r's)
  double sgn, c, len, ilen;     // that state's sign of the normal velocity and speed of sound; |n|

  __device__ __forceinline__ FaceDerivatives(const State& ll, const State& l, const State& r,
                                             const State& rr, const FaceGeometry& f, bool diss,
                                             const Instance& in) {
    nx = f.nx;
    nz = f.nz;
    vn = f.gx * nx + f.gz * nz;
    vl = (nx * l.u[1] + nz * l.u[2]) * l.ir;
    vr = (nx * r.u[1] + nz * r.u[2]) * r.ir;
    len = sqrt_(nx * nx + nz * nz);
    ilen = recip_(len);
    const double cl = sqrt_(kGamma * l.p * l.ir), cr = sqrt_(kGamma * r.p * r.ir);
    const double al = abs_c(vl) + cl * len, ar = abs_c(vr) + cr * len;
    lam_l = al > ar + 1e-8;
    const double lam = lam_l ? al : ar;
    c = lam_l ? cl : cr;
    sgn = (lam_l ? vl : vr) < 0.0 ? -1.0 : 1.0;
    const double num_l = ll.p - 2.0 * l.p + r.p, den_l = ll.p + 2.0 * l.p + r.p;
    const double num_r = l.p - 2.0 * r.p + rr.p, den_r = l.p + 2.0 * r.p + rr.p;
    const double sl = quot_(abs_c(num_l), den_l), sr = quot_(abs_c(num_r), den_r);
    const bool s_l = sl > sr + 1e-8;
    const double S = s_l ? sl : sr;
    const double sg = (s_l ? num_l : num_r) < 0.0 ? -1.0 : 1.0;
    const double inv = recip_(s_l ? den_l : den_r);
    const double outer = (sg - S) * inv, centre = -2.0 * (sg + S) * inv;
    g_ll = s_l ? outer : 0.0;
    g_l = s_l ? centre : outer;
    g_r = s_l ? outer : centre;
    g_rr = s_l ? 0.0 : outer;
    c2 = in.k2 * S * lam;
    c4 = in.k4 * lam - in.c4 * c2;
    const bool active = !(0.0 > c4 + 1e-8);  // max_c(0, c4)
    const double on = diss ? 1.0 : 0.0, on4 = active ? on : 0.0;
    c2 *= on;
    c4 *= on4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double d1 = r.u[k] - l.u[k];
      const double d3 = fma(3.0, l.u[k] - r.u[k], rr.u[k] - ll.u[k]);
      const double by_c2 = -fma(on4 * in.c4, d3, on * d1);  // dF/dc2 (through c4 as well)
      Q[k] = by_c2 * (in.k2 * lam);
      h[k] = fma(by_c2, in.k2 * S, on4 * in.k4 * d3);
    }
  }

  // dF/dl (Left) or dF/dr.
  template <bool Left>
  __device__ __forceinline__ Block of(const State& s) const {
    Block b;
    const double v = Left ? vl : vr, g = Left ? g_l : g_r;
    const bool lam = Left == lam_l;
    // dlambda = sgn dv + len dc, dc = c / (2 p) dp - c / (2 rho) e_0
    const double lp = lam ? quot_(0.5 * len * c, s.p) : 0.0, le = lam ? -0.5 * len * c * s.ir : 0.0;
    const double lv = lam ? sgn : 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double n = k == 1 ? 0.5 * nx : k == 2 ? 0.5 * nz : k == 3 ? 0.5 * v : 0.0;
      b.alpha[k] = fma(h[k], lp, fma(Q[k], g, n));
      b.beta[k] = fma(h[k], lv, 0.5 * (k == 3 ? s.u[3] + s.p : s.u[k]));
      b.extra[k] = h[k] * le;
    }
    b.diag = fma(0.5, v - vn, Left ? fma(3.0, c4, c2) : -fma(3.0, c4, c2));
    return b;
  }

  // Flux component k (the central flux, the grid velocity's part and the dissipation).
  __device__ __forceinline__ double flux(const State& ll, const State& l, const State& r,
                                         const State& rr, int k) const {
    const double n = k == 1 ? nx : k == 2 ? nz : 0.0;
    double f = 0.5 * (fma(l.u[k], vl - vn, r.u[k] * (vr - vn)) + n * (l.p + r.p));
    if (k == 3) f += 0.5 * fma(l.p, vl, r.p * vr);
    const double d1 = r.u[k] - l.u[k];
    const double d3 = fma(3.0, l.u[k] - r.u[k], rr.u[k] - ll.u[k]);
    return fma(c4, d3, fma(-c2, d1, f));
  }

  // Derivative of flux component k by the normal (nx if X, else nz) at fixed states.
  template <bool X>
  __device__ __forceinline__ double by_normal(const State& l, const State& r, const FaceGeometry& f,
                                              int k) const {
    const double ul = X ? l.vx : l.vz, ur = X ? r.vx : r.vz, g = X ? f.gx : f.gz;
    double d = 0.5 * fma(l.u[k], ul - g, r.u[k] * (ur - g));
    if (k == (X ? 1 : 2)) d += 0.5 * (l.p + r.p);
    if (k == 3) d += 0.5 * fma(l.p, ul, r.p * ur);
    const double lam = fma(sgn, lam_l ? ul : ur, c * (X ? nx : nz) * ilen);
    return fma(h[k], lam, d);
  }
};

// block += E, a full 4 x 4 (column-major: entry k + 4 j is dF_k/du_j) of one of the line's states.
__device__ __forceinline__ void add_block(double (&acc)[16], const Block& b, const State& s,
                                          double nx, double nz, double v) {
  double dp[4];
  grad_p(s, dp);
  const double dv[3] = {-v * s.ir, nx * s.ir, nz * s.ir};
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      double e = fma(b.alpha[k], dp[j], acc[k + 4 * j]);
      if (j < 3) e = fma(b.beta[k], dv[j], e);
      if (j == 0) e += b.extra[k];
      if (j == k) e += b.diag;
      acc[k + 4 * j] = e;
    }
}
// The blocks of the line's outer states, Q g (x) dp + diag I.
__device__ __forceinline__ void add_outer(double (&acc)[16], const double (&Q)[4], double g,
                                          double diag, const State& s) {
  double dp[4];
  grad_p(s, dp);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double a = Q[k] * g;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[k + 4 * j] = fma(a, dp[j], acc[k + 4 * j]);
      if (j == k) acc[k + 4 * j] += diag;
    }
  }
}

// acc += E G with G the derivative of the wall ghost by its state.
__device__ __forceinline__ void through_wall(double (&acc)[16], const double (&E)[16],
                                             const Wall& w) {
  const double ax = 2.0 * w.nx * w.inn, az = 2.0 * w.nz * w.inn;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double e1 = E[k + 4], e2 = E[k + 8];
    const double t = fma(e1, ax, e2 * az);  // along the reflected normal
    acc[k] += fma(t, w.gn, E[k]);
    acc[k + 4] += fma(-t, w.nx, e1);
    acc[k + 8] += fma(-t, w.nz, e2);
    acc[k + 12] += E[k + 12];
  }
}

}  // namespace eb
