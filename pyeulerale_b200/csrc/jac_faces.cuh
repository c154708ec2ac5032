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
//
// Everything is a template on the scalar type: double gives the Jacobians (jac_cells.cu), dual
// numbers their derivatives along a direction (second_order.cu).
#pragma once

#include "common.cuh"

namespace eb {

// a b + c with explicit fused multiply-adds, also in the tangents of duals.
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
template <class T, int K, class B, class C>
__device__ __forceinline__ Dual<T, K> mad_dual(const B& a, const C& b, const Dual<T, K>& c) {
  Dual<T, K> r;
  r.v = mad(value(a), value(b), c.v);
#pragma unroll
  for (int i = 0; i < K; ++i) {
    r.d[i] = c.d[i];
    if constexpr (is_dual<B>::value) r.d[i] = mad(a.d[i], value(b), r.d[i]);
    if constexpr (is_dual<C>::value) r.d[i] = mad(value(a), b.d[i], r.d[i]);
  }
  return r;
}
template <class A, class B, class C>
__device__ __forceinline__ std::enable_if_t<is_dual<promote_t<A, promote_t<B, C>>>::value,
                                            promote_t<A, promote_t<B, C>>>
mad(const A& a, const B& b, const C& c) {
  return mad_dual(a, b, lift<promote_t<A, promote_t<B, C>>>(c));
}

template <class T>
struct State {  // a conserved state with what its faces need
  T u[4];            // rho, j1, j2, e
  T p, ir, vx, vz;   // pressure, 1 / rho, velocity
};

template <class T>
__device__ __forceinline__ State<T> make_state(const T& rho, const T& j1, const T& j2, const T& e) {
  State<T> s;
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
template <class T>
__device__ __forceinline__ void grad_p(const State<T>& s, T (&g)[4]) {
  g[0] = (kGm1 * 0.5) * mad(s.vx, s.vx, s.vz * s.vz);
  g[1] = (-kGm1) * s.vx;
  g[2] = (-kGm1) * s.vz;
  g[3] = lift<T>(kGm1);
}

template <class T>
struct Wall {  // a wall face: normal, grid velocity, n.g and 1 / |n|^2
  T nx, nz, gx, gz, gn, inn;
};
template <class T>
__device__ __forceinline__ Wall<T> make_wall(const T& nx, const T& nz, const T& gx, const T& gz) {
  return Wall<T>{nx, nz, gx, gz, nx * gx + nz * gz, recip_(nx * nx + nz * nz)};
}
// make_wall_ghost_state, f90:231-240.
template <class T>
__device__ __forceinline__ State<T> wall_ghost_of(const State<T>& s, const Wall<T>& w) {
  const T proj = w.nx * (s.u[1] - w.gx * s.u[0]) + w.nz * (s.u[2] - w.gz * s.u[0]);
  const T nn = w.nx * w.nx + w.nz * w.nz;
  return make_state<T>(s.u[0], s.u[1] - quot_(2.0 * w.nx * proj, nn),
                       s.u[2] - quot_(2.0 * w.nz * proj, nn), s.u[3]);
}
// make_farfield_ghost_state, f90:269-274: 2 U_inf - U.
template <class T>
__device__ __forceinline__ State<T> farfield_ghost_of(const State<T>& s, const Instance& in) {
  const double speed = in.mach * sqrt_(kGamma);
  const double f1 = speed * in.cos_aoa, f2 = speed * in.sin_aoa;
  const double fe = 1.0 / kGm1 + speed * speed / 2.0;
  return make_state<T>(2.0 - s.u[0], 2.0 * f1 - s.u[1], 2.0 * f2 - s.u[2], 2.0 * fe - s.u[3]);
}

template <class T>
struct FaceGeometry {  // normal, grid velocity
  T nx, nz, gx, gz;
};

// The derivative of a face flux by one of its states, factored (see above).
template <class T>
struct Block {
  T alpha[4], beta[4], extra[4], diag;
};

// A face's flux in its cell's orientation, differentiated. diss = false: the central flux of the
// faces next to the boundaries (f90:197, 219). r may be a ghost state there, whose pressure and
// density can be negative (2 U_inf - U of a cell at twice the free stream's; the reflection at a fast
// wall): it has no speed of sound, and what the dissipation is formed from is replaced by zeros. ll
// and rr need then only be finite.
template <class T>
struct FaceDerivatives {
  T nx, nz, vn, vl, vr;
  T Q[4], h[4];                 // dF/dS, dF/dlambda (zero without dissipation)
  T g_ll, g_l, g_r, g_rr;       // dS/dp of the four states
  T c2, c4;
  bool diss;
  bool lam_l;                   // lambda is l's (else r's)
  double sgn;                   // the sign of that state's normal velocity
  T c, len, ilen;               // its speed of sound; |n| and its inverse

  __device__ __forceinline__ FaceDerivatives(const State<T>& ll, const State<T>& l,
                                             const State<T>& r, const State<T>& rr,
                                             const FaceGeometry<T>& f, bool diss_,
                                             const Instance& in)
      : diss(diss_) {
    nx = f.nx;
    nz = f.nz;
    vn = f.gx * nx + f.gz * nz;
    vl = (nx * l.u[1] + nz * l.u[2]) * l.ir;
    vr = (nx * r.u[1] + nz * r.u[2]) * r.ir;
    const T zero = lift<T>(0.0);
    len = sqrt_(nx * nx + nz * nz);
    ilen = diss ? recip_(len) : zero;
    const T cl = sqrt_(kGamma * l.p * l.ir), cr = sqrt_(kGamma * r.p * r.ir);
    const T al = abs_c(vl) + cl * len, ar = abs_c(vr) + cr * len;
    lam_l = value(al) > value(ar) + 1e-8;
    const T lam = !diss ? zero : lam_l ? al : ar;
    c = !diss ? zero : lam_l ? cl : cr;
    sgn = value(lam_l ? vl : vr) < 0.0 ? -1.0 : 1.0;
    const T num_l = ll.p - 2.0 * l.p + r.p, den_l = ll.p + 2.0 * l.p + r.p;
    const T num_r = l.p - 2.0 * r.p + rr.p, den_r = l.p + 2.0 * r.p + rr.p;
    const T sl = quot_(abs_c(num_l), den_l), sr = quot_(abs_c(num_r), den_r);
    const bool s_l = value(sl) > value(sr) + 1e-8;
    const T S = !diss ? zero : s_l ? sl : sr;
    const double sg = value(s_l ? num_l : num_r) < 0.0 ? -1.0 : 1.0;
    const T inv = recip_(!diss ? lift<T>(1.0) : s_l ? den_l : den_r);
    const T outer = (sg - S) * inv, centre = -2.0 * (sg + S) * inv;
    g_ll = s_l ? outer : zero;
    g_l = s_l ? centre : outer;
    g_r = s_l ? outer : centre;
    g_rr = s_l ? zero : outer;
    c2 = in.k2 * S * lam;
    c4 = in.k4 * lam - in.c4 * c2;
    const bool active = !(0.0 > value(c4) + 1e-8);  // max_c(0, c4)
    const double on4 = diss && active ? 1.0 : 0.0;
    c4 = c4 * on4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T d1 = r.u[k] - l.u[k];
      const T d3 = mad(3.0, l.u[k] - r.u[k], rr.u[k] - ll.u[k]);
      const T by_c2 = -mad(on4 * in.c4, d3, d1);  // dF/dc2 (through c4 as well)
      Q[k] = by_c2 * (in.k2 * lam);
      h[k] = mad(by_c2, in.k2 * S, on4 * in.k4 * d3);
    }
  }

  // dF/dl (Left) or dF/dr.
  template <bool Left>
  __device__ __forceinline__ Block<T> of(const State<T>& s) const {
    Block<T> b;
    const T v = Left ? vl : vr, g = Left ? g_l : g_r;
    const bool lam = diss && Left == lam_l;
    // dlambda = sgn dv + len dc, dc = c / (2 p) dp - c / (2 rho) e_0
    const T zero = lift<T>(0.0);
    const T lp = lam ? quot_(0.5 * len * c, s.p) : zero, le = lam ? -0.5 * len * c * s.ir : zero;
    const double lv = lam ? sgn : 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T n = k == 1 ? 0.5 * nx : k == 2 ? 0.5 * nz : k == 3 ? 0.5 * v : zero;
      b.alpha[k] = mad(h[k], lp, mad(Q[k], g, n));
      b.beta[k] = mad(h[k], lv, 0.5 * (k == 3 ? s.u[3] + s.p : s.u[k]));
      b.extra[k] = h[k] * le;
    }
    b.diag = mad(0.5, v - vn, Left ? mad(3.0, c4, c2) : -mad(3.0, c4, c2));
    return b;
  }

  // Flux component k (the central flux, the grid velocity's part and the dissipation).
  __device__ __forceinline__ T flux(const State<T>& ll, const State<T>& l, const State<T>& r,
                                    const State<T>& rr, int k) const {
    const T n = k == 1 ? nx : k == 2 ? nz : lift<T>(0.0);
    T f = 0.5 * (mad(l.u[k], vl - vn, r.u[k] * (vr - vn)) + n * (l.p + r.p));
    if (k == 3) f = f + 0.5 * mad(l.p, vl, r.p * vr);
    const T d1 = r.u[k] - l.u[k];
    const T d3 = mad(3.0, l.u[k] - r.u[k], rr.u[k] - ll.u[k]);
    return mad(c4, d3, mad(-c2, d1, f));
  }

  // Derivative of flux component k by the normal (nx if X, else nz) at fixed states.
  template <bool X>
  __device__ __forceinline__ T by_normal(const State<T>& l, const State<T>& r,
                                         const FaceGeometry<T>& f, int k) const {
    const T ul = X ? l.vx : l.vz, ur = X ? r.vx : r.vz, g = X ? f.gx : f.gz;
    T d = 0.5 * mad(l.u[k], ul - g, r.u[k] * (ur - g));
    if (k == (X ? 1 : 2)) d = d + 0.5 * (l.p + r.p);
    if (k == 3) d = d + 0.5 * mad(l.p, ul, r.p * ur);
    const T lam = mad(sgn, lam_l ? ul : ur, c * (X ? nx : nz) * ilen);
    return mad(h[k], lam, d);
  }
};

// block += E, a full 4 x 4 (column-major: entry k + 4 j is dF_k/du_j) of one of the line's states.
template <class T>
__device__ __forceinline__ void add_block(T (&acc)[16], const Block<T>& b, const State<T>& s,
                                          const T& nx, const T& nz, const T& v) {
  T dp[4];
  grad_p(s, dp);
  const T dv[3] = {-v * s.ir, nx * s.ir, nz * s.ir};
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      T e = mad(b.alpha[k], dp[j], acc[k + 4 * j]);
      if (j < 3) e = mad(b.beta[k], dv[j], e);
      if (j == 0) e = e + b.extra[k];
      if (j == k) e = e + b.diag;
      acc[k + 4 * j] = e;
    }
}
// The blocks of the line's outer states, Q g (x) dp + diag I.
template <class T>
__device__ __forceinline__ void add_outer(T (&acc)[16], const T (&Q)[4], const T& g, const T& diag,
                                          const State<T>& s) {
  T dp[4];
  grad_p(s, dp);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T a = Q[k] * g;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[k + 4 * j] = mad(a, dp[j], acc[k + 4 * j]);
      if (j == k) acc[k + 4 * j] = acc[k + 4 * j] + diag;
    }
  }
}

// acc += E G with G the derivative of the wall ghost by its state.
template <class T>
__device__ __forceinline__ void through_wall(T (&acc)[16], const T (&E)[16], const Wall<T>& w) {
  const T ax = 2.0 * w.nx * w.inn, az = 2.0 * w.nz * w.inn;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T e1 = E[k + 4], e2 = E[k + 8];
    const T t = mad(e1, ax, e2 * az);  // along the reflected normal
    acc[k] = acc[k] + mad(t, w.gn, E[k]);
    acc[k + 4] = acc[k + 4] + mad(-t, w.nx, e1);
    acc[k + 8] = acc[k + 8] + mad(-t, w.nz, e2);
    acc[k + 12] = acc[k + 12] + E[k + 12];
  }
}

// ---- cells and warps -------------------------------------------------------------------------

// A warp's outputs of D doubles per cell, in rows padded by 16 bytes, so that the threads' 16-byte
// accesses to their own rows fall on distinct banks.
template <int D>
struct WarpRows {
  double2 v[32][D / 2 + 1];
};

// Thread `lane` hands over `mine`; the warp writes the rows of its first `valid` cells to `out`
// (the first cell's place).
template <int D>
__device__ __forceinline__ void write_rows(WarpRows<D>& S, const double (&mine)[D], int lane,
                                           int valid, double* out) {
#pragma unroll
  for (int e = 0; e < D / 2; ++e) S.v[lane][e] = make_double2(mine[2 * e], mine[2 * e + 1]);
  __syncwarp();
  constexpr int kPer = D / 2;
  double2* o = reinterpret_cast<double2*>(out);
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int f = 32 * e + lane;
    if (f < valid * kPer) o[f] = S.v[f / kPer][f % kPer];
  }
  __syncwarp();
}

// Calls body(warp's first cell, thread's cell, lane, valid cells of the warp) for the cells of this
// thread's instance.
// Whole warps stay in the loop together; the body's cell is clamped to the instance.
template <class Body>
__device__ __forceinline__ void for_cells(const Instance& in, Body body) {
  const int64_t cells = (int64_t)in.M * in.N;
  const int lane = threadIdx.x & 31;
  for (int64_t first = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); first < cells;
       first += (int64_t)gridDim.x * blockDim.x) {
    const int valid = (int)min((int64_t)32, cells - first);
    body(first, min(first + lane, cells - 1), lane, valid);
  }
}

// ---- one cell's inputs ------------------------------------------------------------------------

// A cell's place and its inputs as scalars of type T. Kind: the variable whose components carry the
// direction D (interleaved complex: its real and imaginary part are a dual's two components), or
// kDirNone for plain doubles.
template <class T, int Kind>
struct CellAt {
  int m, n;
  int64_t M, N;
  const double *U, *X, *V, *D;  // the instance's arrays (V may be null)

  __device__ __forceinline__ CellAt(const Instance& in, int64_t local, const double* X_,
                                    const double* V_, const double* U_, const double* D_)
      : m((int)(local % in.M)), n((int)(local / in.M)), M(in.M), N(in.N),
        U(U_ + 4 * in.cell_offset), X(X_ + 2 * in.vert_offset),
        V(V_ ? V_ + 2 * in.vert_offset : nullptr),
        D(Kind == kDirNone ? nullptr
                           : D_ + (Kind == kDirStates ? 8 * in.cell_offset : 4 * in.vert_offset)) {}

  template <bool Along>
  __device__ __forceinline__ static T scalar(double v, const double* d) {
    if constexpr (std::is_same<T, double>::value) {
      return v;
    } else {
      T r = lift<T>(v);
      if (Along) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(d));
        r.d[0] = t.x;
        r.d[1] = t.y;
      }
      return r;
    }
  }
  __device__ __forceinline__ State<T> state(int dm, int dn) const {
    int c = n + dn;
    c = c < 0 ? c + (int)N : c >= (int)N ? c - (int)N : c;
    const int64_t at = m + dm + M * c;
    const double2* q = reinterpret_cast<const double2*>(U + 4 * at);
    const double2 a = __ldg(q), b = __ldg(q + 1);
    const double* d = D + 8 * at;
    constexpr bool kAlong = Kind == kDirStates;
    return make_state<T>(scalar<kAlong>(a.x, d), scalar<kAlong>(a.y, d + 2),
                         scalar<kAlong>(b.x, d + 4), scalar<kAlong>(b.y, d + 6));
  }
  // The corners in the order backward-inward, forward-inward, forward-outward, backward-outward:
  // coordinates (Velo = false) or velocities.
  template <bool Velo>
  __device__ __forceinline__ P2<T> corner(int k) const {
    const int64_t v = m + (k >= 2) + (M + 1) * (n + (k == 1 || k == 2));
    const double* A = Velo ? V : X;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 a = A ? __ldg(reinterpret_cast<const double2*>(A + 2 * v)) : zero;
    const double* d = D + 4 * v;
    constexpr bool kAlong = Kind == (Velo ? kDirVelocities : kDirVertices);
    return P2<T>{scalar<kAlong>(a.x, d), scalar<kAlong>(a.y, d + 2)};
  }
};

template <class T>
struct CellGeometry {
  P2<T> x[4];
  FaceGeometry<T> b, f, i, o;  // faces between corners 3-0, 1-2, 0-1 and 2-3 (outward normals)
  T cross;                     // signed area times 2

  template <int Kind>
  __device__ __forceinline__ explicit CellGeometry(const CellAt<T, Kind>& at) {
    P2<T> w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = at.template corner<false>(k);
      w[k] = at.template corner<true>(k);
    }
    auto edge = [&](int p, int q) {
      return FaceGeometry<T>{x[q].z - x[p].z, x[p].x - x[q].x, (w[p].x + w[q].x) * 0.5,
                             (w[p].z + w[q].z) * 0.5};
    };
    i = edge(0, 1);
    f = edge(1, 2);
    o = edge(2, 3);
    b = edge(3, 0);
    cross = (x[2].x - x[0].x) * (x[3].z - x[1].z) - (x[2].z - x[0].z) * (x[3].x - x[1].x);
  }
  __device__ __forceinline__ T inv_area() const { return recip_(abs_c(cross) * 0.5); }
  __device__ __forceinline__ Wall<T> wall() const { return make_wall(i.nx, i.nz, i.gx, i.gz); }
};

// The radial line of a cell, boundary rows included (make_ode's five cases, f90:401-436): the
// inner face has the line (o, c, i, ii), the outer one (i, c, o, oo), with ghost states past the
// ends and the dissipation off on the faces whose line would reach past a ghost.
template <class T>
struct RadialLine {
  State<T> i, o, ii, oo;
  bool diss_i, diss_o;
  template <int Kind>
  __device__ __forceinline__ RadialLine(const CellAt<T, Kind>& at, const State<T>& c,
                                        const CellGeometry<T>& g, const Instance& in) {
    const int m = at.m, M = (int)at.M;
    diss_i = m >= 2;
    diss_o = m <= M - 3;
    i = m > 0 ? at.state(-1, 0) : wall_ghost_of(c, g.wall());
    o = m < M - 1 ? at.state(1, 0) : farfield_ghost_of(c, in);
    ii = diss_i ? at.state(-2, 0) : c;
    oo = diss_o ? at.state(2, 0) : c;
  }
};

template <class T>
__device__ __forceinline__ void clear(T (&a)[16]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) a[e] = lift<T>(0.0);
}

// The derivative of the wall ghost's momentum by the wall's normal (x then z), contracted with
// dF_k by the momentum (e1, e2).
template <class T>
__device__ __forceinline__ P2<T> ghost_by_normal(const Wall<T>& w, const State<T>& c, const T& e1,
                                                 const T& e2) {
  const T mx = c.u[1] - w.gx * c.u[0], mz = c.u[2] - w.gz * c.u[0];
  const T t = w.nx * mx + w.nz * mz, en = mad(e1, w.nx, e2 * w.nz);
  const T q = 2.0 * w.inn, r = q * en;
  return P2<T>{mad(r, 2.0 * t * w.nx * w.inn - mx, -q * t * e1),
               mad(r, 2.0 * t * w.nz * w.inn - mz, -q * t * e2)};
}

// The far-field ghost's derivative by the Mach number.
__device__ __forceinline__ void ghost_by_mach(const Instance& in, double (&d)[4]) {
  const double root = ::sqrt(kGamma), speed = in.mach * root;
  d[0] = 0.0;
  d[1] = 2.0 * root * in.cos_aoa;
  d[2] = 2.0 * root * in.sin_aoa;
  d[3] = 2.0 * speed * root;
}

// ---- faces by number ----------------------------------------------------------------------------

// A cell's face q (0 b, 1 f, 2 i, 3 o) with its line ll, l = c, r, rr, loaded by offsets: one piece
// of code for the four faces, ghosts included, for the kernels that loop over them.
template <class T, int Kind>
struct NumberedFace {
  int dm, dn;         // r's offset; ll is at the opposite one, rr at twice it
  bool r_ghost, ll_ghost, diss;
  FaceGeometry<T> f;
  State<T> ll, r, rr;

  __device__ __forceinline__ NumberedFace(const CellAt<T, Kind>& at, const State<T>& c, int q,
                                          const Instance& in)
      : dm(q < 2 ? 0 : q == 2 ? -1 : 1), dn(q > 1 ? 0 : q == 0 ? -1 : 1) {
    const int M = (int)at.M;
    r_ghost = at.m + dm < 0 || at.m + dm >= M;
    ll_ghost = at.m - dm < 0 || at.m - dm >= M;
    diss = at.m + 2 * dm >= 0 && at.m + 2 * dm < M;
    f = edge(at, q);
    r = r_ghost ? ghost(at, c, in) : at.state(dm, dn);
    ll = ll_ghost ? ghost(at, c, in) : at.state(-dm, -dn);
    rr = diss ? at.state(2 * dm, 2 * dn) : c;
  }
  __device__ __forceinline__ static FaceGeometry<T> edge(const CellAt<T, Kind>& at, int q) {
    const int k = q == 0 ? 3 : q == 1 ? 1 : q == 2 ? 0 : 2, l = (k + 1) & 3;
    const P2<T> a = at.template corner<false>(k), b = at.template corner<false>(l);
    const P2<T> v = at.template corner<true>(k), w = at.template corner<true>(l);
    return FaceGeometry<T>{b.z - a.z, a.x - b.x, (v.x + w.x) * 0.5, (v.z + w.z) * 0.5};
  }
  __device__ __forceinline__ static Wall<T> wall(const CellAt<T, Kind>& at) {
    const FaceGeometry<T> i = edge(at, 2);
    return make_wall<T>(i.nx, i.nz, i.gx, i.gz);
  }
  __device__ __forceinline__ static State<T> ghost(const CellAt<T, Kind>& at, const State<T>& c,
                                                   const Instance& in) {
    return at.m == 0 ? wall_ghost_of<T>(c, wall(at)) : farfield_ghost_of<T>(c, in);
  }
};

// The signed area times 2.
template <class T, int Kind>
__device__ __forceinline__ T cross_of(const CellAt<T, Kind>& at) {
  const P2<T> a = at.template corner<false>(0), b = at.template corner<false>(1);
  const P2<T> c = at.template corner<false>(2), d = at.template corner<false>(3);
  return (c.x - a.x) * (d.z - b.z) - (c.z - a.z) * (d.x - b.x);
}

}  // namespace eb
