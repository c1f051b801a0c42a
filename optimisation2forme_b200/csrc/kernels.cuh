// CUDA kernels of the residual, time step, forces, adjoint operator and shape
// perturbation, templated on the arithmetic type T (double / float).
//
// Every floating-point expression keeps the association order of the
// reference expression it restates (cited per kernel).  The FP64
// instantiation is compiled with -fmad=false, so no multiply-add is fused and
// each operation rounds exactly as the reference's does on x86-64; sqrt and
// division are IEEE round-to-nearest on both sides (quotients that share a
// divisor come from one reciprocal through qdiv, which returns the same bits
// as the division; qdiv.h).  Summations follow the
// reference's Cell::edgeIDs / Vertex::cellIDs order, which the host build
// reproduces (mesh_host.cpp).  The FP64 residual is therefore bit-identical to
// the reference for the same mesh and state.
#pragma once

#include <cfloat>
#include <cstdint>

#include "device_types.hpp"
#include "qdiv.h"

namespace o2f {

constexpr int kBlock = 256;
constexpr int kGradBlock = 128;
constexpr double kDblEps = 2.220446049250313080847263336181640625e-16;  // DBL_EPSILON

// Gate: when `gate` is non-null and *gate != 0 the kernel does nothing.  Used
// by the device-driven loops (time stepping, BiCGSTAB) to turn the launches
// that follow a stop condition into no-ops.
__device__ __forceinline__ bool gated(const int* gate) { return gate != nullptr && *(volatile const int*)gate != 0; }

// std::min / std::max / std::clamp semantics (NaN propagation included).
template <typename T>
__device__ __forceinline__ T smin(T a, T b) { return (b < a) ? b : a; }
template <typename T>
__device__ __forceinline__ T smax(T a, T b) { return (a < b) ? b : a; }
template <typename T>
__device__ __forceinline__ T sclamp(T v, T lo, T hi) { return (v < lo) ? lo : (hi < v) ? hi : v; }

template <typename T>
__device__ __forceinline__ Vec4<T> v4(T a, T b, T c, T d) {
  Vec4<T> r;
  r.a = a;
  r.b = b;
  r.c = c;
  r.d = d;
  return r;
}

// apply_inflow_outflow_bc (src/boundary.cpp:7-45): inlet / far field take the
// freestream, outlet keeps the state, a wall keeps rho and the internal energy
// with zero momentum.
template <typename T>
__device__ __forceinline__ void bc_state(uint8_t code, const Phys& ph, T& r, T& ru, T& rv, T& E) {
  if (code == 'i' || code == 'f') {
    r = (T)ph.fs_rho;
    ru = (T)ph.fs_rhou;
    rv = (T)ph.fs_rhov;
    E = (T)ph.fs_E;
  } else if (code == 'w') {
    const T kinetic_old = (T)0.5 * (ru * ru + rv * rv) / r;
    const T e_internal = E - kinetic_old;
    ru = (T)0.0;
    rv = (T)0.0;
    E = e_internal;
  }
}

// apply_InterfaceStates_boundary_conditions (src/boundary.cpp:48-80): the
// ghost right state of a boundary edge built from its left state.
template <typename T>
__device__ __forceinline__ Vec4<T> bc_ghost(uint8_t code, const Phys& ph, const Vec4<T>& L) {
  Vec4<T> R = L;
  if (code == 'i' || code == 'o' || code == 'f') {
    bc_state(code, ph, R.a, R.b, R.c, R.d);
  } else if (code == 'w') {
    R.b = -L.b;
    R.c = -L.c;
  }
  return R;
}

// pressure / sound_speed (src/advection.cpp:325-332).
template <typename T>
__device__ __forceinline__ T pressure(T rho, T u, T v, T E, T gamma) {
  const T kinetic = (T)0.5 * rho * (u * u + v * v);
  return (gamma - (T)1.0) * (E - kinetic);
}

// compute_hllc_flux (src/advection.cpp:335-412): rotated HLLC with the normal
// -edgeNormal, Davis wave speeds, flux rotated back.
template <typename T>
__device__ __forceinline__ Vec4<T> hllc(const Vec4<T>& Ls, const Vec4<T>& Rs, T enx, T eny, T gamma) {
  const T nx = -enx, ny = -eny;
  const T rho_L = Ls.a;
  const T u_L = (Ls.b * (nx) + Ls.c * ny) / rho_L;
  const T v_L = (Ls.b * (-ny) + Ls.c * nx) / rho_L;
  const T E_L = Ls.d;
  const T p_L = pressure(rho_L, u_L, v_L, E_L, gamma);
  const T c_L = sqrt(gamma * p_L / rho_L);
  const T rho_R = Rs.a;
  const T u_R = (Rs.b * (nx) + Rs.c * ny) / rho_R;
  const T v_R = (Rs.b * (-ny) + Rs.c * nx) / rho_R;
  const T E_R = Rs.d;
  const T p_R = pressure(rho_R, u_R, v_R, E_R, gamma);
  const T c_R = sqrt(gamma * p_R / rho_R);

  const T S_L = smin(u_L - c_L, u_R - c_R);
  const T S_R = smax(u_L + c_L, u_R + c_R);
  const T numer = p_R - p_L + rho_L * u_L * (S_L - u_L) - rho_R * u_R * (S_R - u_R);
  const T denom = rho_L * (S_L - u_L) - rho_R * (S_R - u_R);
  const T S_star = numer / denom;
  const T rho_L_star = rho_L * (S_L - u_L) / (S_L - S_star);
  const T rho_R_star = rho_R * (S_R - u_R) / (S_R - S_star);
  const T rho_v_L_star = rho_L_star * v_L;
  const T rho_v_R_star = rho_R_star * v_R;
  const T p_star = p_L + rho_L * (S_L - u_L) * (S_star - u_L);
  const T E_L_star = ((S_L - u_L) * E_L - p_L * u_L + p_star * S_star) / (S_L - S_star);
  const T E_R_star = ((S_R - u_R) * E_R - p_R * u_R + p_star * S_star) / (S_R - S_star);
  const T rho_u_L_star = rho_L_star * S_star;
  const T rho_u_R_star = rho_R_star * S_star;

  T f_rho, f_u, f_v, f_E;
  if (S_L >= (T)0.0) {
    f_rho = rho_L * u_L;
    f_u = rho_L * u_L * u_L + p_L;
    f_v = rho_L * u_L * v_L;
    f_E = (E_L + p_L) * u_L;
  } else if (S_L <= (T)0.0 && S_star >= (T)0.0) {
    f_rho = rho_u_L_star;
    f_u = rho_u_L_star * rho_u_L_star / rho_L_star + p_star;
    f_v = rho_v_L_star * rho_u_L_star / rho_L_star;
    f_E = (E_L_star + p_star) * rho_u_L_star / rho_L_star;
  } else if (S_star <= (T)0.0 && S_R >= (T)0.0) {
    f_rho = rho_u_R_star;
    f_u = rho_u_R_star * rho_u_R_star / rho_R_star + p_star;
    f_v = rho_v_R_star * rho_u_R_star / rho_R_star;
    f_E = (E_R_star + p_star) * rho_u_R_star / rho_R_star;
  } else {
    f_rho = rho_R * u_R;
    f_u = rho_R * u_R * u_R + p_R;
    f_v = rho_R * u_R * v_R;
    f_E = (E_R + p_R) * u_R;
  }
  return v4<T>(f_rho, (f_u * nx + f_v * (-ny)), (f_u * ny + f_v * (nx)), f_E);
}

// The same flux in FP64 without branches, and with the star state of the one
// side that the flux needs.  Quotients and square roots as in qdiv.h, each
// with the bits of hllc's; false when one left its range (f is then not set
// to the flux).  hllc's divisions and square roots each end in a branch to a
// slow path, so their 35-cycle operations run one chain after the other;
// here they overlap (k_edge_flux 111 -> 96 us at 3.0M edges, k_jt_blocks 1,094
// -> 903; 33 -> 18.5 us at 30,804).
__device__ __forceinline__ bool hllc_flat(const Vec4<double>& Ls, const Vec4<double>& Rs, double enx, double eny,
                                          double gamma, Vec4<double>& f) {
  const double nx = -enx, ny = -eny;
  bool ok = true;
  const double rho_L = Ls.a, rho_R = Rs.a, E_L = Ls.d, E_R = Rs.d;
  const double y_L = recip_fast(rho_L, ok), y_R = recip_fast(rho_R, ok);
  const double u_L = quot(Ls.b * (nx) + Ls.c * ny, rho_L, y_L, ok);
  const double v_L = quot(Ls.b * (-ny) + Ls.c * nx, rho_L, y_L, ok);
  const double u_R = quot(Rs.b * (nx) + Rs.c * ny, rho_R, y_R, ok);
  const double v_R = quot(Rs.b * (-ny) + Rs.c * nx, rho_R, y_R, ok);
  const double p_L = pressure(rho_L, u_L, v_L, E_L, gamma);
  const double p_R = pressure(rho_R, u_R, v_R, E_R, gamma);
  const double c_L = sqrt_fast(quot(gamma * p_L, rho_L, y_L, ok), ok);
  const double c_R = sqrt_fast(quot(gamma * p_R, rho_R, y_R, ok), ok);
  const double S_L = smin(u_L - c_L, u_R - c_R);
  const double S_R = smax(u_L + c_L, u_R + c_R);
  const double numer = p_R - p_L + rho_L * u_L * (S_L - u_L) - rho_R * u_R * (S_R - u_R);
  const double denom = rho_L * (S_L - u_L) - rho_R * (S_R - u_R);
  const double S_star = quot(numer, denom, recip_fast(denom, ok), ok);
  const double p_star = p_L + rho_L * (S_L - u_L) * (S_star - u_L);
  // numbers from here on (ok): the four cases of hllc
  const bool left = S_L >= 0.0 || S_star >= 0.0;
  const bool plain = S_L >= 0.0 || (!left && !(S_R >= 0.0));
  const double rho = left ? rho_L : rho_R, u = left ? u_L : u_R, v = left ? v_L : v_R, E = left ? E_L : E_R,
               p = left ? p_L : p_R, S = left ? S_L : S_R;
  bool star = true;
  const double gap = S - S_star;
  const double y_gap = recip_fast(gap, star);
  const double rho_star = quot(rho * (S - u), gap, y_gap, star);
  const double rho_v_star = rho_star * v;
  const double E_star = quot((S - u) * E - p * u + p_star * S_star, gap, y_gap, star);
  const double rho_u_star = rho_star * S_star;
  const double y_star = recip_fast(rho_star, star);
  double f_rho = rho_u_star;
  double f_u = quot(rho_u_star * rho_u_star, rho_star, y_star, star) + p_star;
  double f_v = quot(rho_v_star * rho_u_star, rho_star, y_star, star);
  double f_E = quot((E_star + p_star) * rho_u_star, rho_star, y_star, star);
  if (plain) {
    f_rho = rho * u;
    f_u = rho * u * u + p;
    f_v = rho * u * v;
    f_E = (E + p) * u;
  }
  f = v4<double>(f_rho, (f_u * nx + f_v * (-ny)), (f_u * ny + f_v * (nx)), f_E);
  return ok && (star || plain);
}

static __device__ __noinline__ Vec4<double> hllc_out_of_range(const Vec4<double> Ls, const Vec4<double> Rs, double enx,
                                                       double eny, double gamma) {
  return hllc(Ls, Rs, enx, eny, gamma);
}
__device__ __forceinline__ Vec4<double> hllc_flux(const Vec4<double>& Ls, const Vec4<double>& Rs, double enx, double eny,
                                                  double gamma) {
  Vec4<double> f;
  if (!hllc_flat(Ls, Rs, enx, eny, gamma, f)) f = hllc_out_of_range(Ls, Rs, enx, eny, gamma);
  return f;
}
__device__ __forceinline__ Vec4<float> hllc_flux(const Vec4<float>& Ls, const Vec4<float>& Rs, float enx, float eny,
                                                 float gamma) {
  return hllc(Ls, Rs, enx, eny, gamma);
}

// computeVenkatAlpha (src/advection.cpp:209-230) with eps = (k h)^3
// precomputed per cell; computeBarthJespersenAlpha (:195-207).
template <typename T>
__device__ __forceinline__ T limiter_alpha(int kind, T phi_i, T phi_pred, T phi_min, T phi_max, T eps) {
  if (kind == 0) {
    const T delta = phi_pred - phi_i;
    if (fabs(delta) < (T)kDblEps) return (T)1.0;
    T a = (delta > (T)0.0) ? (phi_max - phi_i) : (phi_min - phi_i);
    const T d = delta;
    T alpha = (a * a + eps + (T)2.0 * a * d) / (a * a + eps + (T)2.0 * d * d);
    return sclamp(alpha, (T)0.0, (T)1.0);
  }
  T alpha = (T)1.0;
  if (fabs(phi_pred - phi_i) < (T)kDblEps) return alpha;
  if (phi_pred > phi_i) {
    alpha = smin((T)1.0, (phi_max - phi_i) / (phi_pred - phi_i));
  } else if (phi_pred < phi_i) {
    alpha = smin((T)1.0, (phi_min - phi_i) / (phi_pred - phi_i));
  }
  return alpha;
}

// limiter_alpha (kind and semantics) without branches: the FP64 gradient
// keeps a cell's twelve limiter quotients in flight together.  A dependent
// FP64 operation takes some 35 cycles, so twelve quotients one after the other,
// as the early returns and the division's slow-path branch force, are most
// of the kernel's time (k_cell_gradient with / without branches: 22.6 / 8.3
// us at 20,400 triangles, 234 / 217 at 2.0M).  `ok` is cleared where a quotient left quot's range.
__device__ __forceinline__ double limiter_alpha_flat(int kind, double phi_i, double phi_pred, double phi_min,
                                                     double phi_max, double eps, bool& ok) {
  const double delta = phi_pred - phi_i;
  const bool tiny = fabs(delta) < kDblEps;
  const double a = (delta > 0.0 ? phi_max : phi_min) - phi_i;
  double num, den;
  if (kind == 0) {  // uniform
    const double s = a * a + eps;
    num = s + 2.0 * a * delta;
    den = s + 2.0 * delta * delta;
  } else {
    num = a;
    den = tiny ? 1.0 : delta;
  }
  bool in = true;
  const double y = recip_fast(den, in);
  double alpha = quot(num, den, y, in);
  ok &= in | tiny;
  alpha = kind == 0 ? sclamp(alpha, 0.0, 1.0) : smin(1.0, alpha);
  return tiny ? 1.0 : alpha;
}

// ---------------------------------------------------------------------------
// K1: cell -> vertex interpolation of the state (src/advection.cpp:26-131),
// weights precomputed in the reference's order, then the vertex boundary
// override (:129-130).  The generic weighted sum reproduces every valence case
// of the reference exactly: w=1 copies, w=0.5 halves, and the 3- and 4-cell
// sums keep the reference's left-to-right association.
// acc + w u as the vertex sums take it: FP64 rounds twice, as the reference
// does, FP32 once (said here, not left to contraction, which may pick either
// product of a sum of two).
__device__ __forceinline__ double vertex_add(double acc, double w, double u) { return acc + w * u; }
__device__ __forceinline__ float vertex_add(float acc, float w, float u) { return __fmaf_rn(w, u, acc); }

// bc_state of a vertex; in FP32 with the contraction of ru^2 + rv^2 said.
__device__ __forceinline__ void vertex_bc(uint8_t code, const Phys& ph, double& r, double& ru, double& rv, double& E) {
  bc_state(code, ph, r, ru, rv, E);
}
__device__ __forceinline__ void vertex_bc(uint8_t code, const Phys& ph, float& r, float& ru, float& rv, float& E) {
  if (code == 'w') {
    E = E - 0.5f * __fmaf_rn(ru, ru, rv * rv) / r;
    ru = rv = 0.f;
  } else {
    bc_state(code, ph, r, ru, rv, E);
  }
}

// A vertex's cells and weights.  The first kFan of them are in registers, so
// that their gathers are in flight together; a vertex with more goes on in
// order.
constexpr int kFan = 8;
template <typename T>
struct VertexFan {
  int o, n;
  int cid[kFan];
  T w[kFan];
  uint8_t code;
};
template <typename T>
__device__ __forceinline__ VertexFan<T> vertex_fan(int64_t v, const int32_t* __restrict__ voff,
                                                   const int32_t* __restrict__ vcid, const T* __restrict__ vw,
                                                   const uint8_t* __restrict__ vbc) {
  VertexFan<T> f;
  f.o = voff[v];
  f.n = voff[v + 1] - f.o;
  f.code = vbc[v];
#pragma unroll
  for (int k = 0; k < kFan; ++k)
    if (k < f.n) {
      f.cid[k] = vcid[f.o + k];
      f.w[k] = vw[f.o + k];
    }
  return f;
}

template <typename T>
__device__ __forceinline__ Vec4<T> vertex_state_of(const VertexFan<T>& f, const int32_t* __restrict__ vcid,
                                                   const T* __restrict__ vw, const Vec4<T>* U,
                                                   const Phys& ph) {
  T a = (T)0.0, b = (T)0.0, c = (T)0.0, d = (T)0.0;
#pragma unroll
  for (int h = 0; h < kFan; h += 4) {
    if (h >= f.n) break;
    Vec4<T> u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (h + k < f.n) u[k] = U[f.cid[h + k]];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (h + k >= f.n) continue;
      const T w = f.w[h + k];
      if (h + k == 0) {
        a = w * u[k].a;
        b = w * u[k].b;
        c = w * u[k].c;
        d = w * u[k].d;
      } else {
        a = vertex_add(a, w, u[k].a);
        b = vertex_add(b, w, u[k].b);
        c = vertex_add(c, w, u[k].c);
        d = vertex_add(d, w, u[k].d);
      }
    }
  }
  for (int k = f.o + kFan; k < f.o + f.n; ++k) {
    const T w = vw[k];
    const Vec4<T> q = U[vcid[k]];
    a = vertex_add(a, w, q.a);
    b = vertex_add(b, w, q.b);
    c = vertex_add(c, w, q.c);
    d = vertex_add(d, w, q.d);
  }
  if (f.code) vertex_bc(f.code, ph, a, b, c, d);
  return v4<T>(a, b, c, d);
}

template <typename T>
__device__ __forceinline__ Vec4<T> vertex_state_value(int64_t v, const int32_t* __restrict__ voff,
                                                      const int32_t* __restrict__ vcid, const T* __restrict__ vw,
                                                      const uint8_t* __restrict__ vbc,
                                                      const Vec4<T>* __restrict__ U, const Phys& ph) {
  return vertex_state_of<T>(vertex_fan<T>(v, voff, vcid, vw, vbc), vcid, vw, U, ph);
}

template <typename T>
__device__ __forceinline__ void vertex_state_at(int64_t v, int64_t nv, const int32_t* __restrict__ voff,
                                                         const int32_t* __restrict__ vcid,
                                                         const T* __restrict__ vw,
                                                         const uint8_t* __restrict__ vbc,
                                                         const Vec4<T>* __restrict__ U, Phys ph,
                                                         Vec4<T>* __restrict__ vq) {
  vq[v] = vertex_state_value<T>(v, voff, vcid, vw, vbc, U, ph);
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_vertex_state(int64_t nv, const int32_t* __restrict__ voff,
                                                         const int32_t* __restrict__ vcid,
                                                         const T* __restrict__ vw,
                                                         const uint8_t* __restrict__ vbc,
                                                         const Vec4<T>* __restrict__ U, Phys ph,
                                                         Vec4<T>* __restrict__ vq, const int* gate) {
  if (gated(gate)) return;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  vertex_state_at<T>(v, nv, voff, vcid, vw, vbc, U, ph, vq);
}

// K3: the same interpolation for the five viscous quantities
// (src/diffusion.cpp:29-140) with apply_diffusion_bc (src/boundary.cpp:101-127):
// far field and wall vertices are zeroed.
template <typename T>
__device__ __forceinline__ Vec4<T> vertex_visc_of(const VertexFan<T>& f, const int32_t* __restrict__ vcid,
                                                  const T* __restrict__ vw, const Vec4<T>* ctq,
                                                  const T* ctqy, T& qy) {
  T a = (T)0.0, b = (T)0.0, c = (T)0.0, d = (T)0.0, e = (T)0.0;
#pragma unroll
  for (int h = 0; h < kFan; h += 4) {
    if (h >= f.n) break;
    Vec4<T> t[4];
    T q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (h + k < f.n) {
        t[k] = ctq[f.cid[h + k]];
        q[k] = ctqy[f.cid[h + k]];
      }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (h + k >= f.n) continue;
      const T w = f.w[h + k];
      if (h + k == 0) {
        a = w * t[k].a;
        b = w * t[k].b;
        c = w * t[k].c;
        d = w * t[k].d;
        e = w * q[k];
      } else {
        a = vertex_add(a, w, t[k].a);
        b = vertex_add(b, w, t[k].b);
        c = vertex_add(c, w, t[k].c);
        d = vertex_add(d, w, t[k].d);
        e = vertex_add(e, w, q[k]);
      }
    }
  }
  for (int k = f.o + kFan; k < f.o + f.n; ++k) {
    const T w = vw[k];
    const int cid = vcid[k];
    const Vec4<T> x = ctq[cid];
    a = vertex_add(a, w, x.a);
    b = vertex_add(b, w, x.b);
    c = vertex_add(c, w, x.c);
    d = vertex_add(d, w, x.d);
    e = vertex_add(e, w, ctqy[cid]);
  }
  if (f.code == 'f' || f.code == 'w') a = b = c = d = e = (T)0.0;
  qy = e;
  return v4<T>(a, b, c, d);
}

template <typename T>
__device__ __forceinline__ Vec4<T> vertex_visc_value(int64_t v, const int32_t* __restrict__ voff,
                                                     const int32_t* __restrict__ vcid, const T* __restrict__ vw,
                                                     const uint8_t* __restrict__ vbc,
                                                     const Vec4<T>* __restrict__ ctq, const T* __restrict__ ctqy,
                                                     T& qy) {
  return vertex_visc_of<T>(vertex_fan<T>(v, voff, vcid, vw, vbc), vcid, vw, ctq, ctqy, qy);
}

template <typename T>
__device__ __forceinline__ void vertex_visc_at(int64_t v, int64_t nv, const int32_t* __restrict__ voff,
                                                        const int32_t* __restrict__ vcid,
                                                        const T* __restrict__ vw,
                                                        const uint8_t* __restrict__ vbc,
                                                        const Vec4<T>* __restrict__ ctq,
                                                        const T* __restrict__ ctqy,
                                                        Vec4<T>* __restrict__ vtq, T* __restrict__ vtqy) {
  T qy;
  vtq[v] = vertex_visc_value<T>(v, voff, vcid, vw, vbc, ctq, ctqy, qy);
  vtqy[v] = qy;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_vertex_visc(int64_t nv, const int32_t* __restrict__ voff,
                                                        const int32_t* __restrict__ vcid,
                                                        const T* __restrict__ vw,
                                                        const uint8_t* __restrict__ vbc,
                                                        const Vec4<T>* __restrict__ ctq,
                                                        const T* __restrict__ ctqy,
                                                        Vec4<T>* __restrict__ vtq, T* __restrict__ vtqy,
                                                        const int* gate) {
  if (gated(gate)) return;
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  vertex_visc_at<T>(v, nv, voff, vcid, vw, vbc, ctq, ctqy, vtq, vtqy);
}

// K2: per cell -- edge values from the vertex states and the Green-Gauss
// gradient (src/advection.cpp:136-188), neighbour min/max, limiter and
// interface states (:236-321), and the cell viscous stress and heat flux from
// the unlimited gradients (src/diffusion.cpp:223-241).
//
// kPlain = false divides without branches (qdiv.h) and returns false if any
// quotient left its range; the caller then redoes the cell, its stores
// included, with kPlain = true (IEEE divisions), out of line.
//
// kAlpha (linearisations only; 0 everywhere else): 1 stores the limiter
// values of the cell in alpha[c], 2 uses alpha[c] instead of computing them
// (the limiter held at a base state).
//
// VQ: where the states of an edge's two vertices come from (by edge and
// global array, or by tile position, kernels_tile.cuh).
template <typename T>
struct EdgeVertexStates {
  const int2* __restrict__ ev;
  const Vec4<T>* __restrict__ vq;
  using Index = int2;
  __device__ __forceinline__ Index index(int, int e) const { return ev[e]; }
  __device__ __forceinline__ Vec4<T> first(Index i) const { return vq[i.x]; }
  __device__ __forceinline__ Vec4<T> second(Index i) const { return vq[i.y]; }
};

template <typename T, bool kWriteGrad, bool kPlain, int kAlpha = 0, typename VQ>
__device__ __forceinline__ bool cell_gradient_body(int64_t c,
    int64_t nc, const int32_t* __restrict__ slot, Geom<T> g, VQ vq,
    const int2* __restrict__ ec, const uint8_t* __restrict__ ebc, const Vec4<T>* U,
    Phys ph, Vec4<T>* eL, Vec4<T>* eR,
    Vec4<T>* ctq, T* ctqy, Vec4<T>* grad, Vec4<T>* alpha = nullptr) {
  const Vec4<T> cg = g.cgeom[c];
  const T cx = cg.a, cy = cg.b, cv = cg.c, veps = cg.d;
  const Vec4<T> u = U[c];
  // The cell's edges are the slots before the first empty one.  All index
  // and geometry loads of every edge are issued before the arithmetic, so
  // the gathers of one cell overlap instead of forming one chain per edge.
  int sl[4], nk = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) sl[k] = slot[(int64_t)k * nc + c];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (sl[k] >= 0 && nk == k) nk = k + 1;
  typename VQ::Index evv[4];
  int2 cc[4];
  uint8_t code[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k < nk) {
      const int e = sl[k] >> 1;
      evv[k] = vq.index(k, e);
      cc[k] = ec[e];
      code[k] = ebc[e];
    }
  }

  // the eight Green-Gauss terms of every edge divide by the cell volume
  constexpr bool kFlat = !kPlain && sizeof(T) == 8;
  bool ok = true;
  T ycv;
  if constexpr (kFlat) ycv = recip_fast(cv, ok);
  else ycv = recip_for_div(cv);
  auto over_v = [&](T a) -> T {
    if constexpr (kPlain) return a / cv;
    else return quot(a, cv, ycv, ok);
  };
  auto limited = [&](T phi, T pred, T mn, T mx) -> T {
    if constexpr (kFlat) return limiter_alpha_flat(ph.limiter, phi, pred, mn, mx, veps, ok);
    else return limiter_alpha(ph.limiter, phi, pred, mn, mx, veps);
  };
  T gx0 = (T)0.0, gx1 = (T)0.0, gx2 = (T)0.0, gx3 = (T)0.0;
  T gy0 = (T)0.0, gy1 = (T)0.0, gy2 = (T)0.0, gy3 = (T)0.0;
  T mn0 = u.a, mn1 = u.b, mn2 = u.c, mn3 = u.d;
  T mx0 = u.a, mx1 = u.b, mx2 = u.c, mx3 = u.d;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= nk) continue;
    const int s = sl[k];
    const int e = s >> 1;
    const bool left = (s & 1) == 0;
    const Vec4<T> va = vq.first(evv[k]), vb = vq.second(evv[k]);
    const Vec4<T> eg = g.egeom[e];
    const int o = left ? cc[k].y : cc[k].x;
    Vec4<T> un = u;
    if (o >= 0) un = U[o];
    T er = (T)0.5 * (va.a + vb.a);
    T eru = (T)0.5 * (va.b + vb.b);
    T erv = (T)0.5 * (va.c + vb.c);
    T eE = (T)0.5 * (va.d + vb.d);
    if (code[k]) bc_state(code[k], ph, er, eru, erv, eE);
    const T el = eg.c;
    T enx = eg.a, eny = eg.b;
    if (left) {
      enx = -enx;
      eny = -eny;
    }
    gx0 += over_v(er * el * enx);
    gx1 += over_v(eru * el * enx);
    gx2 += over_v(erv * el * enx);
    gx3 += over_v(eE * el * enx);
    gy0 += over_v(er * el * eny);
    gy1 += over_v(eru * el * eny);
    gy2 += over_v(erv * el * eny);
    gy3 += over_v(eE * el * eny);
    if (o >= 0) {
      if (un.a < mn0) mn0 = un.a;
      if (un.a > mx0) mx0 = un.a;
      if (un.b < mn1) mn1 = un.b;
      if (un.b > mx1) mx1 = un.b;
      if (un.c < mn2) mn2 = un.c;
      if (un.c > mx2) mx2 = un.c;
      if (un.d < mn3) mn3 = un.d;
      if (un.d > mx3) mx3 = un.d;
    }
  }

  T al0 = (T)1.0, al1 = (T)1.0, al2 = (T)1.0, al3 = (T)1.0;
  T dxk[4], dyk[4];
  if constexpr (kAlpha == 2) {
    const Vec4<T> a = alpha[c];
    al0 = a.a;
    al1 = a.b;
    al2 = a.c;
    al3 = a.d;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= nk) continue;
      const Vec2<T> ce = g.ectr[sl[k] >> 1];
      dxk[k] = ce.a - cx;
      dyk[k] = ce.b - cy;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= nk) continue;
      const Vec2<T> ce = g.ectr[sl[k] >> 1];
      const T dx = ce.a - cx, dy = ce.b - cy;
      dxk[k] = dx;
      dyk[k] = dy;
      al0 = smin(al0, limited(u.a, u.a + gx0 * dx + gy0 * dy, mn0, mx0));
      al1 = smin(al1, limited(u.b, u.b + gx1 * dx + gy1 * dy, mn1, mx1));
      al2 = smin(al2, limited(u.c, u.c + gx2 * dx + gy2 * dy, mn2, mx2));
      al3 = smin(al3, limited(u.d, u.d + gx3 * dx + gy3 * dy, mn3, mx3));
    }
    if constexpr (kAlpha == 1) alpha[c] = v4<T>(al0, al1, al2, al3);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= nk) continue;
    const int s = sl[k];
    const int e = s >> 1;
    const T dx = dxk[k], dy = dyk[k];
    const Vec4<T> st = v4<T>(u.a + al0 * (gx0 * dx + gy0 * dy), u.b + al1 * (gx1 * dx + gy1 * dy),
                             u.c + al2 * (gx2 * dx + gy2 * dy), u.d + al3 * (gx3 * dx + gy3 * dy));
    if ((s & 1) == 0) {
      eL[e] = st;
      if (code[k]) eR[e] = bc_ghost(code[k], ph, st);
    } else {
      eR[e] = st;
    }
  }

  // Viscous stress and heat flux at the cell (src/diffusion.cpp:227-240).
  const T mu = (T)ph.mu, gamma = (T)ph.gamma, kappa = (T)ph.kappa;
  T yrho;
  if constexpr (kFlat) yrho = recip_fast(u.a, ok);
  else yrho = recip_for_div(u.a);
  auto over_rho = [&](T a) -> T {
    if constexpr (kFlat) return quot(a, u.a, yrho, ok);
    else return qdiv(a, u.a, yrho);
  };
  const T rr = u.a * u.a;
  T yrr = (T)0.0;
  if constexpr (kFlat) yrr = recip_fast(rr, ok);
  auto over_rr = [&](T a) -> T {
    if constexpr (kFlat) return quot(a, rr, yrr, ok);
    else return a / rr;
  };
  const T uu = over_rho(u.b);
  const T vv = over_rho(u.c);
  const T u_x = over_rho(gx1 - uu * gx0);
  const T v_y = over_rho(gy2 - vv * gy0);
  const T u_y = over_rho(gy1 - uu * gy0);
  const T v_x = over_rho(gx2 - vv * gx0);
  const T two_thirds = (T)(2.0 / 3.0);
  const T tau_xx = (T)2 * mu * u_x - two_thirds * mu * (u_x + v_y);
  const T tau_yy = (T)2 * mu * v_y - two_thirds * mu * (u_x + v_y);
  const T tau_xy = mu * (u_y + v_x);
  const T T_x = (gamma - (T)1.0) * (over_rr(gx3 * u.a - u.d * gx0) - (uu * u_x + vv * v_x));
  const T T_y = (gamma - (T)1.0) * (over_rr(gy3 * u.a - u.d * gy0) - (uu * u_y + vv * v_y));
  ctq[c] = v4<T>(tau_xx, tau_yy, tau_xy, -kappa * T_x);
  ctqy[c] = -kappa * T_y;
  if (kWriteGrad) {
    grad[2 * c] = v4<T>(gx0, gx1, gx2, gx3);
    grad[2 * c + 1] = v4<T>(gy0, gy1, gy2, gy3);
  }
  return kPlain || ok;
}

template <typename T, bool kWriteGrad, int kAlpha = 0, typename VQ>
__device__ __noinline__ void cell_gradient_plain(int64_t c,
    int64_t nc, const int32_t* __restrict__ slot, Geom<T> g, VQ vq,
    const int2* __restrict__ ec, const uint8_t* __restrict__ ebc, const Vec4<T>* U,
    Phys ph, Vec4<T>* eL, Vec4<T>* eR,
    Vec4<T>* ctq, T* ctqy, Vec4<T>* grad, Vec4<T>* alpha) {
  cell_gradient_body<T, kWriteGrad, true, kAlpha>(c, nc, slot, g, vq, ec, ebc, U, ph, eL, eR, ctq, ctqy, grad, alpha);
}

template <typename T, bool kWriteGrad, int kAlpha = 0, typename VQ>
__device__ __forceinline__ void cell_gradient_from(int64_t c,
    int64_t nc, const int32_t* __restrict__ slot, Geom<T> g, VQ vq,
    const int2* __restrict__ ec, const uint8_t* __restrict__ ebc, const Vec4<T>* U,
    Phys ph, Vec4<T>* eL, Vec4<T>* eR,
    Vec4<T>* ctq, T* ctqy, Vec4<T>* grad,
    Vec4<T>* alpha = nullptr) {
  if (!cell_gradient_body<T, kWriteGrad, false, kAlpha>(c, nc, slot, g, vq, ec, ebc, U, ph, eL, eR, ctq, ctqy, grad,
                                                        alpha))
    cell_gradient_plain<T, kWriteGrad, kAlpha>(c, nc, slot, g, vq, ec, ebc, U, ph, eL, eR, ctq, ctqy, grad, alpha);
}

template <typename T, bool kWriteGrad, int kAlpha = 0>
__device__ __forceinline__ void cell_gradient_at(int64_t c,
    int64_t nc, const int32_t* __restrict__ slot, Geom<T> g, const int2* __restrict__ ev,
    const int2* __restrict__ ec, const uint8_t* __restrict__ ebc, const Vec4<T>* __restrict__ U,
    const Vec4<T>* __restrict__ vq, Phys ph, Vec4<T>* __restrict__ eL, Vec4<T>* __restrict__ eR,
    Vec4<T>* __restrict__ ctq, T* __restrict__ ctqy, Vec4<T>* __restrict__ grad,
    Vec4<T>* __restrict__ alpha = nullptr) {
  cell_gradient_from<T, kWriteGrad, kAlpha>(c, nc, slot, g, EdgeVertexStates<T>{ev, vq}, ec, ebc, U, ph, eL, eR, ctq,
                                            ctqy, grad, alpha);
}

template <typename T, bool kWriteGrad>
__global__ void __launch_bounds__(kGradBlock, 6) k_cell_gradient(
    int64_t nc, const int32_t* __restrict__ slot, Geom<T> g, const int2* __restrict__ ev,
    const int2* __restrict__ ec, const uint8_t* __restrict__ ebc, const Vec4<T>* __restrict__ U,
    const Vec4<T>* __restrict__ vq, Phys ph, Vec4<T>* __restrict__ eL, Vec4<T>* __restrict__ eR,
    Vec4<T>* __restrict__ ctq, T* __restrict__ ctqy, Vec4<T>* __restrict__ grad, const int* gate) {
  if (gated(gate)) return;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  cell_gradient_at<T, kWriteGrad>(c, nc, slot, g, ev, ec, ebc, U, vq, ph, eL, eR, ctq, ctqy, grad);
}

// K4: per edge -- HLLC flux (src/advection.cpp:433-437) and the edge viscous
// quantities with their boundary conditions (src/diffusion.cpp:145-170).
template <typename T>
__device__ __forceinline__ Vec4<T> edge_visc_value(const Vec4<T>& a, T ay, const Vec4<T>& b, T by, uint8_t code,
                                                   T& qy_out) {
  T txx = (T)0.5 * (a.a + b.a);
  T tyy = (T)0.5 * (a.b + b.b);
  T txy = (T)0.5 * (a.c + b.c);
  T qx = (T)0.5 * (a.d + b.d);
  T qy = (T)0.5 * (ay + by);
  if (code == 'f' || code == 'w') txx = tyy = txy = qx = qy = (T)0.0;
  qy_out = qy;
  return v4<T>(txx, tyy, txy, qx);
}

template <typename T>
__device__ __forceinline__ void edge_flux_at(int64_t e, int64_t ne, Geom<T> g, const int2* __restrict__ ev,
                                                      const uint8_t* __restrict__ ebc,
                                                      const Vec4<T>* __restrict__ eL,
                                                      const Vec4<T>* __restrict__ eR,
                                                      const Vec4<T>* __restrict__ vtq,
                                                      const T* __restrict__ vtqy, Phys ph,
                                                      Vec4<T>* __restrict__ F, Vec4<T>* __restrict__ etq,
                                                      T* __restrict__ etqy) {
  const Vec4<T> eg = g.egeom[e];
  F[e] = hllc_flux(eL[e], eR[e], eg.a, eg.b, (T)ph.gamma);
  const int2 vv = ev[e];
  T qy;
  etq[e] = edge_visc_value<T>(vtq[vv.x], vtqy[vv.x], vtq[vv.y], vtqy[vv.y], ebc[e], qy);
  etqy[e] = qy;
}

template <typename T>
__global__ void __launch_bounds__(kBlock, 4) k_edge_flux(int64_t ne, Geom<T> g, const int2* __restrict__ ev,
                                                      const uint8_t* __restrict__ ebc,
                                                      const Vec4<T>* __restrict__ eL,
                                                      const Vec4<T>* __restrict__ eR,
                                                      const Vec4<T>* __restrict__ vtq,
                                                      const T* __restrict__ vtqy, Phys ph,
                                                      Vec4<T>* __restrict__ F, Vec4<T>* __restrict__ etq,
                                                      T* __restrict__ etqy, const int* gate) {
  if (gated(gate)) return;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  edge_flux_at<T>(e, ne, g, ev, ebc, eL, eR, vtq, vtqy, ph, F, etq, etqy);
}

// Partial sum of squares of a block, written to part[blockIdx.x].
__device__ __forceinline__ double block_sum(double v, double* smem) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += smem[w];
  }
  return s;  // valid in thread 0
}

// RK3 stage parameters for the fused residual + update.
struct RkStage {
  double c0, c1;        // U = c0*U_old + c1*(U + dt*R)
  const double* dt;     // device scalar
  int snapshot;         // 1: copy U to U_old first (stage 1)
  double* norm_part;    // per-block partial sums of R_rho^2 (stage 1), or null
};

// K5: per cell -- residual gather R = -(1/V) sum sign*F*L
// (src/advection.cpp:439-464), then the viscous Green-Gauss divergence added
// to R (src/diffusion.cpp:176-201).  kRk fuses the SSP-RK3 stage update of
// Simulator::rk3_substep (src/simulation.cpp:159-167).
// Returns R_rho^2 of cell c for the residual-norm partial sums (0 unless
// kRk with norm partials requested).
// ED: where an edge's geometry, flux and viscous quantities come from (the
// global arrays, or a tile's, kernels_tile.cuh).  unew: the updated state.
template <typename T>
struct EdgeFluxes {
  const Vec4<T>* __restrict__ egeom;
  const Vec4<T>* __restrict__ F;
  const Vec4<T>* __restrict__ etq;
  const T* __restrict__ etqy;
  __device__ __forceinline__ int at(int, int e) const { return e; }
  __device__ __forceinline__ T length(int i) const { return egeom[i].c; }
  __device__ __forceinline__ Vec4<T> geom(int i) const { return egeom[i]; }
  __device__ __forceinline__ Vec4<T> flux(int i) const { return F[i]; }
  __device__ __forceinline__ Vec4<T> visc(int i) const { return etq[i]; }
  __device__ __forceinline__ T visc_y(int i) const { return etqy[i]; }
};

//
// cell_residual_sum: kPlain = false divides without branches and returns
// false where a quotient left its range (qdiv.h).
template <typename T, bool kPlain, typename ED>
__device__ __forceinline__ bool cell_residual_sum(int64_t c, int64_t nc, const int32_t* __restrict__ slot,
                                                  const Vec4<T>* __restrict__ cgeom, ED ed, const Vec4<T>& u,
                                                  Vec4<T>& out) {
  bool ok = true;
  const T cv = cgeom[c].c;
  int sl[4], nk = 0;  // the cell's edges are the slots before the first empty one
#pragma unroll
  for (int k = 0; k < 4; ++k) sl[k] = slot[(int64_t)k * nc + c];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (sl[k] >= 0 && nk == k) nk = k + 1;
  T a0 = (T)0.0, a1 = (T)0.0, a2 = (T)0.0, a3 = (T)0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= nk) continue;
    const int s = sl[k];
    const int e = s >> 1;
    const T sign = ((s & 1) == 0) ? (T)1.0 : (T)-1.0;
    const int i = ed.at(k, e);
    const T L = ed.length(i);
    const Vec4<T> f = ed.flux(i);
    a0 += sign * f.a * L;
    a1 += sign * f.b * L;
    a2 += sign * f.c * L;
    a3 += sign * f.d * L;
  }
  T invV, ycv, yrho = (T)0.0;
  if constexpr (kPlain) {
    invV = (T)1.0 / cv;
    ycv = recip_for_div(cv, invV);
  } else {
    invV = ycv = recip_fast(cv, ok);
    yrho = recip_fast(u.a, ok);
  }
  auto over_v = [&](T a) -> T {
    if constexpr (kPlain) return qdiv(a, cv, ycv);
    else return quot(a, cv, ycv, ok);
  };
  auto over_rho = [&](T a) -> T {
    if constexpr (kPlain) return a / u.a;
    else return quot(a, u.a, yrho, ok);
  };
  a0 *= -invV;
  a1 *= -invV;
  a2 *= -invV;
  a3 *= -invV;
  const T uu = over_rho(u.b);
  const T vv = over_rho(u.c);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= nk) continue;
    const int s = sl[k];
    const int e = s >> 1;
    const int i = ed.at(k, e);
    const Vec4<T> eg = ed.geom(i);
    const T el = eg.c;
    T enx = eg.a, eny = eg.b;
    if ((s & 1) == 0) {
      enx = -enx;
      eny = -eny;
    }
    const Vec4<T> t = ed.visc(i);
    const T qy = ed.visc_y(i);
    a1 += over_v(t.a * el * enx) + over_v(t.c * el * eny);
    a2 += over_v(t.c * el * enx) + over_v(t.b * el * eny);
    a3 += over_v((uu * t.a + vv * t.c - t.d) * el * enx) + over_v((uu * t.c + vv * t.b - qy) * el * eny);
  }
  out = v4<T>(a0, a1, a2, a3);
  return ok;
}

template <typename T, typename ED>
__device__ __noinline__ Vec4<T> cell_residual_plain(int64_t c, int64_t nc, const int32_t* __restrict__ slot,
                                                    const Vec4<T>* __restrict__ cgeom, ED ed, const Vec4<T> u) {
  Vec4<T> r;
  cell_residual_sum<T, true>(c, nc, slot, cgeom, ed, u, r);
  return r;
}

template <typename T, bool kRk, typename ED>
__device__ __forceinline__ double cell_residual_from(int64_t c, int64_t nc, const int32_t* __restrict__ slot,
                                                     const Vec4<T>* __restrict__ cgeom, ED ed,
                                                     Vec4<T>* U, Vec4<T>* Uold,
                                                     Vec4<T>* R, const RkStage& rk,
                                                     Vec4<T>* unew = nullptr) {
  double r2 = 0.0;
  Vec4<T> u = U[c], r;
  if (!cell_residual_sum<T, false>(c, nc, slot, cgeom, ed, u, r)) r = cell_residual_plain<T>(c, nc, slot, cgeom, ed, u);
  const T a0 = r.a, a1 = r.b, a2 = r.c, a3 = r.d;
  if (!kRk || R) R[c] = r;
  if (kRk) {
    if (rk.norm_part) r2 = (double)a0 * (double)a0;
    const T dt = (T)(*rk.dt);
    const T c0 = (T)rk.c0, c1 = (T)rk.c1;
    Vec4<T> uo;
    if (rk.snapshot) {
      uo = u;
      Uold[c] = u;
    } else {
      uo = Uold[c];
    }
    u.a = c0 * uo.a + c1 * (u.a + dt * (a0));
    u.b = c0 * uo.b + c1 * (u.b + dt * (a1));
    u.c = c0 * uo.c + c1 * (u.c + dt * (a2));
    u.d = c0 * uo.d + c1 * (u.d + dt * (a3));
    U[c] = u;
    if (unew) *unew = u;
  }
  return r2;
}

template <typename T, bool kRk>
__device__ __forceinline__ double cell_residual_at(int64_t c, int64_t nc, const int32_t* __restrict__ slot, Geom<T> g,
                                                   const Vec4<T>* __restrict__ F, const Vec4<T>* __restrict__ etq,
                                                   const T* __restrict__ etqy, Vec4<T>* __restrict__ U,
                                                   Vec4<T>* __restrict__ Uold, Vec4<T>* __restrict__ R,
                                                   const RkStage& rk) {
  return cell_residual_from<T, kRk>(c, nc, slot, g.cgeom, EdgeFluxes<T>{g.egeom, F, etq, etqy}, U, Uold, R, rk);
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_cell_residual(int64_t nc, const int32_t* __restrict__ slot, Geom<T> g,
                                                          const Vec4<T>* __restrict__ F,
                                                          const Vec4<T>* __restrict__ etq,
                                                          const T* __restrict__ etqy, Vec4<T>* __restrict__ U,
                                                          Vec4<T>* __restrict__ R) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) cell_residual_at<T, false>(c, nc, slot, g, F, etq, etqy, U, nullptr, R, RkStage{});
}

}  // namespace o2f
