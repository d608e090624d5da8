// fj_physics.cuh -- per-cell / per-face physics of the famrdp_jax hot path as
// device functions, templated on the flux arithmetic type T (double for the
// drop-in FP64 path, float for the FP32-flux path).
//
// Each function restates the reference expression it cites (famrdp_jax,
// path:line) in the same operation order; nvcc may contract a*b+c into one
// FMA, which changes results by at most one rounding per contraction.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fj {

// Clamp constants of the reference (flux/roe.py:6,23-24,33,39; rhs/invscd.py:93,
// 126; rhs/viscous.py:36).  FP32 cannot represent 1e-300 / 1e-150, so the float
// path uses the smallest normal-range values that keep the same role.
template <typename T> struct Tiny;
template <> struct Tiny<double> {
  static __device__ __forceinline__ double rho() { return 1e-300; }
  static __device__ __forceinline__ double ss() { return 1e-150; }
  static __device__ __forceinline__ double c2() { return 1e-30; }
  static __device__ __forceinline__ double nmag() { return 1e-300; }
};
template <> struct Tiny<float> {
  static __device__ __forceinline__ float rho() { return 1e-37f; }
  static __device__ __forceinline__ float ss() { return 1e-18f; }
  static __device__ __forceinline__ float c2() { return 1e-30f; }
  static __device__ __forceinline__ float nmag() { return 1e-37f; }
};

__device__ __forceinline__ double fj_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float fj_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double fj_abs(double x) { return fabs(x); }
__device__ __forceinline__ float fj_abs(float x) { return fabsf(x); }
__device__ __forceinline__ double fj_max(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float fj_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double fj_min(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float fj_min(float a, float b) { return fminf(a, b); }

// jnp.sign: -1, 0 or +1 (NaN propagates; not reached on finite data).
template <typename T> __device__ __forceinline__ T fj_sign(T x) {
  return x > T(0) ? T(1) : (x < T(0) ? T(-1) : T(0));
}

template <typename T> struct Prim { T rho, u, v, w, p; };
template <typename T> struct Cons { T r, ru, rv, rw, rE; };
template <typename T> struct Vec5 { T a[5]; };

// physics/eos.py:12-17 (no density clamp)
template <typename T>
__device__ __forceinline__ Prim<T> cons_to_prim(T r, T ru, T rv, T rw, T rE, T gm1) {
  Prim<T> o;
  o.rho = r;
  o.u = ru / r;
  o.v = rv / r;
  o.w = rw / r;
  T ke = T(0.5) * (o.u * o.u + o.v * o.v + o.w * o.w);
  o.p = gm1 * (rE - r * ke);
  return o;
}

// physics/eos.py:5-9
template <typename T>
__device__ __forceinline__ Cons<T> prim_to_cons(const Prim<T>& pv, T gm1) {
  Cons<T> o;
  T ke = T(0.5) * (pv.u * pv.u + pv.v * pv.v + pv.w * pv.w);
  o.r = pv.rho;
  o.ru = pv.rho * pv.u;
  o.rv = pv.rho * pv.v;
  o.rw = pv.rho * pv.w;
  o.rE = pv.p / gm1 + pv.rho * ke;
  return o;
}

// physics/reconstruct/muscl2.py:5-7
template <typename T> __device__ __forceinline__ T minmod(T a, T b) {
  T sa = fj_sign(a);
  T s = sa * fj_max(sa * fj_sign(b), T(0));
  return s * fj_min(fj_abs(a), fj_abs(b));
}

// physics/reconstruct/muscl2.py:10-12
template <typename T> __device__ __forceinline__ T vanleer(T a, T b) {
  T sd = fj_abs(a + b) > T(1e-30) ? a + b : T(1);
  return a * b > T(0) ? T(2) * a * b / sd : T(0);
}

template <typename T> __device__ __forceinline__ T limit(T a, T b, int limiter) {
  return limiter == 0 ? minmod(a, b) : vanleer(a, b);
}

// physics/reconstruct/muscl2.py:18-37 for one face between cells c1 and c2:
// pL = c1 + 0.5*lim(c1-c0, c2-c1), pR = c2 - 0.5*lim(c2-c1, c3-c2)
template <typename T>
__device__ __forceinline__ void muscl2(T c0, T c1, T c2, T c3, int limiter, T& L, T& R) {
  T sL = limit(c1 - c0, c2 - c1, limiter);
  T sR = limit(c2 - c1, c3 - c2, limiter);
  L = c1 + T(0.5) * sL;
  R = c2 - T(0.5) * sR;
}

// flux/roe.py:5-18
template <typename T>
__device__ __forceinline__ void physical_flux(const Cons<T>& U, T n0, T n1, T n2, T gm1,
                                              T F[5]) {
  T rho = fj_max(U.r, Tiny<T>::rho());
  T u = U.ru / rho, v = U.rv / rho, w = U.rw / rho;
  T ke = T(0.5) * (u * u + v * v + w * w);
  T p = gm1 * (U.rE - rho * ke);
  T un = u * n0 + v * n1 + w * n2;
  T H = (U.rE + p) / rho;
  F[0] = rho * un;
  F[1] = rho * u * un + p * n0;
  F[2] = rho * v * un + p * n1;
  F[3] = rho * w * un + p * n2;
  F[4] = rho * H * un;
}

// flux/roe.py:21-85: Roe flux along the unit normal (n0, n1, n2) with the
// Harten fix on lambda_1 and lambda_5 and the reference's shear term.
template <typename T>
__device__ __forceinline__ void roe_flux(const Cons<T>& UL, const Cons<T>& UR, T n0, T n1,
                                         T n2, T gm1, T eps_entropy, T F[5]) {
  const T rhoL = fj_max(UL.r, Tiny<T>::rho());
  const T rhoR = fj_max(UR.r, Tiny<T>::rho());
  const T uL = UL.ru / rhoL, vL = UL.rv / rhoL, wL = UL.rw / rhoL;
  const T uR = UR.ru / rhoR, vR = UR.rv / rhoR, wR = UR.rw / rhoR;
  const T keL = T(0.5) * (uL * uL + vL * vL + wL * wL);
  const T keR = T(0.5) * (uR * uR + vR * vR + wR * wR);
  const T pL = gm1 * (UL.rE - rhoL * keL);
  const T pR = gm1 * (UR.rE - rhoR * keR);
  const T HL = (UL.rE + pL) / rhoL;
  const T HR = (UR.rE + pR) / rhoR;

  const T sqL = fj_sqrt(rhoL), sqR = fj_sqrt(rhoR);
  const T ss = fj_max(sqL + sqR, Tiny<T>::ss());
  const T u_h = (sqL * uL + sqR * uR) / ss;
  const T v_h = (sqL * vL + sqR * vR) / ss;
  const T w_h = (sqL * wL + sqR * wR) / ss;
  const T H_h = (sqL * HL + sqR * HR) / ss;
  const T q2 = u_h * u_h + v_h * v_h + w_h * w_h;
  const T c2 = fj_max(gm1 * (H_h - T(0.5) * q2), Tiny<T>::c2());
  const T c_h = fj_sqrt(c2);
  const T un_h = u_h * n0 + v_h * n1 + w_h * n2;
  const T rho_h = sqL * sqR;

  const T eps = eps_entropy * (fj_abs(un_h) + c_h);
  const T lam1 = un_h - c_h, lam5 = un_h + c_h;
  const T al1 = fj_abs(lam1) >= eps ? fj_abs(lam1) : T(0.5) * (lam1 * lam1 / eps + eps);
  const T al5 = fj_abs(lam5) >= eps ? fj_abs(lam5) : T(0.5) * (lam5 * lam5 / eps + eps);
  const T al2 = fj_abs(un_h);

  const T d0 = UR.r - UL.r, d1 = UR.ru - UL.ru, d2 = UR.rv - UL.rv, d3 = UR.rw - UL.rw,
          d4 = UR.rE - UL.rE;
  const T dp = gm1 * (d4 - u_h * d1 - v_h * d2 - w_h * d3 + T(0.5) * q2 * d0);
  const T dun = (d1 * n0 + d2 * n1 + d3 * n2) - un_h * d0;
  const T a1 = (dp - rho_h * c_h * dun) / (T(2) * c2);
  const T a5 = (dp + rho_h * c_h * dun) / (T(2) * c2);
  const T a23 = d0 - dp / c2;

  const T du_t = d1 / rho_h - u_h * d0 / rho_h;
  const T dv_t = d2 / rho_h - v_h * d0 / rho_h;
  const T dw_t = d3 / rho_h - w_h * d0 / rho_h;
  const T dun_full = du_t * n0 + dv_t * n1 + dw_t * n2;
  const T tu = du_t - dun_full * n0, tv = dv_t - dun_full * n1, tw = dw_t - dun_full * n2;
  const T dvt1 = rho_h * tu, dvt2 = rho_h * tv, dvt3 = rho_h * tw;
  const T dvt4 = rho_h * (u_h * tu + v_h * tv + w_h * tw);

  const T s1 = al1 * a1, s5 = al5 * a5;
  T A[5];
  A[0] = s1 + s5 + al2 * a23;
  A[1] = s1 * (u_h - c_h * n0) + s5 * (u_h + c_h * n0) + al2 * (a23 * u_h + dvt1);
  A[2] = s1 * (v_h - c_h * n1) + s5 * (v_h + c_h * n1) + al2 * (a23 * v_h + dvt2);
  A[3] = s1 * (w_h - c_h * n2) + s5 * (w_h + c_h * n2) + al2 * (a23 * w_h + dvt3);
  A[4] = s1 * (H_h - c_h * un_h) + s5 * (H_h + c_h * un_h) + al2 * (a23 * (T(0.5) * q2) + dvt4);

  T FL[5], FR[5];
  physical_flux(UL, n0, n1, n2, gm1, FL);
  physical_flux(UR, n0, n1, n2, gm1, FR);
#pragma unroll
  for (int v = 0; v < 5; ++v) F[v] = T(0.5) * (FL[v] + FR[v]) - T(0.5) * A[v];
}

// One inviscid face of rhs/invscd.py:62-100 between cells c1 and c2 along an
// axis: MUSCL on the primitives of the four cells c0..c3, prim->cons, face
// normal = 0.5*(kxyz row of c1 + row of c2), |n| + tiny, Roe, times |n|.
template <typename T>
__device__ __forceinline__ void invscd_face(const Prim<T> c[4], T kl0, T kl1, T kl2, T kr0,
                                            T kr1, T kr2, T gm1, T eps_entropy, int limiter,
                                            T F[5]) {
  Prim<T> L, R;
  muscl2(c[0].rho, c[1].rho, c[2].rho, c[3].rho, limiter, L.rho, R.rho);
  muscl2(c[0].u, c[1].u, c[2].u, c[3].u, limiter, L.u, R.u);
  muscl2(c[0].v, c[1].v, c[2].v, c[3].v, limiter, L.v, R.v);
  muscl2(c[0].w, c[1].w, c[2].w, c[3].w, limiter, L.w, R.w);
  muscl2(c[0].p, c[1].p, c[2].p, c[3].p, limiter, L.p, R.p);
  const Cons<T> UL = prim_to_cons(L, gm1);
  const Cons<T> UR = prim_to_cons(R, gm1);
  const T nf0 = T(0.5) * (kl0 + kr0), nf1 = T(0.5) * (kl1 + kr1), nf2 = T(0.5) * (kl2 + kr2);
  const T nmag = fj_sqrt(nf0 * nf0 + nf1 * nf1 + nf2 * nf2) + Tiny<T>::nmag();
  roe_flux(UL, UR, nf0 / nmag, nf1 / nmag, nf2 / nmag, gm1, eps_entropy, F);
#pragma unroll
  for (int v = 0; v < 5; ++v) F[v] = F[v] * nmag;
}

// ---------------------------------------------------------------------------
// Reformulated face flux for the fused kernels.  Same mathematics as
// roe_flux + prim_to_cons above, rearranged to cut divisions and recomputation:
//   * the face states stay primitive (the reference rebuilds u = (rho u)/rho,
//     p = (g-1)(rhoE - rho ke) from the conserved states it just built, which
//     returns the same values up to rounding);
//   * one reciprocal per divisor (1/(sqL+sqR), 1/c^2, 1/eps, 1/rho);
//   * the shear term rho_h (du_t - (du_t . n) n) of flux/roe.py:69-79 equals
//     (dU_m - u_h,m dU_0) - dun n_m with dun the normal-velocity jump of
//     flux/roe.py:57, so it needs no division by rho_h.
// For T = float the reciprocals and square roots use the fast MUFU-based
// intrinsics (__fdividef, rsqrtf); the FP32-flux path's tolerance is 1e-5.
// ---------------------------------------------------------------------------
template <typename T> struct FastMath;
template <> struct FastMath<double> {
  // __drcp_rn: the IEEE round-to-nearest reciprocal, the same value as 1.0 / x
  static __device__ __forceinline__ double rcp(double x) { return __drcp_rn(x); }
  static __device__ __forceinline__ double sqrt_pos(double x) { return sqrt(x); }
};
template <> struct FastMath<float> {
  static __device__ __forceinline__ float rcp(float x) { return __fdividef(1.0f, x); }
  // x must be > 0
  static __device__ __forceinline__ float sqrt_pos(float x) { return x * rsqrtf(x); }
  // x >= 0
  static __device__ __forceinline__ float sqrt_nn(float x) { return x > 0.0f ? x * rsqrtf(x) : 0.0f; }
  // The same for an x that is no subnormal number: one instruction, where the
  // forms above also scale subnormal arguments (three more).  The same values
  // otherwise.  With the clamped minmod of muscl2_fast and host-rounded constants:
  // 30.4 -> 26.9 warp instructions a cell in the flux kernel, 145 -> 135 us for
  // 4.0 M cells, the same bits.
  static __device__ __forceinline__ float rcp_n(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
  }
  static __device__ __forceinline__ float sqrt_n(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return x * r;
  }
};

// minmod(a, b) of muscl2.py:5-7 in four min/max: the smaller-magnitude argument when
// both have the same sign, else 0 (one of the two terms is 0).  No product of the
// arguments, which would underflow where both are small.
template <typename T> __device__ __forceinline__ T minmod_sel(T a, T b) {
  return fj_max(fj_min(a, b), T(0)) + fj_min(fj_max(a, b), T(0));
}

// MINMOD: the limiter, else van Leer.
template <typename T, bool MINMOD>
__device__ __forceinline__ void muscl2_one(T c0, T c1, T c2, T c3, T& L, T& R) {
  const T d0 = c1 - c0, d1 = c2 - c1, d2 = c3 - c2;
  T sL, sR;
  if constexpr (!MINMOD) {
    sL = vanleer(d0, d1);
    sR = vanleer(d1, d2);
  } else if constexpr (sizeof(T) == 4) {
    // minmod(d, d1) clamps d to the interval between 0 and d1, which both
    // slopes share: six min/max instead of two products, four comparisons
    // and four selections (the same values; where |d d1| underflows, the
    // smaller magnitude instead of 0, as the reference)
    const T lo = fj_min(d1, T(0)), hi = fj_max(d1, T(0));
    sL = fj_min(fj_max(d0, lo), hi);
    sR = fj_min(fj_max(d2, lo), hi);
  } else {
    // picks the outer difference where it is smaller than the face's own d1, and
    // 0 where the signs differ; the sign test reads the sign bits (a zero argument
    // gives 0 either way), which keeps a multiplication and a comparison off the
    // FP64 pipe.  A NaN outer difference loses the comparison, so it reaches no
    // face whose own two cells are finite.
    const auto pick = [&](T o) {
      const T m = fj_abs(o) < fj_abs(d1) ? o : d1;
      return (__double2hiint(o) ^ __double2hiint(d1)) < 0 ? T(0) : m;
    };
    sL = pick(d0);
    sR = pick(d2);
  }
  L = c1 + T(0.5) * sL;
  R = c2 - T(0.5) * sR;
}

// The face states of all five variables.  FP64 tests the limiter once, so that the
// variables' arithmetic is one straight run of instructions (FP64 step of 4.0 M
// cells 1.776 -> 1.751 ms).  FP32 tests it per variable: in one run the compiler
// fuses the states' last operations into the flux, which changes its rounding and
// gains nothing.
template <typename T>
__device__ __forceinline__ void muscl2_fast(const Prim<T> c[4], int limiter, Prim<T>& L, Prim<T>& R) {
#define FJ_MUSCL(K, f) muscl2_one<T, K>(c[0].f, c[1].f, c[2].f, c[3].f, L.f, R.f);
#define FJ_MUSCL_TEST(f)       \
  if (limiter == 0) {          \
    FJ_MUSCL(true, f)          \
  } else {                     \
    FJ_MUSCL(false, f)         \
  }
  if constexpr (sizeof(T) == 4) {
    FJ_MUSCL_TEST(rho) FJ_MUSCL_TEST(u) FJ_MUSCL_TEST(v) FJ_MUSCL_TEST(w) FJ_MUSCL_TEST(p)
  } else if (limiter == 0) {
    FJ_MUSCL(true, rho) FJ_MUSCL(true, u) FJ_MUSCL(true, v) FJ_MUSCL(true, w) FJ_MUSCL(true, p)
  } else {
    FJ_MUSCL(false, rho) FJ_MUSCL(false, u) FJ_MUSCL(false, v) FJ_MUSCL(false, w) FJ_MUSCL(false, p)
  }
#undef FJ_MUSCL_TEST
#undef FJ_MUSCL
}

// Roe flux (flux/roe.py:21-85) in FP32 of the primitive face states L, R along the
// unit normal n; inv_gm1 = 1/(gamma-1).  (FP64: roe_face_f64.)
//
// POFF (the FP32-flux split path): the states carry the pressure OFFSET
// p' = p - p_ref instead of p.  The energies and enthalpies add p_ref back as
// constants, energy differences use p' differences, and the momentum
// components leave out the constant part p_ref n of their pressure term
// (p n = p' n + p_ref n), which the caller adds in FP64.  In FP32 that keeps
// the rounding of the large, nearly uniform pressure out of the small
// momentum fluxes and pressure jumps.  The two forms are equal in exact
// arithmetic; POFF = false is the reference arrangement.
template <typename T, bool POFF = false>
__device__ __forceinline__ void roe_prim(const Prim<T>& L, const Prim<T>& R, T n0, T n1, T n2,
                                         T gm1, T inv_gm1, T eps_entropy, T F[5], T p_ref = T(0)) {
  static_assert(sizeof(T) == 4, "FP64 faces: roe_face_f64");
  using M = FastMath<T>;
  // arguments of rcp_n / sqrt_n are clamped above the subnormal range (eps is
  // used only where it exceeds an eigenvalue)
  const T rhoL = fj_max(L.rho, Tiny<T>::rho()), rhoR = fj_max(R.rho, Tiny<T>::rho());
  const T keL = T(0.5) * (L.u * L.u + L.v * L.v + L.w * L.w);
  const T keR = T(0.5) * (R.u * R.u + R.v * R.v + R.w * R.w);
  // conserved energies (eos.py:8) and enthalpies
  const T eL = L.p * inv_gm1 + L.rho * keL, eR = R.p * inv_gm1 + R.rho * keR;
  const T Ec = POFF ? p_ref * inv_gm1 : T(0), Hc = POFF ? p_ref * (inv_gm1 + T(1)) : T(0);
  const T EL = POFF ? eL + Ec : eL;
  const T ER = POFF ? eR + Ec : eR;
  const T irL = M::rcp_n(rhoL), irR = M::rcp_n(rhoR);
  const T HL = (POFF ? (eL + L.p) + Hc : EL + L.p) * irL;
  const T HR = (POFF ? (eR + R.p) + Hc : ER + R.p) * irR;
  // Roe weights sqL / (sqL + sqR), sqR / (sqL + sqR) and rho_h = sqL sqR
  const T sqL = M::sqrt_n(rhoL), sqR = M::sqrt_n(rhoR);
  const T inv_ss = M::rcp_n(fj_max(sqL + sqR, Tiny<T>::ss()));
  const T wl = sqL * inv_ss, wr = sqR * inv_ss, rho_h = sqL * sqR;
  const T u_h = wl * L.u + wr * R.u;
  const T v_h = wl * L.v + wr * R.v;
  const T w_h = wl * L.w + wr * R.w;
  const T H_h = wl * HL + wr * HR;
  const T q2 = u_h * u_h + v_h * v_h + w_h * w_h;
  const T c2 = fj_max(gm1 * (H_h - T(0.5) * q2), Tiny<T>::c2());
  const T c_h = M::sqrt_n(c2), inv_c2 = M::rcp_n(c2);
  const T un_h = u_h * n0 + v_h * n1 + w_h * n2;

  const T eps = eps_entropy * (fj_abs(un_h) + c_h);
  const T lam1 = un_h - c_h, lam5 = un_h + c_h;
  T al1 = fj_abs(lam1), al5 = fj_abs(lam5);
  const T inv_eps = M::rcp_n(eps);  // Harten's fix (flux/roe.py:45-52)
  al1 = al1 >= eps ? al1 : T(0.5) * (lam1 * lam1 * inv_eps + eps);
  al5 = al5 >= eps ? al5 : T(0.5) * (lam5 * lam5 * inv_eps + eps);
  const T al2 = fj_abs(un_h);

  const T d0 = R.rho - L.rho;
  const T d1 = R.rho * R.u - L.rho * L.u;
  const T d2 = R.rho * R.v - L.rho * L.v;
  const T d3 = R.rho * R.w - L.rho * L.w;
  const T d4 = POFF ? eR - eL : ER - EL;
  const T dp = gm1 * (d4 - u_h * d1 - v_h * d2 - w_h * d3 + T(0.5) * q2 * d0);
  const T dun = (d1 * n0 + d2 * n1 + d3 * n2) - un_h * d0;
  const T rcd = rho_h * c_h * dun;
  const T hc2 = T(0.5) * inv_c2;
  const T a1 = (dp - rcd) * hc2;
  const T a5 = (dp + rcd) * hc2;
  const T a23 = d0 - dp * inv_c2;
  const T t1 = (d1 - u_h * d0) - dun * n0;
  const T t2 = (d2 - v_h * d0) - dun * n1;
  const T t3 = (d3 - w_h * d0) - dun * n2;
  const T t4 = u_h * t1 + v_h * t2 + w_h * t3;

  const T s1 = al1 * a1, s5 = al5 * a5;
  const T cn0 = c_h * n0, cn1 = c_h * n1, cn2 = c_h * n2, cun = c_h * un_h;
  const T unL = L.u * n0 + L.v * n1 + L.w * n2;
  const T unR = R.u * n0 + R.v * n1 + R.w * n2;
  const T mL = rhoL * unL, mR = rhoR * unR;
  F[0] = T(0.5) * (mL + mR) - T(0.5) * (s1 + s5 + al2 * a23);
  const T pL = L.p, pR = R.p;  // p' with POFF: the p_ref n part is the caller's
  F[1] = T(0.5) * ((mL * L.u + pL * n0) + (mR * R.u + pR * n0)) -
         T(0.5) * (s1 * (u_h - cn0) + s5 * (u_h + cn0) + al2 * (a23 * u_h + t1));
  F[2] = T(0.5) * ((mL * L.v + pL * n1) + (mR * R.v + pR * n1)) -
         T(0.5) * (s1 * (v_h - cn1) + s5 * (v_h + cn1) + al2 * (a23 * v_h + t2));
  F[3] = T(0.5) * ((mL * L.w + pL * n2) + (mR * R.w + pR * n2)) -
         T(0.5) * (s1 * (w_h - cn2) + s5 * (w_h + cn2) + al2 * (a23 * w_h + t3));
  F[4] = T(0.5) * (mL * HL + mR * HR) -
         T(0.5) * (s1 * (H_h - cun) + s5 * (H_h + cun) + al2 * (a23 * (T(0.5) * q2) + t4));
}

// 1/x, 1/sqrt(x) and sqrt(x) in FP64 for a normal, finite x (whose result is normal
// too), without the special cases of the general functions: the hardware's seed
// (relative error 1e-6, measured) and one step of Householder's iteration of the
// second order (A. S. Householder, The Numerical Treatment of a Single Nonlinear
// Equation, 1970): the series of 1/(1 - e) and 1/sqrt(1 - e) up to e^2, e the
// seed's residual, which the FMA gives without rounding (P. Markstein, IBM J. Res.
// Dev. 34(1), 1990).  The root takes one more such step from x times the reciprocal
// root.  Largest relative errors over 2^-1020 .. 2^1000 (4 million arguments), in
// units of 2^-53 (half a unit in the last place): rcp_normal 1.00, rsqrt_normal
// 1.25, sqrt_normal 1.00, held to 1.02, 2.05 and 1.02 by tests/test_gpu_f64_roots.py.
__device__ __forceinline__ double rcp_normal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// 1/x of any x: where the seed is no start for the step (0, infinities, NaN, a
// result below the normal range), the seed itself: inf, 0, NaN, 0.
__device__ __forceinline__ double rcp_any(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fabs(e) < 0.5 ? fma(y, fma(e, e, e), y) : y;
}
__device__ __forceinline__ double rsqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}
// r = rsqrt_normal(x).  x r = y + d exactly (but for d's last bit), and the step's
// residual is 1 - x r^2, which stays far from the subnormal range, as x - y^2 does
// not.
__device__ __forceinline__ double sqrt_normal(double x, double r) {
  const double y = x * r, d = fma(x, r, -y);
  const double e = fma(-d, r, fma(-y, r, 1.0));
  return y + fma(0.5 * y, e, d);
}

// Roe flux times |n| (flux/roe.py:21-85, rhs/invscd.py:87-100) in FP64, of the
// primitive face states and the unnormalised face normal n.  The FP64 kernels
// are bound by the FP64 pipe and by what each thread holds, so the same sums are
// grouped for the fewest operations:
//   * the dissipation's shear term t_m = (d_m - u_m d0) - dun n_m enters
//     linearly, so the five components of |A| dU are
//       A_0 = h + a2 d0,  A_m = h u_m + g n_m + a2 d_m,
//       A_4 = (s1 + s5) H + g un + a2 (u.d - q2/2 (d0 + dp/c2))
//     with h = s1 + s5 - a2 dp/c2 and g = c (s5 - s1) - a2 dun;
//   * |n| and 1/|n|, c and 1/c2, and sqrt(rhoR/rhoL) from one reciprocal square
//     root each; 1/rhoR and the Roe weight 1/(1 + t) from one reciprocal;
//   * the two fluxes through the face as it is (u . n with the unnormalised n), so
//     that |n| and 1/|n| are rounded into the dissipation only, which is small: the
//     inviscid right-hand side of a curvilinear block is 7.4e-15 off the exact one,
//     7.8e-15 to 8.0e-15 with both scaled by |n| (the reference's expressions in
//     plain FP64: 7.7e-15), at the same number of operations.
// FP64 step of four 128^3 blocks 5.27 -> 5.12 ms, of the 32^3 block 49.8 -> 48.2 us,
// both right-hand sides of a 131 x 70 x 55 block 126 -> 123 us.
__device__ __forceinline__ void roe_face_f64(const Prim<double>& L, const Prim<double>& R, double nx, double ny,
                                             double nz, double gm1, double inv_gm1, double eps_entropy, double F[5]) {
  const double n2 = nx * nx + ny * ny + nz * nz;
  const bool face = n2 > 2.3e-308;  // a zero (or subnormal) |n|^2 leaves no dissipation
  const double rn = face ? rsqrt_normal(n2) : 0.0;
  const double hn = 0.5 * (face ? n2 * rn : Tiny<double>::nmag());
  const double n0 = nx * rn, n1 = ny * rn, n2u = nz * rn;

  const double rhoL = fj_max(L.rho, Tiny<double>::rho()), rhoR = fj_max(R.rho, Tiny<double>::rho());
  const double eL = L.p * inv_gm1 + (0.5 * L.rho) * (L.u * L.u + L.v * L.v + L.w * L.w);
  const double eR = R.p * inv_gm1 + (0.5 * R.rho) * (R.u * R.u + R.v * R.v + R.w * R.w);
  const double epL = eL + L.p, epR = eR + R.p;
  // t = sqrt(rhoR / rhoL): wl = 1 / (1 + t), wr = t / (1 + t), rho_h = rhoL t
  const double irL = rcp_normal(rhoL);
  const double t2 = fj_max(rhoR * irL, Tiny<double>::rho());  // (a clamped density over a large one)
  const double t = t2 * rsqrt_normal(t2);
  const double ix = rcp_normal((1.0 + t) * rhoR);
  const double irR = ix * (1.0 + t), wl = ix * rhoR, wr = t * wl;
  const double u = wl * L.u + wr * R.u;
  const double v = wl * L.v + wr * R.v;
  const double w = wl * L.w + wr * R.w;
  const double H = wl * (epL * irL) + wr * (epR * irR);
  const double hq = 0.5 * (u * u + v * v + w * w);
  const double c2 = fj_max(gm1 * (H - hq), Tiny<double>::c2());
  const double ic = rsqrt_normal(c2);
  const double c = c2 * ic, ic2 = ic * ic;
  const double un = u * n0 + v * n1 + w * n2u;

  // Harten's fix (flux/roe.py:45-52) only where |lambda| < eps
  const double a2 = fabs(un);
  const double eps = eps_entropy * (a2 + c);
  double al1 = fabs(un - c), al5 = fabs(un + c);
  if (al1 < eps || al5 < eps) {
    const double inv_eps = __drcp_rn(eps);
    if (al1 < eps) al1 = 0.5 * (al1 * al1 * inv_eps + eps);
    if (al5 < eps) al5 = 0.5 * (al5 * al5 * inv_eps + eps);
  }

  const double d0 = R.rho - L.rho;
  const double d1 = R.rho * R.u - L.rho * L.u;
  const double d2 = R.rho * R.v - L.rho * L.v;
  const double d3 = R.rho * R.w - L.rho * L.w;
  const double ud = u * d1 + v * d2 + w * d3;
  const double dp = gm1 * ((eR - eL) - ud + hq * d0);
  const double dun = (d1 * n0 + d2 * n1 + d3 * n2u) - un * d0;
  const double rcd = rhoL * t * c * dun;
  const double hc2 = 0.5 * ic2;
  const double s1 = al1 * ((dp - rcd) * hc2), s5 = al5 * ((dp + rcd) * hc2);
  const double dpc = dp * ic2, sp = s1 + s5;
  const double h = sp - a2 * dpc, g = c * (s5 - s1) - a2 * dun;
  const double qL = L.u * nx + L.v * ny + L.w * nz, qR = R.u * nx + R.v * ny + R.w * nz;
  const double mL = rhoL * qL, mR = rhoR * qR, p2 = L.p + R.p;
  F[0] = 0.5 * (mL + mR) - hn * (h + a2 * d0);
  F[1] = 0.5 * (mL * L.u + mR * R.u + p2 * nx) - hn * (h * u + g * n0 + a2 * d1);
  F[2] = 0.5 * (mL * L.v + mR * R.v + p2 * ny) - hn * (h * v + g * n1 + a2 * d2);
  F[3] = 0.5 * (mL * L.w + mR * R.w + p2 * nz) - hn * (h * w + g * n2u + a2 * d3);
  F[4] = 0.5 * (qL * epL + qR * epR) - hn * (sp * H + g * un + a2 * (ud - hq * (d0 + dpc)));
}

// One inviscid face (rhs/invscd.py:62-100) in the reformulated arithmetic:
// MUSCL on the four cells' primitives, face normal from the two adjacent
// cells' kxyz rows, Roe, times |n|.
template <typename T, bool POFF = false>
__device__ __forceinline__ void invscd_face_fast(const Prim<T> c[4], T kl0, T kl1, T kl2, T kr0,
                                                 T kr1, T kr2, T gm1, T inv_gm1, T eps_entropy,
                                                 int limiter, T F[5], T p_ref = T(0)) {
  Prim<T> L, R;
  muscl2_fast(c, limiter, L, R);
  if constexpr (sizeof(T) == 8) {
    roe_face_f64(L, R, 0.5 * (kl0 + kr0), 0.5 * (kl1 + kr1), 0.5 * (kl2 + kr2), gm1, inv_gm1, eps_entropy, F);
  } else {
    const T nf0 = T(0.5) * (kl0 + kr0), nf1 = T(0.5) * (kl1 + kr1), nf2 = T(0.5) * (kl2 + kr2);
    const T nmag = FastMath<T>::sqrt_nn(nf0 * nf0 + nf1 * nf1 + nf2 * nf2) + Tiny<T>::nmag();
    const T inv = FastMath<T>::rcp_n(nmag);
    roe_prim<T, POFF>(L, R, nf0 * inv, nf1 * inv, nf2 * inv, gm1, inv_gm1, eps_entropy, F, p_ref);
#pragma unroll
    for (int v = 0; v < 5; ++v) F[v] = F[v] * nmag;
  }
}

// physics/eos.py:24-25 (or the constant law)
template <typename T>
__device__ __forceinline__ T viscosity(T Tt, int law, T mu0, T T0, T Ts) {
  if (law == 1) return mu0;
  const T r = Tt / T0;
  return mu0 * (r * fj_sqrt(r)) * (T0 + Ts) / (Tt + Ts);
}

}  // namespace fj
