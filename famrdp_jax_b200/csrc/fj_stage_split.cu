// fj_stage_split.cu -- one TVD-RK3 stage (or one RHS) of MANY blocks in three
// barrier-free, high-occupancy kernels, each launched once for all blocks:
//
//   k_split_prims    q -> primitives (rho, u, v, w, p, T) per padded cell
//                    (physics/eos.py:12-17; T = p / max(rho R, 1e-300),
//                    rhs/viscous.py:36); skipped where the producer of q left
//                    them (the previous stage's assembly, or the kernels that
//                    fill a step's start state)
//   k_split_fluxes   per cell c: the viscous flux components G(c)
//                    (rhs/viscous.py:36-105, neighbours wrap around the padded
//                    block like jnp.roll) and the Roe faces c | c+e_a of the
//                    axes i and j (rhs/invscd.py:53-100) for c_a in [1, n_a-3]
//   k_split_assemble per cell: the Roe faces along k (a lane's right face by
//                    shuffle), -(F_a(c) - F_a(c-e_a)) / (vol + 1e-300) over
//                    the axes where c_a in [2, n_a-3] (rhs/invscd.py:119-131),
//                    the viscous divergence of G with the cell's own kxyz
//                    (rhs/viscous.py:86-117) and the TVD-RK3 combine
//                    (solver/step.py:45-53)
//
// (fm:: for the FP64 path, whose face and viscous fluxes are field-major).  Small
// tables run a whole stage in one launch (fj_split_small.cuh).
//
// Intermediates live in scratch in the flux type.  On the FP32-flux path they are
// per-cell RECORDS, so that a cell's fields sit at compile-time offsets from one
// address and move with 16- and 32-byte vector loads and stores:
//   P  8 floats per cell: rho u v w p' T (2 pad)
//   F  8 floats per cell: the face c | c+e_i (5) and the first three of
//      c | c+e_j; the other two of c | c+e_j as a pair in an array of their own
//   G  8 floats per cell: tau_00 tau_01 tau_02 tau_11 tau_12 tau_22, the energy
//      flux components 0 and 1; component 2 in an array of its own
// A plan also keeps the metrics as records (kRecK<T> T per cell: the nine
// kxyz[l][m], l-major, then pad), converted once from the caller's FP64
// field-major kxyz; without one the kernels read kxyz field by field.
// Each launch covers every block of a table; a CTA handles 128 (assembly: 124)
// consecutive cells of one block, and neighbours are read through L1/L2.
#include <type_traits>

#include "fj_common.cuh"
#include "fj_physics.cuh"
#include "fj_rhs.cuh"
#include "fj_split.cuh"

#include "fj_split_dev.cuh"

namespace fj {

namespace {

using namespace sd;

template <typename T, int NW, class TB>
__global__ void __launch_bounds__(32 * NW) k_split_prims(const TB tab, const double gm1, const double R,
                                                         const double iR, const double p_ref) {
  const int b = find_block(tab, blockIdx.x);
  if (threadIdx.x == 0) prefetch_state(tab.b[b], blockIdx.x, 32 * NW);
  grid_dep_wait();
  const SplitBlock& B = tab.b[b].blk;
  const int32_t c = (blockIdx.x - B.cta_begin) * (32 * NW) + threadIdx.x;
  if (c >= B.ni * B.nj * B.nk) return;
  prims_cell<T>(B, c, gm1, R, iR, p_ref);
}

template <typename T, bool K_AOS, int OCC, int NT, class TB>
__global__ void __launch_bounds__(NT, OCC) k_split_fluxes(const TB tab, const Phys ph, const int flags) {
  const int b = find_block(tab, blockIdx.x);
  if (threadIdx.x == 0) prefetch_fluxes<T, K_AOS, false>(tab.b[b], blockIdx.x, NT);
  grid_dep_wait();
  Cell x;
  if (!decode_cell(tab.b[b], (int64_t)(blockIdx.x - tab.b[b].blk.cta_begin) * NT + threadIdx.x, x)) return;
  flux_cell<T, K_AOS, true>(tab.b[b].blk, tab.b[b].blk.prim, x, ph, flags);
}

template <typename T, bool K_AOS, int OCC, int NW, class TB>
__global__ void __launch_bounds__(32 * NW, OCC) k_split_assemble(const TB tab, const int flags, const int stage,
                                                                 const int next_prims, const double gm1,
                                                                 const double R, const double iR, const Phys ph) {
  const int b = find_block_asm(tab, blockIdx.x);
  const Dev& d = tab.b[b];
  const SplitBlock& B = d.blk;
  if (threadIdx.x == 0) prefetch_assembly<T, K_AOS, false>(d, blockIdx.x, flags, stage, 31 * NW, B.cta_begin_asm);
  grid_dep_wait();
  asm_chunk<T, K_AOS, true>(d, TablePtrs{B}, (int64_t)(blockIdx.x - B.cta_begin_asm) * (31 * NW), flags, stage,
                            next_prims, gm1, R, iR, ph);
}

// ---- field-major variant (the FP64 path) ----------------------------------
// The FP64 path keeps its primitives as 48-byte records (three 16-byte loads
// per neighbour) and its face and viscous fluxes field-major (10 + 9 arrays of
// N): flux records would cost FP64 more registers (two doubles per vector
// lane) and padding bytes than the index arithmetic they save.
namespace fm {

template <typename T, int NW, class TB>
__global__ void __launch_bounds__(32 * NW) k_fm_prims(const TB tab, const double gm1,
                                                              const double R, const double iR) {
  const int b = find_block(tab, blockIdx.x);
  if (threadIdx.x == 0) prefetch_state(tab.b[b], blockIdx.x, 32 * NW);
  grid_dep_wait();
  const SplitBlock& B = tab.b[b].blk;
  const int64_t N = (int64_t)B.ni * B.nj * B.nk;
  const int64_t c = (int64_t)(blockIdx.x - B.cta_begin) * (32 * NW) + threadIdx.x;
  if (c >= N) return;
  const double* q = B.q + c;
  const double qc[5] = {q[0], q[N], q[2 * N], q[3 * N], q[4 * N]};
  store_prim_record<T>(B.prim, (size_t)c, qc, gm1, R, iR, 0.0);
}

template <typename T>
__device__ __forceinline__ T metric(const SplitBlock& B, int64_t N, int lm, int64_t c) {
  return (T)__ldg(B.kxyz + lm * N + c);
}

// Primitives (rho, u, v, w, p[, T]) of one cell from the field-major scratch.
template <typename T>
struct Cell6 {
  T r, u, v, w, p, t;
};

// (values a caller does not use are not loaded: the loads are whole 16-byte pairs)
template <typename T>
__device__ __forceinline__ Cell6<T> load_cell(const T* __restrict__ P, int32_t c) {
  T x[kRecP64];
  ld_rec<T, kRecP64>(P + (size_t)c * kRecP64, x);
  return Cell6<T>{x[4], x[0], x[1], x[2], x[5], x[3]};
}

// Roe face c | c+e_a from the primitives of c-e_a, c, c+e_a, c+2e_a and the
// kxyz rows of c and c+e_a (rhs/invscd.py:62-100).
template <typename T>
__device__ __forceinline__ void face_from_cells(const Cell6<T>& a0, const Cell6<T>& a1, const Cell6<T>& a2,
                                                const Cell6<T>& a3, const T kl[3], const T kr[3],
                                                const Phys& ph, T F[5]) {
  Prim<T> cell[4] = {{a0.r, a0.u, a0.v, a0.w, a0.p}, {a1.r, a1.u, a1.v, a1.w, a1.p},
                     {a2.r, a2.u, a2.v, a2.w, a2.p}, {a3.r, a3.u, a3.v, a3.w, a3.p}};
  invscd_face_fast<T>(cell, kl[0], kl[1], kl[2], kr[0], kr[1], kr[2], (T)ph.gm1, (T)ph.inv_gm1,
                      (T)ph.eps_entropy, ph.limiter, F);
}

template <typename T>
__device__ __forceinline__ void metric_row(const SplitBlock& B, int32_t N, int row, int32_t c, T k[3]) {
  const double* K = B.kxyz + 3 * row * N + c * B.kstep;
  k[0] = (T)__ldg(K);
  k[1] = (T)__ldg(K + N);
  k[2] = (T)__ldg(K + 2 * N);
}

// The viscous flux components G(c) (rhs/viscous.py:36-105) from the primitives of c
// and its six neighbours and the metrics of c.
template <typename T>
__device__ __forceinline__ void visc_components(const SplitBlock& B, const Cell6<T>& C0, const Cell6<T>& Im,
                                                const Cell6<T>& Ip, const Cell6<T>& Jm, const Cell6<T>& Jp,
                                                const Cell6<T>& Km, const Cell6<T>& Kp, const T kk[9], const Phys& ph,
                                                T G[9]) {
  // the central differences' factor 1/2 is carried by mu and kappa (exact)
  const T d[4][3] = {{Ip.u - Im.u, Jp.u - Jm.u, Kp.u - Km.u},
                     {Ip.v - Im.v, Jp.v - Jm.v, Kp.v - Km.v},
                     {Ip.w - Im.w, Jp.w - Jm.w, Kp.w - Km.w},
                     {Ip.t - Im.t, Jp.t - Jm.t, Kp.t - Km.t}};
  T g[4][3];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int m = 0; m < 3; ++m) g[s][m] = d[s][0] * kk[m] + d[s][1] * kk[3 + m] + d[s][2] * kk[6 + m];
  T mu = (T)B.mu0;
  if (ph.visc_law == 0) {  // Sutherland (physics/eos.py:24-25)
    const T r = C0.t * (T)ph.inv_T0;
    mu = (T)B.mu0 * (r * FastMath<T>::sqrt_pos(r)) * (T)ph.sfac * FastMath<T>::rcp(C0.t + (T)ph.Ts);
  }
  const T muh = T(0.5) * mu, kappa = (T)ph.kap_fac * muh;
  const T third = (T)(1.0 / 3.0);
  const T div_u = g[0][0] + g[1][1] + g[2][2];
  const T t00 = mu * (g[0][0] - div_u * third);
  const T t01 = muh * (g[0][1] + g[1][0]);
  const T t02 = muh * (g[0][2] + g[2][0]);
  const T t11 = mu * (g[1][1] - div_u * third);
  const T t12 = muh * (g[1][2] + g[2][1]);
  const T t22 = mu * (g[2][2] - div_u * third);
  G[0] = t00;
  G[1] = t01;
  G[2] = t02;
  G[3] = t11;
  G[4] = t12;
  G[5] = t22;
  G[6] = C0.u * t00 + C0.v * t01 + C0.w * t02 + kappa * g[3][0];
  G[7] = C0.u * t01 + C0.v * t11 + C0.w * t12 + kappa * g[3][1];
  G[8] = C0.u * t02 + C0.v * t12 + C0.w * t22 + kappa * g[3][2];
}

// FL: the one kind of term that the kernel is compiled for, or 0: `flags_` at run
// time (a step's kernels; compiled for both terms they take the same time on 4.0 M
// cells).
template <typename T, int OCC, int NT, class TB, int FL>
__global__ void __launch_bounds__(NT, OCC) k_fm_fluxes(const TB tab, const Phys ph, const int flags_) {
  const int flags = FL ? FL : flags_;
  const int b = find_block(tab, blockIdx.x);
  if (threadIdx.x == 0) prefetch_fluxes<T, false, true>(tab.b[b], blockIdx.x, NT);
  grid_dep_wait();
  Cell x;
  const SplitBlock& B = tab.b[b].blk;
  if (!decode_cell(tab.b[b], (int64_t)(blockIdx.x - B.cta_begin) * NT + threadIdx.x, x)) return;
  // 32-bit offsets: 15 N < 2^31 is checked on the host
  const int32_t N = (int32_t)x.N, c = (int32_t)x.c;
  const int32_t si = x.nj * x.nk, sj = x.nk;
  const T* __restrict__ P = (const T*)B.prim;
  const bool vis = (flags & kRhsViscous) != 0, inv = (flags & kRhsInvscd) != 0;

  // neighbour offsets with the padded-array wrap (jnp.roll) for the viscous
  // stencil; faces exist only where no wrap is involved
  const int32_t ip = x.i + 1 == x.ni ? c - (x.ni - 1) * si : c + si;
  const int32_t im = x.i == 0 ? c + (x.ni - 1) * si : c - si;
  const int32_t jp = x.j + 1 == x.nj ? c - (x.nj - 1) * sj : c + sj;
  const int32_t jm = x.j == 0 ? c + (x.nj - 1) * sj : c - sj;
  const int32_t kp = x.k + 1 == x.nk ? c - (x.nk - 1) : c + 1;
  const int32_t km = x.k == 0 ? c + (x.nk - 1) : c - 1;

  const Cell6<T> C0 = load_cell<T>(P, c);
  const Cell6<T> Im = load_cell<T>(P, im), Ip = load_cell<T>(P, ip);
  const Cell6<T> Jm = load_cell<T>(P, jm), Jp = load_cell<T>(P, jp);
  const Cell6<T> Km = load_cell<T>(P, km), Kp = load_cell<T>(P, kp);

  if (vis) {
    T kk[9], g[9];
    metric_row<T>(B, N, 0, c, kk);
    metric_row<T>(B, N, 1, c, kk + 3);
    metric_row<T>(B, N, 2, c, kk + 6);
    visc_components(B, C0, Im, Ip, Jm, Jp, Km, Kp, kk, ph, g);
    T* __restrict__ G = (T*)B.G;
#pragma unroll
    for (int m = 0; m < 9; ++m) G[m * N + c] = g[m];
  }
  if (inv) {
    // the three faces c | c+e_a with face index c_a - 1 in [0, n_a - 4]
    T* __restrict__ F = (T*)B.F;
    T kc[3], kn[3], Fo[5];
    if (x.i >= 1 && x.i <= x.ni - 3) {
      const Cell6<T> I2 = load_cell<T>(P, c + 2 * si);
      metric_row<T>(B, N, 0, c, kc);
      metric_row<T>(B, N, 0, c + si, kn);
      face_from_cells<T>(Im, C0, Ip, I2, kc, kn, ph, Fo);
#pragma unroll
      for (int v = 0; v < 5; ++v) F[v * N + c] = Fo[v];
    }
    if (x.j >= 1 && x.j <= x.nj - 3) {
      const Cell6<T> J2 = load_cell<T>(P, c + 2 * sj);
      metric_row<T>(B, N, 1, c, kc);
      metric_row<T>(B, N, 1, c + sj, kn);
      face_from_cells<T>(Jm, C0, Jp, J2, kc, kn, ph, Fo);
#pragma unroll
      for (int v = 0; v < 5; ++v) F[(5 + v) * N + c] = Fo[v];
    }
    // the k faces are evaluated in the assembly (this kernel is bound by the
    // FP64 pipe, the assembly by memory latency)
  }
}

// The FP64 flux work of one cell in separate parts (k_small_stage), the same
// arithmetic as k_fm_fluxes and the k faces of k_fm_assemble.
template <typename T>
__device__ __forceinline__ void face_value(const SplitBlock& B, int32_t N, int axis, int32_t c, int32_t sa, int ia,
                                           int na, const Phys& ph, T F[5]) {
  const T* __restrict__ P = (const T*)B.prim;
#pragma unroll
  for (int v = 0; v < 5; ++v) F[v] = T(0);
  if (ia < 1 || ia > na - 3) return;
  const Cell6<T> a0 = load_cell<T>(P, c - sa), a1 = load_cell<T>(P, c), a2 = load_cell<T>(P, c + sa),
                 a3 = load_cell<T>(P, c + 2 * sa);
  T kc[3], kn[3];
  metric_row<T>(B, N, axis, c, kc);
  metric_row<T>(B, N, axis, c + sa, kn);
  face_from_cells<T>(a0, a1, a2, a3, kc, kn, ph, F);
}

template <typename T>
__device__ __forceinline__ void visc_value(const SplitBlock& B, const Cell& x, const Phys& ph, T G[9]) {
  const int32_t N = (int32_t)x.N, c = (int32_t)x.c;
  const int32_t si = x.nj * x.nk, sj = x.nk;
  const T* __restrict__ P = (const T*)B.prim;
  const int32_t ip = x.i + 1 == x.ni ? c - (x.ni - 1) * si : c + si;
  const int32_t im = x.i == 0 ? c + (x.ni - 1) * si : c - si;
  const int32_t jp = x.j + 1 == x.nj ? c - (x.nj - 1) * sj : c + sj;
  const int32_t jm = x.j == 0 ? c + (x.nj - 1) * sj : c - sj;
  const int32_t kp = x.k + 1 == x.nk ? c - (x.nk - 1) : c + 1;
  const int32_t km = x.k == 0 ? c + (x.nk - 1) : c - 1;
  const Cell6<T> C0 = load_cell<T>(P, c);
  const Cell6<T> Im = load_cell<T>(P, im), Ip = load_cell<T>(P, ip);
  const Cell6<T> Jm = load_cell<T>(P, jm), Jp = load_cell<T>(P, jp);
  const Cell6<T> Km = load_cell<T>(P, km), Kp = load_cell<T>(P, kp);
  T kk[9];
  metric_row<T>(B, N, 0, c, kk);
  metric_row<T>(B, N, 1, c, kk + 3);
  metric_row<T>(B, N, 2, c, kk + 6);
  visc_components(B, C0, Im, Ip, Jm, Jp, Km, Kp, kk, ph, G);
}

// The k face c-1 | c (rhs/invscd.py:62-100) of the FP64 path from the
// primitive records of c-2 .. c+1 and the k rows of kxyz at c-1 and c.
template <typename T>
__device__ __forceinline__ void fm_k_face_left(const SplitBlock& B, int32_t N, int32_t c, const Phys& ph, T F[5]) {
  const T* __restrict__ P = (const T*)B.prim;
  const Cell6<T> a0 = load_cell<T>(P, c - 2), a1 = load_cell<T>(P, c - 1),
                 a2 = load_cell<T>(P, c), a3 = load_cell<T>(P, c + 1);
  T kl[3], kr[3];
  metric_row<T>(B, N, 2, c - 1, kl);
  metric_row<T>(B, N, 2, c, kr);
  face_from_cells<T>(a0, a1, a2, a3, kl, kr, ph, F);
}

// Where the assembly of cell c finds its differences of face fluxes and viscous
// components: the scratch arrays (k faces given), or shared memory (k_small_stage).
template <typename T>
struct GlobalSrc {
  const T* F;  // at c
  const T* G;
  int32_t N, si, sj;
  const T* fl;
  const T* fr;
  // F(c) - F(c-e_a); a face that does not count is read at the cell itself
  __device__ __forceinline__ void faces(bool on_i, bool on_j, T di[5], T dj[5], T dk[5]) const {
    const T* __restrict__ Fi = F - (on_i ? si : 0);
    const T* __restrict__ Fj = F - (on_j ? sj : 0);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      di[v] = __ldg(F + v * N) - __ldg(Fi + v * N);
      dj[v] = __ldg(F + (5 + v) * N) - __ldg(Fj + (5 + v) * N);
      dk[v] = fr[v] - fl[v];
    }
  }
  // G(cp) - G(cm), the neighbours along axis l
  __device__ __forceinline__ void gdiff(int, int32_t cp, int32_t cm, T g[9]) const {
#pragma unroll
    for (int m = 0; m < 9; ++m) g[m] = __ldg(G + cp + m * N) - __ldg(G + cm + m * N);
  }
};

// The assembly of one cell (rhs/invscd.py:119-131, rhs/viscous.py:86-117,
// solver/step.py:45-53).
// Bound by the latency of its loads (about 100 values a cell, most from L2): what
// counts is how many times a thread waits, so the faces are one batch of loads
// and the viscous components one per axis, with nothing branched around (4.0 M
// cells: 369 -> 330 us against a branch per face and equation).
template <typename T, class Src>
__device__ __forceinline__ void assemble_inv(const SplitBlock& B, const Cell& x, const Src& src, double r[5]) {
  // every face value in one batch of loads: a face that does not count is read
  // at the cell itself and left out of the sum, not branched around
  const bool on_i = x.i >= 2 && x.i <= x.ni - 3, on_j = x.j >= 2 && x.j <= x.nj - 3, on_k = x.k >= 2 && x.k <= x.nk - 3;
  // (the caller's volumes may be anything: the general reciprocal, 0 of an infinite
  // volume; a cell with no face that counts keeps 0 whatever its volume is)
  const double neg_ivd = on_i || on_j || on_k ? -rcp_any(__ldg(B.vol + x.c) + 1e-300) : 0.0;
  T di[5], dj[5], dk[5];
  src.faces(on_i, on_j, di, dj, dk);
#pragma unroll
  for (int v = 0; v < 5; ++v)  // axis by axis like the reference
    r[v] = ((on_i ? di[v] : 0.0) + (on_j ? dj[v] : 0.0) + (on_k ? dk[v] : 0.0)) * neg_ivd;
}

// sum over l of 0.5 kxyz[l][jj] (G(c+e_l) - G(c-e_l)): the 18 components of an axis
// in one batch of loads
template <typename T, class Src>
__device__ __forceinline__ void assemble_visc(const SplitBlock& B, const Cell& x, const Src& src, T acc[4]) {
  const int32_t N = (int32_t)x.N, c = (int32_t)x.c;
  const int n[3] = {x.ni, x.nj, x.nk};
  const int idx[3] = {x.i, x.j, x.k};
  const int32_t st[3] = {x.nj * x.nk, x.nk, 1};
  const T* __restrict__ K = B.kxyz + c * B.kstep;
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = T(0);
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    T g[9];
    src.gdiff(l, idx[l] + 1 == n[l] ? c - (n[l] - 1) * st[l] : c + st[l],
              idx[l] == 0 ? c + (n[l] - 1) * st[l] : c - st[l], g);
    const T k0 = T(0.5) * __ldg(K + (3 * l) * N), k1 = T(0.5) * __ldg(K + (3 * l + 1) * N),
            k2 = T(0.5) * __ldg(K + (3 * l + 2) * N);
    acc[0] += g[0] * k0 + g[1] * k1 + g[2] * k2;
    acc[1] += g[1] * k0 + g[3] * k1 + g[4] * k2;
    acc[2] += g[2] * k0 + g[4] * k1 + g[5] * k2;
    acc[3] += g[6] * k0 + g[7] * k1 + g[8] * k2;
  }
}

template <typename T, class Src>
__device__ __forceinline__ void assemble_cell(const SplitBlock& B, const Cell& x, const Src& src, int flags, int stage,
                                              int next_prims, double gm1, double R, double iR) {
  double r[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (flags & kRhsInvscd) assemble_inv<T>(B, x, src, r);
  if (flags & kRhsViscous) {
    T acc[4];
    assemble_visc<T>(B, x, src, acc);
#pragma unroll
    for (int e = 0; e < 4; ++e) r[e + 1] = __dadd_rn(r[e + 1], acc[e]);  // (as in sd::assemble_cell)
  }
  sd::assemble_out<T>(B, TablePtrs{B}, x, stage, next_prims, gm1, R, iR, 0.0, r);
}

// Each warp assembles 31 consecutive cells; lane l evaluates the k face on the
// left of its cell and takes the one on its right from lane l+1 by shuffle
// (lane 31's cell is the next warp's first, for which it only supplies the
// face), as in the FP32 assembly.
template <typename T, int OCC, int NW, class TB, int FL>
__global__ void __launch_bounds__(32 * NW, OCC) k_fm_assemble(const TB tab, const int flags_, const int stage,
                                                              const int next_prims, const double gm1, const double R,
                                                              const double iR, const Phys ph) {
  const int flags = FL ? FL : flags_;
  const int b = find_block_asm(tab, blockIdx.x);
  const Dev& dv = tab.b[b];
  const SplitBlock& B = dv.blk;
  if (threadIdx.x == 0) prefetch_assembly<T, false, true>(dv, blockIdx.x, flags, stage, 31 * NW, B.cta_begin_asm);
  grid_dep_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Cell x;
  x.N = (int64_t)B.ni * B.nj * B.nk;
  x.c = (int64_t)(blockIdx.x - B.cta_begin_asm) * (31 * NW) + warp * 31 + lane;
  const bool alive = x.c < x.N;
  if (alive) {
    const uint32_t t1 = dv.dk.div((uint32_t)x.c);
    x.k = (int)((uint32_t)x.c - t1 * (uint32_t)B.nk);
    x.i = (int)dv.dj.div(t1);
    x.j = (int)(t1 - (uint32_t)x.i * (uint32_t)B.nj);
    x.ni = B.ni;
    x.nj = B.nj;
    x.nk = B.nk;
  }
  T fl[5] = {T(0), T(0), T(0), T(0), T(0)}, fr[5];
  // face c-1 | c exists for k-1 in [1, nk-3]
  if ((flags & kRhsInvscd) && alive && x.k >= 2 && x.k <= x.nk - 2)
    fm_k_face_left<T>(B, (int32_t)x.N, (int32_t)x.c, ph, fl);
#pragma unroll
  for (int v = 0; v < 5; ++v) fr[v] = __shfl_down_sync(0xffffffffu, fl[v], 1);
  if (lane == 31 || !alive) return;
  const GlobalSrc<T> src{(const T*)B.F + x.c, (const T*)B.G, (int32_t)x.N, x.nj * x.nk, x.nk, fl, fr};
  assemble_cell<T>(B, x, src, flags, stage, next_prims, gm1, R, iR);
}

}  // namespace fm

#include "fj_split_small.cuh"

// Record of cell c: the nine kxyz[l][m], then (FP32 records) the three
// gcl[m] = sum over the axes a with c_a in [2, n_a-3] of
// 0.5 (kxyz[a][m](c+e_a) - kxyz[a][m](c-e_a)), evaluated in FP64: the sum of
// the face-normal differences n_a(c) - n_a(c-e_a) the assembly multiplies by
// p_ref (rhs/invscd.py:87-89, 119-131).
template <typename T>
__global__ void k_metric_records(const double* __restrict__ kxyz, T* __restrict__ out, int ni, int nj, int nk) {
  const int64_t N = (int64_t)ni * nj * nk;
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= N) return;
  T rec[kRecK<T>];
#pragma unroll
  for (int lm = 0; lm < 9; ++lm) rec[lm] = (T)kxyz[lm * N + c];
#pragma unroll
  for (int lm = 9; lm < kRecK<T>; ++lm) rec[lm] = T(0);
  if (kRecK<T> >= 12) {
    const int k = (int)(c % nk), j = (int)((c / nk) % nj), i = (int)(c / ((int64_t)nk * nj));
    const int idx[3] = {i, j, k}, n[3] = {ni, nj, nk};
    const int64_t st[3] = {(int64_t)nj * nk, nk, 1};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double g = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (idx[a] >= 2 && idx[a] <= n[a] - 3)
          g += 0.5 * (kxyz[(3 * a + m) * N + c + st[a]] - kxyz[(3 * a + m) * N + c - st[a]]);
      if (9 + m < kRecK<T>) rec[9 + m] = (T)g;
    }
  }
  st_rec<T, kRecK<T>>(out + c * kRecK<T>, rec);
}

// flags[b] := 1 where a word of a field of block b differs from word % period of it
// (bits): n[b] words a field, fields blockIdx.y, strides a multiple of `period`, so
// that a thread compares with one word.  CTAs of a block whose flag is set have
// nothing to do.  A block that is not uniform mostly shows it anywhere: a first launch
// (`sample`) of one CTA a field looks at 32 places spread over the block, and the
// second, at all words, then ends at once.  (In one launch the CTAs of the first wave
// all store the flag, 4 ns each: 0.15 ms for the four 128^3 blocks of a wavy grid
// instead of 0.02; polling the flag as they go takes longer still.)
struct WordsTable {
  const unsigned long long* m[kMaxSplitBlocks];
  int64_t n[kMaxSplitBlocks];
};
constexpr int kWordThreads = 192;
__global__ void __launch_bounds__(kWordThreads) k_words_differ(const WordsTable tab, int sample, int period,
                                                               int* flags) {
  const int64_t n = tab.n[blockIdx.z];
  const unsigned long long* m = tab.m[blockIdx.z] + blockIdx.y * n;
  int* flag = flags + blockIdx.z;
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)flag)) return;
  const int lane = threadIdx.x & 31;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t step = sample ? max((int64_t)1, n / (32 * kWordThreads)) * kWordThreads : (int64_t)gridDim.x * blockDim.x;
  const unsigned long long ref = m[t0 % period];
  constexpr int kU = 4;  // words in flight
  for (int64_t t = t0; t - lane < n; t += kU * step) {
    bool differ = false;
#pragma unroll
    for (int u = 0; u < kU; ++u) differ |= t + u * step < n && m[t + u * step] != ref;
    if (__any_sync(0xffffffffu, differ)) {
      if (lane == 0) *flag = 1;
      return;
    }
  }
}

// Sum of (pressure) over a block, one partial per CTA (fixed grid, fixed
// summation order: the result does not depend on scheduling).
constexpr int kPsumCtas = 592, kPsumThreads = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  }
  return r;
}

__global__ void k_pressure_partial(const double* __restrict__ q, int64_t N, double gm1, double* __restrict__ part) {
  __shared__ double sh[32];
  double s = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N; c += (int64_t)gridDim.x * blockDim.x) {
    const double r = q[c], u = q[N + c] / r, v = q[2 * N + c] / r, w = q[3 * N + c] / r;
    s += gm1 * (q[4 * N + c] - r * (0.5 * (u * u + v * v + w * w)));
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void k_fold_sum(const double* __restrict__ part, int n, double* __restrict__ out) {
  __shared__ double sh[32];
  double s = 0.0;
  for (int t = threadIdx.x; t < n; t += blockDim.x) s += part[t];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *out = s;
}

// Launch shapes of the split kernels, selected per plan by the autotuner
// (index 0 is the default): the minimum resident CTAs per SM of the flux and
// assembly kernels, i.e. their register caps, for CTAs of 4 warps (8-warp CTAs
// at the same registers leave an SM idler between CTAs: 1.057 against 1.049 ms
// for an FP32 step of 4.0 M cells, 1.867 against 1.813 ms in FP64; 2-warp CTAs
// 1.33 and 1.81).  These are the FP32 record kernels' shapes; kSplitVariants64
// below are the FP64 kernels'.
struct SplitShape {
  int flux_occ, asm_occ;
};
constexpr int kWarps32 = 4;  // warps per CTA
constexpr SplitShape kSplitVariants[] = {{9, 8}, {8, 8}, {7, 8}, {6, 8}, {8, 6}, {4, 8}};
static_assert(sizeof(kSplitVariants) / sizeof(kSplitVariants[0]) == FJ_NUM_SPLIT_VARIANTS, "variant table");

// Launch shapes of the FP64 field-major kernels (the same variant index; FP64
// face arithmetic needs more registers at the same occupancy).
constexpr int kWarps64 = 4;
constexpr SplitShape kSplitVariants64[] = {{4, 5}, {4, 6}, {4, 4}, {5, 5}, {5, 6}, {3, 5}};
static_assert(sizeof(kSplitVariants64) / sizeof(kSplitVariants64[0]) == FJ_NUM_SPLIT_VARIANTS, "variant table");

// Shapes of the right-hand sides with one kind of term only.  Kernels compiled for
// both and branching on the flags kept the registers of both (128 and 96 a thread):
// too few warps to cover the viscous terms' loads.  Compiled for their own terms
// the viscous ones need 80 / 64 (inviscid 128 / 96, at the caps).  Viscous calls at {6, 8} and,
// in brackets, at the steps' {4, 5}, at {5, 8}, {6, 6} and {7, 8}: 70 x 50 x 40 cells
// 16.4 us (16.6, 16.6, 16.8, 16.9), 96^3 86.6 (90.6, 87.8, 91.2, 89.1), 160 x 97 x 61
// 95.5 (99.8, 97.9, 100.7, 98.0).  Inviscid calls at {4, 5} and at {5, 5}, {4, 4} and
// {4, 6}: 21.5 (22.6, 21.5, 22.0), 102.7 (104.9, 102.4, 103.1), 115.6 (118.9, 115.7,
// 115.4).
constexpr SplitShape kShape64Inv{4, 5}, kShape64Vis{6, 8};

template <int FLUX_OCC, int ASM_OCC, int FL, class TB>
void launch_pair64(const TB& tab, int ctas, int asm_ctas, const Phys& ph, int stage, int np, cudaStream_t st,
                   cudaEvent_t after_fluxes) {
  constexpr int nt = 32 * kWarps64;
  pdl_launch(fm::k_fm_fluxes<double, FLUX_OCC, nt, TB, FL>, ctas, nt, 0, st, tab, ph, kRhsInvscd | kRhsViscous);
  if (after_fluxes) cudaEventRecord(after_fluxes, st);
  pdl_launch(fm::k_fm_assemble<double, ASM_OCC, kWarps64, TB, FL>, asm_ctas, nt, 0, st, tab, kRhsInvscd | kRhsViscous,
             stage, np, ph.gm1, ph.R, 1.0 / ph.R, ph);
}

template <int V, class TB>
void launch_both64(const TB& tab, int ctas, int asm_ctas, const Phys& ph, int stage, int np, cudaStream_t st,
                   cudaEvent_t after_fluxes) {
  constexpr SplitShape sh = kSplitVariants64[V];
  launch_pair64<sh.flux_occ, sh.asm_occ, 0>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes);
}

template <typename T, bool K_AOS, int V, class TB>
void launch_pair(const TB& tab, int ctas, int asm_ctas, const Phys& ph, int flags, int stage, int np,
                 cudaStream_t st, cudaEvent_t after_fluxes) {
  constexpr SplitShape sh = kSplitVariants[V];
  constexpr int nt = 32 * kWarps32;
  pdl_launch(k_split_fluxes<T, K_AOS, sh.flux_occ, nt, TB>, ctas, nt, 0, st, tab, ph, flags);
  if (after_fluxes) cudaEventRecord(after_fluxes, st);
  pdl_launch(k_split_assemble<T, K_AOS, sh.asm_occ, kWarps32, TB>, asm_ctas, nt, 0, st, tab, flags, stage, np, ph.gm1,
             ph.R, 1.0 / ph.R, ph);
}

template <typename T, bool K_AOS, class TB>
int launch_tab(const TB& tab, int ctas, int asm_ctas, const Phys& ph, int flags, int stage, bool prims_ready,
               bool next_prims, int variant, cudaStream_t st, cudaEvent_t after_fluxes) {
  const int np = next_prims ? 1 : 0;
  if constexpr (sizeof(T) == 8) {
    if (!prims_ready)
      pdl_launch(fm::k_fm_prims<double, kWarps64, TB>, ctas, 32 * kWarps64, 0, st, tab, ph.gm1, ph.R, 1.0 / ph.R);
    if (flags == kRhsInvscd) {
      launch_pair64<kShape64Inv.flux_occ, kShape64Inv.asm_occ, kRhsInvscd>(tab, ctas, asm_ctas, ph, stage, np, st,
                                                                           after_fluxes);
      return prims_ready ? 2 : 3;
    }
    if (flags == kRhsViscous) {
      launch_pair64<kShape64Vis.flux_occ, kShape64Vis.asm_occ, kRhsViscous>(tab, ctas, asm_ctas, ph, stage, np, st,
                                                                            after_fluxes);
      return prims_ready ? 2 : 3;
    }
    switch (variant) {
      case 1: launch_both64<1>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes); break;
      case 2: launch_both64<2>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes); break;
      case 3: launch_both64<3>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes); break;
      case 4: launch_both64<4>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes); break;
      case 5: launch_both64<5>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes); break;
      default: launch_both64<0>(tab, ctas, asm_ctas, ph, stage, np, st, after_fluxes);
    }
  } else {
    if (!prims_ready)
      pdl_launch(k_split_prims<T, kWarps32, TB>, ctas, 32 * kWarps32, 0, st, tab, ph.gm1, ph.R, 1.0 / ph.R,
                 K_AOS ? ph.p_ref : 0.0);
    // without records (no plan) the kernels convert FP64 metrics and want the registers
    // of shape 1: a viscous right-hand side of 127 x 66 x 51 cells takes 30.4 us (shape
    // 0: 30.9), of 160 x 97 x 61 64.1 (66.0), the inviscid ones the same in both
    switch (K_AOS ? variant : 1) {
      case 1: launch_pair<T, K_AOS, 1>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes); break;
      case 2: launch_pair<T, K_AOS, 2>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes); break;
      case 3: launch_pair<T, K_AOS, 3>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes); break;
      case 4: launch_pair<T, K_AOS, 4>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes); break;
      case 5: launch_pair<T, K_AOS, 5>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes); break;
      default: launch_pair<T, K_AOS, 0>(tab, ctas, asm_ctas, ph, flags, stage, np, st, after_fluxes);
    }
  }
  return prims_ready ? 2 : 3;
}

// Raises the shared-memory limit of one instance of k_small_stage on the current
// device.  The limit belongs to the function on the device, which other contexts
// launch from other threads: it is always the largest box's, never this table's,
// so that nobody's setting refuses another's launch.  Once per context, device and
// instance (a call for each launch is host time in steps whose pace the host sets).
template <typename T, bool K_AOS, int NB>
int small_ready(fj_ctx* ctx) {
  constexpr unsigned bit = 1u << ((sizeof(T) == 4 ? 0 : 1) + (K_AOS ? 2 : 0) + (NB == 1 ? 0 : NB == kFewBlocks ? 4 : 8));
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && dev != ctx->small_device) {
    ctx->small_device = dev;
    ctx->small_ready = 0;
  }
  if (e == cudaSuccess && !(ctx->small_ready & bit)) {
    e = cudaFuncSetAttribute(small::k_small_stage<T, K_AOS, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             small::kMaxValues * (int)sizeof(T));
    if (e == cudaSuccess) ctx->small_ready |= bit;
  }
  return e == cudaSuccess ? FJ_OK : cuda_status(ctx, e, "small stage: shared memory attribute");
}

// A small table: the primitives (unless the producer of q left them), then the
// whole stage in one launch.  ctas: boxes (numbered by cta_begin_asm); prim_ctas:
// 128-cell ranges (by cta_begin).
template <typename T, bool K_AOS, int NB>
int launch_small(const SmallTableN<NB>& small_tab, int ctas, int prim_ctas, size_t smem, const Phys& ph, int flags, int stage,
                 bool prims_ready, bool next_prims, cudaStream_t st, cudaEvent_t after_fluxes) {
  using TB = TableN<NB>;
  const TB& tab = small_tab;
  if (!prims_ready) {
    if constexpr (sizeof(T) == 8)
      pdl_launch(fm::k_fm_prims<double, kWarps64, TB>, prim_ctas, 32 * kWarps64, 0, st, tab, ph.gm1, ph.R, 1.0 / ph.R);
    else
      pdl_launch(k_split_prims<T, kWarps32, TB>, prim_ctas, 32 * kWarps32, 0, st, tab, ph.gm1, ph.R, 1.0 / ph.R,
                 K_AOS ? ph.p_ref : 0.0);
  }
  pdl_launch(small::k_small_stage<T, K_AOS, NB>, ctas, 32 * small::kWarpsOf<T>, smem, st, small_tab, flags, stage, next_prims ? 1 : 0, ph.gm1, ph.R,
             1.0 / ph.R, ph);
  if (after_fluxes) cudaEventRecord(after_fluxes, st);
  return prims_ready ? 1 : 2;
}

template <typename T>
int launch_split(fj_ctx* ctx, const SplitBlock* blocks, int nblocks, const Phys& ph, int flags,
                 int stage, bool prims_ready, bool next_prims, int variant, cudaStream_t st,
                 cudaEvent_t after_fluxes) {
  const int sms = ctx->sms;
  for (int base = 0; base < nblocks; base += kMaxSplitBlocks) {
    Table tab;
    tab.n = std::min(kMaxSplitBlocks, nblocks - base);
    int64_t cells = 0;
    for (int t = 0; t < tab.n; ++t) cells += (int64_t)blocks[base + t].ni * blocks[base + t].nj * blocks[base + t].nk;
    // a small table runs in one launch if its boxes fit the SMs once
    Tile tiles[kMaxSplitBlocks];
    bool small_tab = cells <= small::kMaxCellsPerSm * (int64_t)sms;
    int boxes = 0;
    size_t smem = 0;
    for (int t = 0; t < tab.n && small_tab; ++t) {
      const SplitBlock& sb = blocks[base + t];
      const int64_t N = (int64_t)sb.ni * sb.nj * sb.nk;
      tab.b[t].blk.cta_begin_asm = boxes;
      boxes += small::cut(sb.ni, sb.nj, sb.nk, std::max(1, (int)(sms * N / cells)), tiles[t]);
      smem = std::max(smem, small::values(tiles[t]) * sizeof(T));
      small_tab = boxes <= sms;
    }
    constexpr int nw = sizeof(T) == 8 ? kWarps64 : kWarps32, fcells = 32 * nw, acells = 31 * nw;
    int ctas = 0, asm_ctas = 0;
    const bool k_aos = blocks[base].kaos != nullptr;
    for (int t = 0; t < tab.n; ++t) {
      const SplitBlock& sb = blocks[base + t];
      // the kernels index cells and records with 32-bit offsets
      if ((int64_t)kRecF * sb.ni * sb.nj * sb.nk > INT32_MAX)
        return set_err(ctx, FJ_ERR_INVALID_ARGUMENT, "block too large for the split pipeline");
      if ((sb.kaos != nullptr) != k_aos)
        return set_err(ctx, FJ_ERR_INVALID_ARGUMENT, "metric records on some blocks only");
      const int box0 = tab.b[t].blk.cta_begin_asm;
      tab.b[t].blk = sb;
      tab.b[t].blk.cta_begin = ctas;
      tab.b[t].blk.cta_begin_asm = small_tab ? box0 : asm_ctas;
      tab.b[t].dk.init((uint32_t)sb.nk);
      tab.b[t].dj.init((uint32_t)sb.nj);
      const int64_t N = (int64_t)sb.ni * sb.nj * sb.nk;
      ctas += (int)((N + fcells - 1) / fcells);
      asm_ctas += (int)((N + acells - 1) / acells);
    }
    if (k_aos && sizeof(T) == 8)
      return set_err(ctx, FJ_ERR_INVALID_ARGUMENT, "the FP64 split path reads kxyz directly");
    // the event marks the first chunk's flux launch
    cudaEvent_t ev = base == 0 ? after_fluxes : nullptr;
    auto launch = [&](auto nb, auto aos) {  // kernels launched, or -1 (the error is set)
      constexpr int NB = decltype(nb)::value;
      constexpr bool AOS = decltype(aos)::value;
      if (small_tab) {
        if (small_ready<T, AOS, NB>(ctx) != FJ_OK) return -1;
        SmallTableN<NB> t;
        t.n = tab.n;
        std::copy(tab.b, tab.b + tab.n, t.b);
        std::copy(tiles, tiles + tab.n, t.tile);
        return launch_small<T, AOS, NB>(t, boxes, ctas, smem, ph, flags, stage, prims_ready, next_prims, st, ev);
      }
      if constexpr (NB == kMaxSplitBlocks) {
        return launch_tab<T, AOS>(tab, ctas, asm_ctas, ph, flags, stage, prims_ready, next_prims, variant, st, ev);
      } else {
        TableN<NB> t;
        t.n = tab.n;
        std::copy(tab.b, tab.b + tab.n, t.b);
        return launch_tab<T, AOS>(t, ctas, asm_ctas, ph, flags, stage, prims_ready, next_prims, variant, st, ev);
      }
    };
    auto pick = [&](auto nb) {
      if constexpr (sizeof(T) == 4) {
        if (k_aos) return launch(nb, std::true_type());
      }
      return launch(nb, std::false_type());
    };
    const int launched = tab.n == 1             ? pick(std::integral_constant<int, 1>())
                         : tab.n <= kFewBlocks  ? pick(std::integral_constant<int, kFewBlocks>())
                                                : pick(std::integral_constant<int, kMaxSplitBlocks>());
    if (launched < 0) return FJ_ERR_CUDA;
    ctx->launches += launched;
    int s = launch_status(ctx, "split stage launch");
    if (s != FJ_OK) return s;
  }
  return FJ_OK;
}

}  // namespace

int split_metric_records(const double* kxyz, void* out, int ni, int nj, int nk, int precision, cudaStream_t st) {
  const int64_t N = (int64_t)ni * nj * nk;
  if (N <= 0) return FJ_OK;
  const int grid = (int)((N + 255) / 256);
  if (precision == FJ_PREC_F32FLUX)
    k_metric_records<float><<<grid, 256, 0, st>>>(kxyz, (float*)out, ni, nj, nk);
  else
    k_metric_records<double><<<grid, 256, 0, st>>>(kxyz, (double*)out, ni, nj, nk);
  return cudaGetLastError() == cudaSuccess ? FJ_OK : FJ_ERR_CUDA;
}

int split_metrics_differ(const void* const* records, const fj_block* blocks, int nblocks, int* flags, cudaStream_t st) {
  constexpr int nt = kWordThreads, per = kRecK<float> / 2;  // 8-byte words of an FP32 record
  static_assert(nt % per == 0, "a thread's words all have the same place in their record");
  for (int base = 0; base < nblocks; base += kMaxSplitBlocks) {
    WordsTable tab;
    const int nb = std::min(kMaxSplitBlocks, nblocks - base);
    int64_t most = 0;
    for (int b = 0; b < nb; ++b) {
      const fj_block& B = blocks[base + b];
      const int64_t N = (int64_t)B.ni * B.nj * B.nk;
      tab.m[b] = (const unsigned long long*)(records ? records[base + b] : B.kxyz);
      tab.n[b] = records ? N * per : N;
      most = std::max(most, tab.n[b]);
    }
    const unsigned ctas = (unsigned)std::min<int64_t>((most + nt - 1) / nt, records ? 148 * 10 : 148 * 2);
    const unsigned fields = records ? 1 : 9, step = records ? per : 1;
    k_words_differ<<<dim3(1, fields, nb), nt, 0, st>>>(tab, 1, step, flags + base);
    k_words_differ<<<dim3(ctas, fields, nb), nt, 0, st>>>(tab, 0, step, flags + base);
  }
  return cudaGetLastError() == cudaSuccess ? FJ_OK : FJ_ERR_CUDA;
}

size_t mean_pressure_scratch_bytes(int nblocks) { return ((size_t)kPsumCtas * nblocks + 1) * sizeof(double); }

int mean_pressure(const fj_block* blocks, int nblocks, double gm1, double* scratch, cudaStream_t st, double* out) {
  double* part = scratch;
  const size_t n = (size_t)kPsumCtas * nblocks;
  int64_t cells = 0;
  for (int b = 0; b < nblocks; ++b) {
    const int64_t N = (int64_t)blocks[b].ni * blocks[b].nj * blocks[b].nk;
    cells += N;
    k_pressure_partial<<<kPsumCtas, kPsumThreads, 0, st>>>(blocks[b].q, N, gm1, part + (size_t)b * kPsumCtas);
  }
  k_fold_sum<<<1, 1024, 0, st>>>(part, (int)n, part + n);
  double h = 0.0;
  cudaError_t e = cudaMemcpyAsync(&h, part + n, sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess || cudaGetLastError() != cudaSuccess) return FJ_ERR_CUDA;
  *out = cells > 0 ? h / (double)cells : 0.0;
  return FJ_OK;
}

size_t split_metric_record_bytes(int precision, int64_t N) {
  return precision == FJ_PREC_F32FLUX ? (size_t)N * kRecK<float> * sizeof(float)
                                      : (size_t)N * kRecK<double> * sizeof(double);
}

// Values per cell of each intermediate: records (FP32-flux) or field-major
// arrays (FP64).
static void split_counts(int precision, int& nP, int& nF, int& nG) {
  const bool rec = precision == FJ_PREC_F32FLUX;
  // the stage input's primitives and the next stage's: the assembly reads the
  // first (its k faces) while writing the second
  nP = rec ? 2 * kRecP : 2 * kRecP64;
  // the i and j faces: records (FP32), field-major (FP64); the k faces stay in
  // the assembly
  nF = rec ? kRecFA + kRecFB : 10;
  nG = 9;  // records: kRecG per cell in G, then one per cell in Gz
}

size_t split_scratch_bytes(int precision, int64_t cells) {
  const size_t t = precision == FJ_PREC_F32FLUX ? sizeof(float) : sizeof(double);
  int nP, nF, nG;
  split_counts(precision, nP, nF, nG);
  return (size_t)(nP + nF + nG) * (size_t)cells * t + 3 * 256;
}

void split_assign_scratch(int precision, SplitBlock* blocks, int nblocks, void* scratch) {
  const size_t t = precision == FJ_PREC_F32FLUX ? sizeof(float) : sizeof(double);
  int nP, nF, nG;
  split_counts(precision, nP, nF, nG);
  char* p = (char*)scratch;
  auto al = [](char* x) { return (char*)(((uintptr_t)x + 255) & ~(uintptr_t)255); };
  int64_t total = 0;
  for (int b = 0; b < nblocks; ++b) total += (int64_t)blocks[b].ni * blocks[b].nj * blocks[b].nk;
  char* prim = al(p);
  char* F = al(prim + nP * total * t);
  char* G = al(F + nF * total * t);
  int64_t off = 0;
  for (int b = 0; b < nblocks; ++b) {
    const int64_t N = (int64_t)blocks[b].ni * blocks[b].nj * blocks[b].nk;
    // records are multiples of 16 bytes: [input | next] primitive records
    const int rp = precision == FJ_PREC_F32FLUX ? kRecP : kRecP64;
    blocks[b].prim = prim + rp * off * t;
    blocks[b].prim_next = prim + (rp * total + rp * off) * t;
    if (precision == FJ_PREC_F32FLUX) {
      blocks[b].F = F + kRecFA * off * t;
      blocks[b].Fz = F + (kRecFA * total + kRecFB * off) * t;
    } else {
      blocks[b].F = F + nF * off * t;
      blocks[b].Fz = nullptr;
    }
    if (precision == FJ_PREC_F32FLUX) {
      blocks[b].G = G + kRecG * off * t;
      blocks[b].Gz = G + (kRecG * total + off) * t;
    } else {
      blocks[b].G = G + nG * off * t;
      blocks[b].Gz = nullptr;
    }
    off += N;
  }
}

int split_stage(fj_ctx* ctx, const SplitBlock* blocks, int nblocks, const Phys& ph, int flags,
                int stage, int precision, cudaStream_t st, bool prims_ready, bool next_prims, int variant,
                cudaEvent_t after_fluxes) {
  if (next_prims && (stage < 1 || stage > 2)) return set_err(ctx, FJ_ERR_INVALID_ARGUMENT, "next_prims needs stage 1 or 2");
  if (variant < 0 || variant >= FJ_NUM_SPLIT_VARIANTS) return set_err(ctx, FJ_ERR_INVALID_ARGUMENT, "unknown variant");
  if (precision == FJ_PREC_F32FLUX)
    return launch_split<float>(ctx, blocks, nblocks, ph, flags, stage, prims_ready, next_prims, variant, st,
                               after_fluxes);
  return launch_split<double>(ctx, blocks, nblocks, ph, flags, stage, prims_ready, next_prims, variant, st,
                              after_fluxes);
}

}  // namespace fj
