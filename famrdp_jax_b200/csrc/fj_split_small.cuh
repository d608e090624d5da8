// fj_split_small.cuh -- one stage (or RHS) of a SMALL table in one launch, every
// intermediate in shared memory.  Included by fj_stage_split.cu.
//
// A small table is bound by latency: by the launches and by each thread's chain of
// loads and arithmetic, not by bandwidth.  Each CTA takes a box of cells of one
// block; its warps first evaluate the box's i, j and k faces and the viscous
// components of the box and its six-neighbour rim (32 values of one kind a warp
// and turn), then, after one barrier, assemble the cells.  The rim's components and
// the faces between boxes are evaluated by both neighbours (about 1.4 times the
// work of the two-kernel stage at 36^3 cells), which costs less than the second
// launch and the trip through L2.  The arithmetic is the split kernels' (the same
// bits).
// Steps (graph replays; FP32, FP64) against the two-kernel stages, of blocks of
// 20^3 interior cells 30.8 -> 22.6 us, 31.6 -> 26.7; 28^3 31.4 -> 28.8, 37.0 -> 34.9;
// 32^3 32.9 -> 30.8, 41.0 -> 39.0; from 36^3 on (432 padded cells an SM) the two
// kernels are faster (34.9 against 39.0, 43.3 against 51.5).  Submitting a step takes
// 4 launches instead of 7.
#pragma once

namespace small {

// A table is small up to this many cells an SM, if its boxes fit the SMs once.  30
// blocks (cubes and long ones), a step with two kernels a stage over a step with one:
// 11 from 90 to 320 cells an SM 0.96 to 1.36 in FP32 (mean 1.09) and 0.95 to 1.18 in
// FP64 (1.04); 9 from 330 to 360 0.95 to 1.06 (1.00) and 0.88 to 1.04 (0.95); 10 from
// 360 to 432 0.85 to 0.99 and 0.74 to 0.92.
constexpr int kMaxCellsPerSm = 320;
// Warps per CTA (one CTA per SM; FP32 at 96 registers a thread, FP64 at 128): 16 to
// 30 measured alike in FP32, 16 and 20 in FP64 (24 spill).
template <typename T>
constexpr int kWarpsOf = sizeof(T) == 4 ? 20 : 16;
// Largest box extents: bounds the shared memory (FP64 205 KB).
constexpr int kMaxI = 7, kMaxJ = 6, kMaxK = 18;

inline int pieces(int n, int most) { return (n + most - 1) / most; }

// Boxes of a block: k and j cut evenly into at most kMaxK and kMaxJ, i into as
// many pieces as keep the block's share `ctas` of the SMs busy once.  Returns the
// number of boxes.
inline int cut(int ni, int nj, int nk, int ctas, sd::Tile& T) {
  const int pk = pieces(nk, kMaxK), pj = pieces(nj, kMaxJ);
  T.t[2] = pieces(nk, pk);
  T.t[1] = pieces(nj, pj);
  const int want = std::max(1, std::min(ctas / (pj * pk), (ni + 1) / 2));
  T.t[0] = std::min(pieces(ni, want), kMaxI);
  T.pk.init((uint32_t)pieces(nk, T.t[2]));
  T.pj.init((uint32_t)pieces(nj, T.t[1]));
  T.tk.init((uint32_t)T.t[2]);
  T.tj.init((uint32_t)T.t[1]);
  T.tk1.init((uint32_t)T.t[2] + 1);
  T.tj1.init((uint32_t)T.t[1] + 1);
  return pieces(ni, T.t[0]) * pieces(nj, T.t[1]) * pieces(nk, T.t[2]);
}

// Values of type T in the shared memory of a box: nine components of the box with
// its rim, five of each face.
inline size_t values(const sd::Tile& T) {
  const int a = T.t[0], b = T.t[1], c = T.t[2];
  return 9 * (size_t)((a + 2) * (b + 2) * (c + 2)) + 5 * (size_t)((a + 1) * b * c + a * (b + 1) * c + a * b * (c + 1));
}

// The same for the largest box: every launch may use this much.
constexpr int kMaxValues = 9 * (kMaxI + 2) * (kMaxJ + 2) * (kMaxK + 2) +
                           5 * ((kMaxI + 1) * kMaxJ * kMaxK + kMaxI * (kMaxJ + 1) * kMaxK + kMaxI * kMaxJ * (kMaxK + 1));
static_assert(kMaxValues * sizeof(double) <= 227 * 1024, "shared memory of a CTA");

// The assembly's view of the shared memory: the slots of one cell.
template <typename T>
struct BoxSrc {
  const T* G;         // at the cell, component stride gn
  const T* f[3];      // the faces on the cell's low side, component stride nf[a]
  int gn, gs[3], nf[3], fs[3];  // slot steps to the next cell along each axis
  __device__ __forceinline__ T lo(int a, int v) const { return f[a][v * nf[a]]; }
  __device__ __forceinline__ T hi(int a, int v) const { return f[a][v * nf[a] + fs[a]]; }
  // sd::assemble_cell (FP32)
  __device__ __forceinline__ void F_rec(int32_t, T* o) const {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      o[v] = hi(0, v);
      o[5 + v] = hi(1, v);
    }
  }
  __device__ __forceinline__ void F_axis(int32_t, int a, T* o) const {
#pragma unroll
    for (int v = 0; v < 5; ++v) o[v] = lo(a, v);
  }
  __device__ __forceinline__ void G_nb(int l, int side, int32_t, T* o) const {
#pragma unroll
    for (int m = 0; m < 9; ++m) o[m] = G[m * gn + (side == 0 ? gs[l] : -gs[l])];
  }
  // fm::assemble_cell (FP64)
  __device__ __forceinline__ void faces(bool, bool, T di[5], T dj[5], T dk[5]) const {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      di[v] = hi(0, v) - lo(0, v);
      dj[v] = hi(1, v) - lo(1, v);
      dk[v] = hi(2, v) - lo(2, v);
    }
  }
  __device__ __forceinline__ void gdiff(int l, int32_t, int32_t, T g[9]) const {
#pragma unroll
    for (int m = 0; m < 9; ++m) g[m] = G[m * gn + gs[l]] - G[m * gn - gs[l]];
  }
};

template <typename T, bool K_AOS, int NB>
__global__ void __launch_bounds__(32 * kWarpsOf<T>, 1)
    k_small_stage(const SmallTableN<NB> tab, const int flags, const int stage, const int next_prims, const double gm1,
                  const double R, const double iR, const Phys ph) {
  constexpr int kWarps = kWarpsOf<T>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int blk = find_block_asm(static_cast<const TableN<NB>&>(tab), blockIdx.x);
  const SplitBlock& B = tab.b[blk].blk;
  const Tile& S = tab.tile[blk];
  const int ti = S.t[0], tj = S.t[1], tk = S.t[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ni = B.ni, nj = B.nj, nk = B.nk;
  const int32_t sj = nk, si = nj * nk, N = ni * si;
  // the box: cells (i0 .. , j0 .. , k0 .. ), clipped by the block
  const uint32_t cta = blockIdx.x - B.cta_begin_asm;
  const uint32_t t1 = S.pk.div(cta), t2 = S.pj.div(t1);
  const int k0 = (int)(cta - t1 * S.pk.d) * tk, j0 = (int)(t1 - t2 * S.pj.d) * tj, i0 = (int)t2 * ti;
  // slots
  const int gsj = tk + 2, gsi = (tj + 2) * gsj, gn = (ti + 2) * gsi;
  const int nI = (ti + 1) * tj * tk, nJ = ti * (tj + 1) * tk, nK = ti * tj * (tk + 1);
  T* const G = reinterpret_cast<T*>(smem);
  T* const FI = G + 9 * gn;
  T* const FJ = FI + 5 * nI;
  T* const FK = FJ + 5 * nJ;
  const bool inv = (flags & kRhsInvscd) != 0, vis = (flags & kRhsViscous) != 0;
  const int box = ti * tj * tk, ri = tj * tk, rj = ti * tk, rk = ti * tj;  // cells of the box and of its sides
  const int wI = inv ? (nI + 31) / 32 : 0, wJ = inv ? (nJ + 31) / 32 : 0, wK = inv ? (nK + 31) / 32 : 0;
  const int wG = vis ? (box + 2 * (ri + rj + rk) + 31) / 32 : 0;
  grid_dep_wait();

  for (int w = warp; w < wI + wJ + wK + wG; w += kWarps) {
    int u = w;
    if (u < wI + wJ + wK) {
      // a face on the low side of cell (i, j, k) along `axis`: the axes share one
      // copy of the face code (a small launch fetches its instructions cold)
      int axis, t, i, j, k, nf;
      T* o;
      if (u < wI) {
        t = u * 32 + lane;
        const int m = (int)S.tk.div((uint32_t)t), a = (int)S.tj.div((uint32_t)m);
        axis = 0, nf = nI, o = FI, i = i0 + a, j = j0 + m - a * tj, k = k0 + t - m * tk;
      } else if (u < wI + wJ) {
        t = (u - wI) * 32 + lane;
        const int m = (int)S.tk.div((uint32_t)t), a = (int)S.tj1.div((uint32_t)m);
        axis = 1, nf = nJ, o = FJ, i = i0 + a, j = j0 + m - a * (tj + 1), k = k0 + t - m * tk;
      } else {
        t = (u - wI - wJ) * 32 + lane;
        const int m = (int)S.tk1.div((uint32_t)t), a = (int)S.tj.div((uint32_t)m);
        axis = 2, nf = nK, o = FK, i = i0 + a, j = j0 + m - a * tj, k = k0 + t - m * (tk + 1);
      }
      const int32_t sa = axis == 0 ? si : (axis == 1 ? sj : 1);
      const int ia = (axis == 0 ? i : (axis == 1 ? j : k)) - 1, na = axis == 0 ? ni : (axis == 1 ? nj : nk);
      if (t >= nf || i >= ni || j >= nj || k >= nk) continue;
      T F[5];
      const int32_t c = i * si + j * sj + k - sa;
      if constexpr (sizeof(T) == 8)
        fm::face_value<T>(B, N, axis, c, sa, ia, na, ph, F);
      else
        sd::face_value<T, K_AOS>(B, B.prim, N, axis, c, sa, ia, na, ph, F);
#pragma unroll
      for (int v = 0; v < 5; ++v) o[v * nf + t] = F[v];
    } else {
      // viscous components: the box, then its six sides
      u -= wI + wJ;
      int t = (u - wK) * 32 + lane, a, b, c;
      if (t < box) {
        const int m = (int)S.tk.div((uint32_t)t);
        c = t - m * tk;
        a = (int)S.tj.div((uint32_t)m);
        b = m - a * tj;
      } else if ((t -= box) < 2 * ri) {
        a = t < ri ? -1 : ti;
        t = t < ri ? t : t - ri;
        b = (int)S.tk.div((uint32_t)t);
        c = t - b * tk;
      } else if ((t -= 2 * ri) < 2 * rj) {
        b = t < rj ? -1 : tj;
        t = t < rj ? t : t - rj;
        a = (int)S.tk.div((uint32_t)t);
        c = t - a * tk;
      } else if ((t -= 2 * rj) < 2 * rk) {
        c = t < rk ? -1 : tk;
        t = t < rk ? t : t - rk;
        a = (int)S.tj.div((uint32_t)t);
        b = t - a * tj;
      } else {
        continue;
      }
      // the padded array wraps around (jnp.roll); past the cell after the last
      // one there is nothing a cell of the box reads
      Cell x;
      x.i = i0 + a;
      x.j = j0 + b;
      x.k = k0 + c;
      if (x.i > ni || x.j > nj || x.k > nk) continue;
      x.i = x.i < 0 ? ni - 1 : (x.i == ni ? 0 : x.i);
      x.j = x.j < 0 ? nj - 1 : (x.j == nj ? 0 : x.j);
      x.k = x.k < 0 ? nk - 1 : (x.k == nk ? 0 : x.k);
      x.ni = ni;
      x.nj = nj;
      x.nk = nk;
      x.N = N;
      x.c = x.i * si + x.j * sj + x.k;
      T g[9];
      if constexpr (sizeof(T) == 8)
        fm::visc_value<T>(B, x, ph, g);
      else
        sd::visc_value<T, K_AOS>(B, B.prim, x, ph, g);
      T* o = G + (a + 1) * gsi + (b + 1) * gsj + c + 1;
#pragma unroll
      for (int m = 0; m < 9; ++m) o[m * gn] = g[m];
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < box; t += 32 * kWarps) {
    const int m = (int)S.tk.div((uint32_t)t), a = (int)S.tj.div((uint32_t)m);
    const int b = m - a * tj, c = t - m * tk;
    Cell x;
    x.i = i0 + a;
    x.j = j0 + b;
    x.k = k0 + c;
    if (x.i >= ni || x.j >= nj || x.k >= nk) continue;
    x.ni = ni;
    x.nj = nj;
    x.nk = nk;
    x.N = N;
    x.c = x.i * si + x.j * sj + x.k;
    BoxSrc<T> src;
    src.G = G + (a + 1) * gsi + (b + 1) * gsj + c + 1;
    src.gn = gn;
    src.gs[0] = gsi;
    src.gs[1] = gsj;
    src.gs[2] = 1;
    src.f[0] = FI + t;
    src.f[1] = FJ + (a * (tj + 1) + b) * tk + c;
    src.f[2] = FK + m * (tk + 1) + c;
    src.nf[0] = nI;
    src.nf[1] = nJ;
    src.nf[2] = nK;
    src.fs[0] = ri;
    src.fs[1] = tk;
    src.fs[2] = 1;
    if constexpr (sizeof(T) == 8) {
      fm::assemble_cell<T>(B, x, src, flags, stage, next_prims, gm1, R, iR);
    } else {
      T kk[9], gcl[3] = {T(0), T(0), T(0)}, fl[5], fr[5];
      sd::metric9<T, K_AOS>(B, N, (int32_t)x.c, kk, K_AOS ? gcl : nullptr);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        fl[v] = inv ? src.lo(2, v) : T(0);
        fr[v] = inv ? src.hi(2, v) : T(0);
      }
      sd::assemble_cell<T, K_AOS>(B, TablePtrs{B}, x, src, flags, stage, next_prims, gm1, R, iR,
                                  K_AOS ? ph.p_ref : 0.0, fl, fr, kk, gcl);
    }
  }
}

}  // namespace small
