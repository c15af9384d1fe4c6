// libaq.so: hand-written adjoint of the MLS-MPM substep with segment
// checkpointing, for the quantization sensitivities of the reference's
// autodiff pass (MPMSolver.run_forward_with_ad_nlogn, mpm_exps/engine/
// mpm_solver.py:1093-1302; Taichi's generated p2g.grad / grid_op.grad /
// g2p.grad, taichi_submission/taichi/transforms/auto_diff.cpp).
//
// State: n x NS unquantized values per particle in the record slot order
// x(d), v(d), C(d*d), F(d*d) | J; one material (fluid, or the reference's
// elastic law).  Forward substep s -> s' (same formulas as k_step):
//   P2G  m_i  = sum_p w_ip m,   P_i = sum_p w_ip (m v_p + A_p dpos_ip),
//        A_p = k sigma(F_p) + m C_p,  k = -dt p_vol 4/dx^2,
//        dpos_ip = x_i - x_p,  w_ip = prod_d N(x_pd/dx - i_d)
//   grid v_i = P_i / (m_i + 1e-10) - dt g e_y, then wall masks per component
//   G2P  v'_p = sum_i w_ip v_i,  C'_p = 4/dx^2 sum_i w_ip v_i dpos_ip^T,
//        x'_p = x_p + dt v'_p,  F'_p = (I + dt C'_p) F_p  (J'_p = (1+dt tr C'_p) J_p)
// Reverse (bars are adjoints), per substep:
//   G2P^T   Fbar += (I+dt C')^T F'bar;  C'bar += dt F'bar F^T;
//           v'bar += dt x'bar;  xbar += x'bar;
//           vbar_i += w v'bar + (4/dx^2) w C'bar dpos;
//           wbar_ip = v_i.v'bar + (4/dx^2) v_i^T C'bar dpos;
//           xbar -= (4/dx^2) w C'bar^T v_i  (through dpos);  xbar += wbar grad_x w
//   grid^T  masked components get no gradient; Pbar = vbar/(m+eps),
//           mbar = -vbar.P/(m+eps)^2
//   P2G^T   vbar += w m Pbar_i;  Abar += w Pbar_i dpos^T;
//           wbar = m mbar_i + Pbar_i.(m v + A dpos);  xbar -= w A^T Pbar_i;
//           xbar += wbar grad_x w;  Cbar += m Abar;  sigma_bar = k Abar;
//           Fbar += dsigma/dF^T sigma_bar  (fluid: Jbar += la tr(sigma_bar);
//           2D: fixed-corotated with the closed-form rotation derivative;
//           3D reference law: mu (sbar + sbar^T) F + la sum(sbar) F^-T)
// The derivative of the B-spline base index is zero almost everywhere.
//
// Sensitivities: sens[s] = sum over substeps t = 1..T-1 and particles of
// (dL/d state_t[s])^2 in f64, the quantity accu_grad accumulates
// (mpm_solver.py:1232-1271; the initial and the final state are not
// accumulated there either, :1190-1196).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cub/device/device_radix_sort.cuh>
#include <new>
#include <vector>

#include "aq_common.cuh"
#include "aq_kernels.cuh"

namespace aq {

template <class R>
struct AdK {
  int res[3], mat;
  R inv_dx, dx, dt, p_mass, kst, four_inv_dx2, grav, mu, lam;
  int wlo[3], whi[3];  // walls: node indices below wlo / above whi
  // rotating SDF collider (3D; col_on = 0: none), the fields collider_at
  // reads; pose is this substep's angle and height
  int col_on, col_n, col_dims[3], col_off[3], col_lo[3], col_hi[3];
  const float* col_sdf;
  const float* col_nrm;
  R col_omega;
  ColPose<R> pose;
};

template <int D>
__device__ __forceinline__ int64_t ad_cell(const int (&res)[3], const int* I) {
  return D == 3 ? ((int64_t)I[0] * res[1] + I[1]) * res[2] + I[2] : (int64_t)I[0] * res[1] + I[1];
}

template <int D, class R>
__device__ __forceinline__ void ad_weights(const R* x, const AdK<R>& K, int (&base)[3], R (&fx)[3], R (&w)[3][3]) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    R t = x[d] * K.inv_dx - (R)0.5;
    int b = (int)floor(t);
    b = min(max(b, 0), K.res[d] - 3);
    base[d] = b;
    fx[d] = x[d] * K.inv_dx - (R)b;
    w[0][d] = (R)0.5 * ((R)1.5 - fx[d]) * ((R)1.5 - fx[d]);
    w[1][d] = (R)0.75 - (fx[d] - (R)1) * (fx[d] - (R)1);
    w[2][d] = (R)0.5 * (fx[d] - (R)0.5) * (fx[d] - (R)0.5);
  }
}

// dN/dx per unit x
template <int D, class R>
__device__ __forceinline__ void ad_dweights(const AdK<R>& K, const R (&fx)[3], R (&dw)[3][3]) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    dw[0][d] = -((R)1.5 - fx[d]) * K.inv_dx;
    dw[1][d] = (R)-2 * (fx[d] - (R)1) * K.inv_dx;
    dw[2][d] = (fx[d] - (R)0.5) * K.inv_dx;
  }
}

template <int D, class R>
__device__ __forceinline__ R inv_det_cof(const R* F, R* cof) {  // cofactor matrix (dJ/dF) and J
  if (D == 2) {
    cof[0] = F[3];
    cof[1] = -F[2];
    cof[2] = -F[1];
    cof[3] = F[0];
    return F[0] * F[3] - F[1] * F[2];
  }
  cof[0] = F[4] * F[8] - F[5] * F[7];
  cof[1] = F[5] * F[6] - F[3] * F[8];
  cof[2] = F[3] * F[7] - F[4] * F[6];
  cof[3] = F[2] * F[7] - F[1] * F[8];
  cof[4] = F[0] * F[8] - F[2] * F[6];
  cof[5] = F[1] * F[6] - F[0] * F[7];
  cof[6] = F[1] * F[5] - F[2] * F[4];
  cof[7] = F[2] * F[3] - F[0] * F[5];
  cof[8] = F[0] * F[4] - F[1] * F[3];
  return F[0] * cof[0] + F[1] * cof[1] + F[2] * cof[2];
}

// stress sigma(F) of the reference materials
template <int D, bool HF, class R>
__device__ __forceinline__ void ad_sigma(const AdK<R>& K, const R* s, R* sig) {
  typedef Sch<D, HF, false> S;
#pragma unroll
  for (int k = 0; k < D * D; ++k) sig[k] = 0;
  if (!HF) {
#pragma unroll
    for (int d = 0; d < D; ++d) sig[d * D + d] = K.lam * (s[S::FJ] - (R)1);
    return;
  }
  const R* F = s + S::FJ;
  R cof[9];
  const R J = inv_det_cof<D, R>(F, cof);
  if (K.mat == AQ_MAT_FLUID) {
#pragma unroll
    for (int d = 0; d < D; ++d) sig[d * D + d] = K.lam * (J - (R)1);
    return;
  }
  if (D == 2) {
    R Rm[4];
    polar_rot<2, R>(F, Rm);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        R a = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) a += (F[i * 2 + k] - Rm[i * 2 + k]) * F[j * 2 + k];
        sig[i * 2 + j] = (R)2 * K.mu * a + (i == j ? K.lam * J * (J - (R)1) : (R)0);
      }
  } else {
    const R lj = K.lam * log(J);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        R a = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) a += F[i * 3 + k] * F[j * 3 + k];
        sig[i * 3 + j] = K.mu * (a - (i == j ? (R)1 : (R)0)) + lj;
      }
  }
}

// Fbar (or Jbar) += dsigma/dF^T sbar
template <int D, bool HF, class R>
__device__ __forceinline__ void ad_sigma_bwd(const AdK<R>& K, const R* s, const R* sb, R* gb) {
  typedef Sch<D, HF, false> S;
  R tr = 0, sum = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) tr += sb[d * D + d];
#pragma unroll
  for (int k = 0; k < D * D; ++k) sum += sb[k];
  if (!HF) {
    gb[S::FJ] += K.lam * tr;
    return;
  }
  const R* F = s + S::FJ;
  R* Fb = gb + S::FJ;
  R cof[9];
  const R J = inv_det_cof<D, R>(F, cof);
  if (K.mat == AQ_MAT_FLUID) {
#pragma unroll
    for (int k = 0; k < D * D; ++k) Fb[k] += K.lam * tr * cof[k];
    return;
  }
  if (D == 2) {
    // sigma = 2 mu (F - R) F^T + la J (J-1) I,  R = [[c,-s],[s,c]]
    R Rm[4];
    polar_rot<2, R>(F, Rm);
    R G[4], Gb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) G[k] = F[k] - Rm[k];
    // Gbar = 2 mu sbar F ; Fbar += 2 mu sbar^T G
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        R a = 0, b = 0;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          a += sb[i * 2 + k] * F[k * 2 + j];
          b += sb[k * 2 + i] * G[k * 2 + j];
        }
        Gb[i * 2 + j] = (R)2 * K.mu * a;
        Fb[i * 2 + j] += (R)2 * K.mu * b + Gb[i * 2 + j];
      }
    const R Jb = K.lam * ((R)2 * J - (R)1) * tr;
#pragma unroll
    for (int k = 0; k < 4; ++k) Fb[k] += Jb * cof[k];
    // Rbar = -Gbar ; c = x/r, s = y/r with x = F00+F11, y = F10-F01
    const R cb = -(Gb[0] + Gb[3]);
    const R sbb = -(-Gb[1] + Gb[2]);
    const R x = F[0] + F[3], y = F[2] - F[1];
    const R r2 = x * x + y * y, r = sqrt(r2), r3 = r2 * r;
    const R xb = (cb * y * y - sbb * x * y) / r3;
    const R yb = (-cb * x * y + sbb * x * x) / r3;
    Fb[0] += xb;
    Fb[3] += xb;
    Fb[2] += yb;
    Fb[1] -= yb;
  } else {
    // sigma = mu (F F^T - I) + la log J (every entry)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        R a = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) a += (sb[i * 3 + k] + sb[k * 3 + i]) * F[k * 3 + j];
        Fb[i * 3 + j] += K.mu * a + K.lam * sum * cof[i * 3 + j] / J;
      }
  }
}

// ------------------------------------------------------------- layout
//
// States and their adjoints inside the library: the particles in the order
// of k_ad_keys, in groups of 32 that hold slot s of all 32 side by side, so
// that a warp's loads and stores of a slot are one coalesced access.

__host__ __device__ __forceinline__ int64_t ad_padded(int64_t n) { return (n + 31) & ~int64_t(31); }

template <int NS>
__device__ __forceinline__ int64_t ad_at(int64_t p, int s) {
  return ((p >> 5) * NS + s) * 32 + (p & 31);
}

template <int NS, int LO, int HI, class R>
__device__ __forceinline__ void ad_load(const R* st, int64_t p, R (&s)[NS]) {
#pragma unroll
  for (int k = LO; k < HI; ++k) s[k] = st[ad_at<NS>(p, k)];
}

// ------------------------------------------------------------- warp tiles
//
// Every kernel works warp by warp: 32 particles, neighbours on the grid, and
// the box of nodes their stencils reach.  Where the box fits AdTile nodes the
// warp gathers from a copy of it in shared memory (the node's own operation
// - grid_op or its transpose - applied once per node as it is copied) and
// scatters into a zeroed copy that goes to the grid with one vector reduction
// per node; otherwise (particles that have drifted far apart) straight from
// and to the grid.  No two warps share a tile, so there is no CTA barrier.
// Particle by particle with scalar global atomics, from rows of 96 bytes and
// with the grid's operation in kernels of its own, a substep of the 3D
// falling block (262,144 particles, FP32) took 127 us forward (now 46) and
// 287 us backward, recomputed sums and squares included (now 144).
//
// Half a block's cells (4 x 2 x 4, and 4 x 8 in 2D) reach 6 x 4 x 6 = 144
// nodes (6 x 10 = 60); AdTile leaves room for a cell of drift on every side,
// and for the warps whose particles lie in two blocks.
template <int D>
struct AdTile {
  static constexpr int N = D == 3 ? 416 : 192;
};

// In 3D the tile's stride of axis 0 is padded to 4 mod 8 nodes, so that the
// planes of a warp's neighbouring cells fall in different 16-byte bank groups
// (a forward pass 52 -> 49 us at 262,144 particles).
struct AdBox {
  int o[3], e1, e2, n;  // origin, extents of axes 1 and 2, nodes
  int sa;               // tile stride of axis 0
  int size;             // tile nodes with the padding
  bool fits;
};

// the box of the lanes with `on` (none: an empty box)
template <int D>
__device__ __forceinline__ AdBox ad_box(bool on, const int (&base)[3]) {
  AdBox b;
  int e[3] = {1, 1, 1};
  const bool any = __any_sync(0xffffffffu, on);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    b.o[d] = 0;
    if (d < D) {
      const int lo = __reduce_min_sync(0xffffffffu, on ? base[d] : 0x7fffffff);
      const int hi = __reduce_max_sync(0xffffffffu, on ? base[d] : -1);
      b.o[d] = any ? lo : 0;
      e[d] = any ? hi - lo + 3 : 3;
    }
  }
  b.e1 = e[1];
  b.e2 = D == 3 ? e[2] : 1;
  b.fits = any;
#pragma unroll
  for (int d = 0; d < D; ++d) b.fits = b.fits && e[d] <= AdTile<D>::N;
  // each extent <= AdTile::N: no overflow
  b.n = b.fits ? e[0] * e[1] * e[2] : 0;
  b.sa = D == 3 ? ((b.e1 * b.e2 + 3) & ~7) + 4 : b.e1;
  b.size = b.fits ? e[0] * b.sa : 0;
  b.fits = b.fits && b.size <= AdTile<D>::N;
  return b;
}

// node j of a box: its grid index; returns its place in the tile (exact float
// floors: j < 2^10)
template <int D>
__device__ __forceinline__ int ad_node(const AdBox& b, int j, int (&I)[3]) {
  if (D == 3) {
    const int q = (int)(((float)j + 0.5f) / (float)b.e2);
    const int i0 = (int)(((float)q + 0.5f) / (float)b.e1), i1 = q - i0 * b.e1, i2 = j - q * b.e2;
    I[0] = b.o[0] + i0;
    I[1] = b.o[1] + i1;
    I[2] = b.o[2] + i2;
    return i0 * b.sa + i1 * b.e2 + i2;
  }
  const int i0 = (int)(((float)j + 0.5f) / (float)b.e1);
  I[0] = b.o[0] + i0;
  I[1] = b.o[1] + (j - i0 * b.e1);
  I[2] = 0;
  return j;
}

// wall mask of component k at node I given the velocity sign (grid_op)
template <class R>
__device__ __forceinline__ bool ad_wall(const AdK<R>& K, const int (&I)[3], int k, R vk) {
  return (I[k] < K.wlo[k] && vk < (R)0) || (I[k] > K.whi[k] && vk > (R)0);
}

// Grid velocity of a node from its sums (m, P): (0, v).
template <int D, class R>
struct AdGridOp {
  typedef typename R4T<R>::type R4;
  typedef R4 Raw;
  static constexpr int STAGE = 3;
  const AdK<R>& K;
  const R4* grid;
  __device__ __forceinline__ Raw fetch(const int (&I)[3]) const { return grid[ad_cell<D>(K.res, I)]; }
  __device__ __forceinline__ R4 operator()(const int (&I)[3]) const { return apply(fetch(I), I); }
  __device__ __forceinline__ R4 apply(R4 g, const int (&I)[3]) const {
    const R inv_m = (R)1 / (g.x + (R)1e-10);
    R v[3] = {inv_m * g.y, inv_m * g.z, D == 3 ? inv_m * g.w : (R)0};
    v[1] -= K.dt * K.grav;
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (ad_wall<R>(K, I, k, v[k])) v[k] = 0;
    if (D == 3 && K.col_on) collide_node<R, true>(K, K.pose, I[0], I[1], I[2], v);  // sdf_collision_no_arg
    g.x = 0;
    g.y = v[0];
    g.z = v[1];
    g.w = v[2];
    return g;
  }
};

// Adjoint of a node's sums, (mbar, Pbar), from the sums and the adjoint of
// its velocity (grid^T).
template <int D, class R>
struct AdGridOpT {
  typedef typename R4T<R>::type R4;
  struct Raw {
    R4 g, b;
  };
  static constexpr int STAGE = 2;
  const AdK<R>& K;
  const R4* grid;
  const R4* gvb;
  __device__ __forceinline__ Raw fetch(const int (&I)[3]) const {
    const int64_t c = ad_cell<D>(K.res, I);
    return Raw{grid[c], gvb[c]};
  }
  __device__ __forceinline__ R4 operator()(const int (&I)[3]) const { return apply(fetch(I), I); }
  __device__ __forceinline__ R4 apply(const Raw& raw, const int (&I)[3]) const {
    const R4 g = raw.g, b = raw.b;
    const R P[3] = {g.y, g.z, g.w};
    const R inv_m = (R)1 / (g.x + (R)1e-10);
    R v[3] = {inv_m * P[0], inv_m * P[1], D == 3 ? inv_m * P[2] : (R)0};
    v[1] -= K.dt * K.grav;
    R vb[3] = {b.y, b.z, D == 3 ? b.w : (R)0};
    if (D == 3 && K.col_on) {
      // collider^T: where the node is inside and moving into the surface
      // (relative to the collider), the forward removed the normal part of
      // the velocity, v' = v - ((v - cv).n) n, so vbar' = vbar - (vbar.n) n
      R nrm[3], cv[3];
      if (collider_at<R, true>(K, K.pose, I[0], I[1], I[2], nrm, cv)) {
        R dn = 0, bn = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const R vw = ad_wall<R>(K, I, k, v[k]) ? (R)0 : v[k];  // the collider's input
          dn += (vw - cv[k]) * nrm[k];
          bn += vb[k] * nrm[k];
        }
        if (dn < (R)0)
#pragma unroll
          for (int k = 0; k < 3; ++k) vb[k] -= bn * nrm[k];
      }
    }
    R4 r;
    R mb = 0, Pb[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const R bd = ad_wall<R>(K, I, d, v[d]) ? (R)0 : vb[d];
      Pb[d] = bd * inv_m;
      mb -= bd * P[d] * inv_m * inv_m;
    }
    r.x = mb;
    r.y = Pb[0];
    r.z = Pb[1];
    r.w = Pb[2];
    return r;
  }
};

// copy a box into a tile through the node's operation, F::STAGE nodes of a
// lane in flight at a time
template <int D, class R4, class F>
__device__ __forceinline__ void ad_stage(const AdBox& b, R4* tile, const F& node) {
  for (int j0 = threadIdx.x & 31; j0 < b.n; j0 += 32 * F::STAGE) {
    typename F::Raw raw[F::STAGE];
    int I[F::STAGE][3], at[F::STAGE];
#pragma unroll
    for (int q = 0; q < F::STAGE; ++q) {
      at[q] = -1;
      if (j0 + 32 * q < b.n) {
        at[q] = ad_node<D>(b, j0 + 32 * q, I[q]);
        raw[q] = node.fetch(I[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < F::STAGE; ++q)
      if (at[q] >= 0) tile[at[q]] = node.apply(raw[q], I[q]);
  }
  __syncwarp();
}

template <class R4>
__device__ __forceinline__ void ad_zero(const AdBox& b, R4* tile) {
  R4 z;
  z.x = z.y = z.z = z.w = 0;
  for (int j = threadIdx.x & 31; j < b.size; j += 32) tile[j] = z;
  __syncwarp();
}

template <int D, class R, class R4>
__device__ __forceinline__ void ad_flush(const AdK<R>& K, const AdBox& b, const R4* tile, R4* grid) {
  __syncwarp();
  for (int j = threadIdx.x & 31; j < b.n; j += 32) {
    int I[3];
    const R4 v = tile[ad_node<D>(b, j, I)];
    if (v.x == (R)0 && v.y == (R)0 && v.z == (R)0 && v.w == (R)0) continue;
    red_add_node(grid + ad_cell<D>(K.res, I), v.x, v.y, v.z, v.w);
  }
}

template <int D>
__device__ __forceinline__ int ad_local(const AdBox& b, const int (&base)[3]) {
  return D == 3 ? (base[0] - b.o[0]) * b.sa + (base[1] - b.o[1]) * b.e2 + (base[2] - b.o[2])
                : (base[0] - b.o[0]) * b.e1 + (base[1] - b.o[1]);
}

// The particle's view of its 3^D nodes, in the tile (TILE) or on the grid
// through the node's operation.
template <int D, class R, bool TILE, class F>
struct AdSrc {
  typedef typename R4T<R>::type R4;
  const R4* t;  // the base node in the tile
  int sa, sb;   // tile strides of axes 0 and 1
  const F& node;
  const int (&base)[3];
  __device__ __forceinline__ R4 operator()(int a, int b, int c) const {
    if (TILE) return t[a * sa + b * sb + c];
    const int I[3] = {base[0] + a, base[1] + b, D == 3 ? base[2] + c : 0};
    return node(I);
  }
};

// Offsets of a particle's nodes from it, per axis: dp[o][d] = (o - fx_d) dx.
// Every sum over a particle's nodes is of terms of these offsets, node by
// node.  Taking fx out of the sums (sum w g off - fx sum w g, and m v - A fx +
// A off) is a third fewer operations (3D falling block, 262,144 particles,
// FP32, 32 substeps forward and back: 6.5 ms against 7.4), but the difference
// of two larger sums: the FP32 error of the adjoint of C was 1.3 to 2.3 times
// this form's, that of the new C up to 1.6 times (2D and 3D fluid).
template <int D, class R>
__device__ __forceinline__ void ad_offsets(const AdK<R>& K, const R (&fx)[3], R (&dp)[3][3]) {
#pragma unroll
  for (int o = 0; o < 3; ++o)
#pragma unroll
    for (int d = 0; d < D; ++d) dp[o][d] = ((R)o - fx[d]) * K.dx;
}

// nv = sum w g, nC = 4/dx^2 sum w g dpos^T over the nodes' (y, z, w).
template <int D, class R, bool TILE, class S>
__device__ __forceinline__ void ad_gather(const S& src, const AdK<R>& K, const R (&w)[3][3], const R (&dp)[3][3],
                                          R (&nv)[3], R (&nC)[9]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) nv[d] = 0;
#pragma unroll
  for (int k = 0; k < D * D; ++k) nC[k] = 0;
#pragma unroll(TILE ? 3 : 1)
  for (int a = 0; a < 3; ++a)
#pragma unroll(TILE ? 3 : 1)
    for (int b = 0; b < 3; ++b) {
      const R wab = w[a][0] * w[b][1];
#pragma unroll(TILE ? 3 : 1)
      for (int c = 0; c < (D == 3 ? 3 : 1); ++c) {
        const auto g = src(a, b, c);
        const R wt = D == 3 ? wab * w[c][2] : wab, fw = K.four_inv_dx2 * wt;
        const R gv[3] = {g.y, g.z, g.w};
        const R dpos[3] = {dp[a][0], dp[b][1], D == 3 ? dp[c][2] : (R)0};
#pragma unroll
        for (int d = 0; d < D; ++d) {
          nv[d] += wt * gv[d];
          const R fg = fw * gv[d];
#pragma unroll
          for (int e = 0; e < D; ++e) nC[d * D + e] += fg * dpos[e];
        }
      }
    }
}

// The reverse kernels' walk over a particle's nodes: f(node, dpos, w, grad w).
template <int D, class R, bool TILE, class S, class F>
__device__ __forceinline__ void ad_visit(const S& src, const R (&w)[3][3], const R (&dw)[3][3], const R (&dp)[3][3],
                                         const F& f) {
#pragma unroll(TILE ? 3 : 1)
  for (int a = 0; a < 3; ++a)
#pragma unroll(TILE ? 3 : 1)
    for (int b = 0; b < 3; ++b) {
      const R wab = w[a][0] * w[b][1];
#pragma unroll(TILE ? 3 : 1)
      for (int c = 0; c < (D == 3 ? 3 : 1); ++c) {
        const auto g = src(a, b, c);
        const R dpos[3] = {dp[a][0], dp[b][1], D == 3 ? dp[c][2] : (R)0};
        R gw[3] = {dw[a][0] * w[b][1], dw[b][1] * w[a][0], 0};
        if (D == 3) {
          gw[0] *= w[c][2];
          gw[1] *= w[c][2];
          gw[2] = dw[c][2] * w[a][0] * w[b][1];
        }
        f(g, dpos, D == 3 ? wab * w[c][2] : wab, gw);
      }
    }
}

// h = h0 + A dpos of a node, A's columns in turn
template <int D, class R>
__device__ __forceinline__ void ad_affine(const R (&h0)[3], const R (&A)[9], const R (&dpos)[3], R (&h)[3]) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    h[d] = h0[d];
#pragma unroll
    for (int e = 0; e < D; ++e) h[d] += A[d * D + e] * dpos[e];
  }
}

// Add w (m0, h(dpos)) into the particle's nodes: in the tile with plain
// read-add-writes (lanes of the same base cell take turns, and an offset's
// updates are visible to the warp before the next one's: lanes of
// neighbouring cells reach a node at different offsets), else with global
// reductions.  All lanes call it.
template <int D, class R, bool TILE, class R4, class H>
__device__ __forceinline__ void ad_scatter(const AdK<R>& K, bool on, const int (&base)[3], R4* tile, const AdBox& box,
                                           R4* grid, const R (&w)[3][3], const R (&dp)[3][3], R m0, const H& hf) {
  const int lane = threadIdx.x & 31;
  const int lb = TILE ? ad_local<D>(box, base) : 0;
  int rank = 0, rounds = 1;
  if (TILE) {
    const unsigned peers = __match_any_sync(0xffffffffu, on ? lb : -1 - lane);
    rank = __popc(peers & ((1u << lane) - 1u));
    rounds = (int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(peers));
  }
  const int sb = D == 3 ? box.e2 : 1, sa = box.sa;
  for (int r = 0; r < rounds; ++r) {
    const bool mine = on && rank == r;
    const unsigned tm = __ballot_sync(0xffffffffu, mine);
    if (mine) {
#pragma unroll(TILE ? 3 : 1)
      for (int a = 0; a < 3; ++a)
#pragma unroll(TILE ? 3 : 1)
        for (int b = 0; b < 3; ++b) {
          const R wab = w[a][0] * w[b][1];
#pragma unroll(TILE ? 3 : 1)
          for (int c = 0; c < (D == 3 ? 3 : 1); ++c) {
            const R wt = D == 3 ? wab * w[c][2] : wab;
            const R dpos[3] = {dp[a][0], dp[b][1], D == 3 ? dp[c][2] : (R)0};
            R h[3], val[3] = {0, 0, 0};
            hf(dpos, h);
#pragma unroll
            for (int d = 0; d < D; ++d) val[d] = mul_rn(wt, h[d]);
            if (TILE) {
              R4& t = tile[lb + a * sa + b * sb + c];
              R4 v = t;
              v.x += mul_rn(wt, m0);
              v.y += val[0];
              v.z += val[1];
              if (D == 3) v.w += val[2];
              t = v;
              __syncwarp(tm);
            } else {
              const int I[3] = {base[0] + a, base[1] + b, D == 3 ? base[2] + c : 0};
              red_add_node(grid + ad_cell<D>(K.res, I), wt * m0, val[0], val[1], val[2]);
            }
          }
        }
    }
    __syncwarp();
  }
}

// zero a grid for a later scatter (grid-stride over its nodes)
template <class R4>
__device__ __forceinline__ void ad_clear(R4* g, int64_t nodes) {
  if (!g) return;
  R4 z;
  z.x = z.y = z.z = z.w = 0;
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nodes; j += (int64_t)gridDim.x * blockDim.x)
    g[j] = z;
}

// P2G terms of a particle: its momentum mv and A, so that a node gets w (m, mv + A dpos).
template <int D, bool HF, class R>
__device__ __forceinline__ void ad_p2g_terms(const AdK<R>& K, const R* s, R (&mv)[3], R (&A)[9]) {
  typedef Sch<D, HF, false> S;
  R sig[9];
  ad_sigma<D, HF, R>(K, s, sig);
#pragma unroll
  for (int k = 0; k < D * D; ++k) A[k] = K.kst * sig[k] + K.p_mass * s[S::C + k];
#pragma unroll
  for (int d = 0; d < D; ++d) mv[d] = mul_rn(K.p_mass, s[S::V + d]);
}

// Threads per CTA.  A CTA is no unit of work here; two warps keep the
// granularity of shared memory fine.
constexpr int AD_T = 64;

// ------------------------------------------------------------- forward

// A pass of the forward chain: G2P of one substep (state in -> out, from the
// sums in gin) and / or P2G of the next (of the new state, or of `in`) into
// gout, which is zero; gclr (may be null) is zeroed for the pass after.
template <int D, bool HF, class R, bool G2P, bool P2G>
__global__ void __launch_bounds__(AD_T) k_ad_pass(const __grid_constant__ AdK<R> K, const R* in,
                                                  R* out, int64_t n,
                                                  const typename R4T<R>::type* gin,
                                                  typename R4T<R>::type* gout, typename R4T<R>::type* gclr,
                                                  int64_t nodes) {
  typedef Sch<D, HF, false> S;
  typedef typename R4T<R>::type R4;
  constexpr int NS = S::NS;
  __shared__ __align__(16) R4 tiles[AD_T / 32][AdTile<D>::N];
  R4* const tile = tiles[threadIdx.x >> 5];
  kernel_begin();
  ad_clear(gclr, nodes);
  const int64_t p = (int64_t)blockIdx.x * AD_T + threadIdx.x;
  if (p - threadIdx.x >= n) return;  // a CTA for the clear alone
  const bool on = p < n;
  R s[NS];
  int base[3] = {0, 0, 0};
  R fx[3] = {0, 0, 0}, w[3][3], dp[3][3];
  if (on) ad_load<NS, 0, NS>(in, p, s);
  if (G2P) {
    if (on) ad_weights<D, R>(s + S::X, K, base, fx, w);
    const AdBox box = ad_box<D>(on, base);
    const AdGridOp<D, R> node{K, gin};
    R nv[3], nC[9];
    if (on) ad_offsets<D, R>(K, fx, dp);
    if (box.fits) {
      ad_stage<D>(box, tile, node);
      const AdSrc<D, R, true, AdGridOp<D, R>> src{tile + (on ? ad_local<D>(box, base) : 0),
                                                  box.sa, D == 3 ? box.e2 : 1, node, base};
      if (on) ad_gather<D, R, true>(src, K, w, dp, nv, nC);
      __syncwarp();
    } else if (on) {
      const AdSrc<D, R, false, AdGridOp<D, R>> src{nullptr, 0, 0, node, base};
      ad_gather<D, R, false>(src, K, w, dp, nv, nC);
    }
    if (on) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        s[S::X + d] += K.dt * nv[d];
        s[S::V + d] = nv[d];
      }
#pragma unroll
      for (int k = 0; k < D * D; ++k) s[S::C + k] = nC[k];
      if (HF) {
        R nF[9];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j) {
            R a = 0;
#pragma unroll
            for (int k = 0; k < D; ++k) a += ((i == k ? (R)1 : (R)0) + K.dt * nC[i * D + k]) * s[S::FJ + k * D + j];
            nF[i * D + j] = a;
          }
#pragma unroll
        for (int k = 0; k < D * D; ++k) s[S::FJ + k] = nF[k];
      } else {
        R tr = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) tr += nC[d * D + d];
        s[S::FJ] = ((R)1 + K.dt * tr) * s[S::FJ];
      }
#pragma unroll
      for (int k = 0; k < NS; ++k) out[ad_at<NS>(p, k)] = s[k];
    }
  }
  if (P2G) {
    R mv[3], A[9];
    if (on) {
      ad_weights<D, R>(s + S::X, K, base, fx, w);
      ad_offsets<D, R>(K, fx, dp);
      ad_p2g_terms<D, HF, R>(K, s, mv, A);
    }
    const auto momentum = [&](const R (&dpos)[3], R (&h)[3]) { ad_affine<D, R>(mv, A, dpos, h); };
    const AdBox box = ad_box<D>(on, base);
    if (box.fits) {
      ad_zero(box, tile);
      ad_scatter<D, R, true>(K, on, base, tile, box, gout, w, dp, K.p_mass, momentum);
      ad_flush<D, R>(K, box, tile, gout);
    } else {
      ad_scatter<D, R, false>(K, on, base, tile, box, gout, w, dp, K.p_mass, momentum);
    }
  }
}

// ------------------------------------------------------------- reverse

// G2P^T: from the adjoint of the new state (ab_out) to the x and F|J parts
// of the old state's adjoint (ab_in) and the grid velocity's adjoint (added
// to gvb, zero before).  With h = v'bar + 4/dx^2 C'bar dpos:
// vbar_i += w h, wbar_i = v_i . h, and through dpos
// xbar -= 4/dx^2 w C'bar^T v_i.
template <int D, bool HF, class R>
__global__ void __launch_bounds__(AD_T) k_ad_g2p_bwd(const __grid_constant__ AdK<R> K, const R* st,
                                                     const R* ab_out, R* ab_in, int64_t n,
                                                     const typename R4T<R>::type* grid,
                                                     typename R4T<R>::type* gvb, typename R4T<R>::type* gclr,
                                                     int64_t nodes) {
  typedef Sch<D, HF, false> S;
  typedef typename R4T<R>::type R4;
  constexpr int NS = S::NS;
  extern __shared__ __align__(16) unsigned char ad_smem[];
  R4* const tile = reinterpret_cast<R4*>(ad_smem) + (threadIdx.x >> 5) * 2 * AdTile<D>::N;
  R4* const stile = tile + AdTile<D>::N;
  kernel_begin();
  ad_clear(gclr, nodes);
  const int64_t p = (int64_t)blockIdx.x * AD_T + threadIdx.x;
  if (p - threadIdx.x >= n) return;  // a CTA for the clear alone
  const bool on = p < n;
  R s[NS], bo[NS];
  int base[3] = {0, 0, 0};
  R fx[3] = {0, 0, 0}, w[3][3];
  if (on) {
    ad_load<NS, S::X, S::X + D>(st, p, s);
    ad_load<NS, S::FJ, NS>(st, p, s);
    ad_load<NS, 0, NS>(ab_out, p, bo);
    ad_weights<D, R>(s + S::X, K, base, fx, w);
  }
  const AdBox box = ad_box<D>(on, base);
  const AdGridOp<D, R> node{K, grid};
  R nC[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, vpb[3], Cpb[9], dp[3][3], dw[3][3], xb[3];
  if (on) {
    // Cpb: the new C's adjoint, with F' = (I + dt C') F's (J' = (1 + dt tr C') J's) part
#pragma unroll
    for (int k = 0; k < D * D; ++k) Cpb[k] = bo[S::C + k];
    if (HF) {
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) {
          R c = 0;
#pragma unroll
          for (int k = 0; k < D; ++k) c += bo[S::FJ + i * D + k] * s[S::FJ + j * D + k];  // F'bar F^T
          Cpb[i * D + j] += K.dt * c;
        }
    } else {
      const R trb = K.dt * s[S::FJ] * bo[S::FJ];
#pragma unroll
      for (int d = 0; d < D; ++d) Cpb[d * D + d] += trb;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xb[d] = bo[S::X + d];
      vpb[d] = bo[S::V + d] + K.dt * bo[S::X + d];
    }
    ad_dweights<D, R>(K, fx, dw);
    ad_offsets<D, R>(K, fx, dp);
  }
  // v'bar + 4/dx^2 C'bar dpos
  const auto velocity = [&](const R (&dpos)[3], R (&h)[3]) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      R cd = 0;
#pragma unroll
      for (int e = 0; e < D; ++e) cd += Cpb[d * D + e] * dpos[e];
      h[d] = vpb[d] + K.four_inv_dx2 * cd;
    }
  };
  // per node (weight wt, velocity g): C' and, through w and dpos, xbar
  const auto visit = [&](const R4& g, const R (&dpos)[3], R wt, const R (&gw)[3]) {
    const R gv[3] = {g.y, g.z, g.w}, fw = K.four_inv_dx2 * wt;
    R h[3], wb = 0;
    velocity(dpos, h);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const R fg = fw * gv[d];
#pragma unroll
      for (int e = 0; e < D; ++e) nC[d * D + e] += fg * dpos[e];
      wb += gv[d] * h[d];
    }
#pragma unroll
    for (int e = 0; e < D; ++e) {
      R t = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) t += Cpb[d * D + e] * gv[d];
      xb[e] -= fw * t;
    }
#pragma unroll
    for (int d = 0; d < D; ++d) xb[d] += wb * gw[d];
  };
  if (box.fits) {
    ad_stage<D>(box, tile, node);
    ad_zero(box, stile);
    const AdSrc<D, R, true, AdGridOp<D, R>> src{tile + (on ? ad_local<D>(box, base) : 0), box.sa, D == 3 ? box.e2 : 1,
                                                node, base};
    if (on) ad_visit<D, R, true>(src, w, dw, dp, visit);
  } else if (on) {
    const AdSrc<D, R, false, AdGridOp<D, R>> src{nullptr, 0, 0, node, base};
    ad_visit<D, R, false>(src, w, dw, dp, visit);
  }
  if (on) {
    if (HF) {
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) {
          R a = 0;
#pragma unroll
          for (int k = 0; k < D; ++k)
            a += ((k == i ? (R)1 : (R)0) + K.dt * nC[k * D + i]) * bo[S::FJ + k * D + j];  // (I+dtC')^T F'bar
          ab_in[ad_at<NS>(p, S::FJ + i * D + j)] = a;
        }
    } else {
      R tr = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) tr += nC[d * D + d];
      ab_in[ad_at<NS>(p, S::FJ)] = ((R)1 + K.dt * tr) * bo[S::FJ];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) ab_in[ad_at<NS>(p, S::X + d)] = xb[d];
  }
  if (box.fits) {
    ad_scatter<D, R, true>(K, on, base, stile, box, gvb, w, dp, (R)0, velocity);
    ad_flush<D, R>(K, box, stile, gvb);
  } else {
    ad_scatter<D, R, false>(K, on, base, stile, box, gvb, w, dp, (R)0, velocity);
  }
}

// Sums over the warp of NS values per lane, in 31 exchanges: in each step the
// two halves of a lane group keep half of the values each.  Lane l returns
// the sum of value l.
template <int NS>
__device__ __forceinline__ double ad_warp_sums(const double (&v)[NS]) {
  double a[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) a[k] = k < NS ? v[k] : 0.0;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 16; h; h >>= 1) {
    const bool up = lane & h;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const double keep = up ? a[k + h] : a[k], give = up ? a[k] : a[k + h];
      a[k] = keep + __shfl_xor_sync(0xffffffffu, give, h);
    }
  }
  return a[0];
}

constexpr int AD_SENS_COPIES = 32;  // copies of the sensitivity sums, so that CTAs' additions do not queue on one

// P2G^T: the old state's adjoint, completed (ab_in holds G2P^T's part on
// entry); with sens, its squares are added to the sensitivity sums in FP64.
template <int D, bool HF, class R>
__global__ void __launch_bounds__(AD_T) k_ad_p2g_bwd(const __grid_constant__ AdK<R> K, const R* st,
                                                     R* ab_in, int64_t n,
                                                     const typename R4T<R>::type* grid,
                                                     const typename R4T<R>::type* gvb,
                                                     double* sens) {
  typedef Sch<D, HF, false> S;
  typedef typename R4T<R>::type R4;
  constexpr int NS = S::NS;
  __shared__ __align__(16) R4 tiles[AD_T / 32][AdTile<D>::N];
  R4* const tile = tiles[threadIdx.x >> 5];
  kernel_begin();
  const int64_t p = (int64_t)blockIdx.x * AD_T + threadIdx.x;
  const bool on = p < n;
  R s[NS], bi[NS];
  int base[3] = {0, 0, 0};
  R fx[3] = {0, 0, 0}, w[3][3];
  if (on) {
    ad_load<NS, 0, NS>(st, p, s);
    ad_load<NS, S::X, S::X + D>(ab_in, p, bi);
    ad_load<NS, S::FJ, NS>(ab_in, p, bi);
    ad_weights<D, R>(s + S::X, K, base, fx, w);
  }
  const AdBox box = ad_box<D>(on, base);
  const AdGridOpT<D, R> node{K, grid, gvb};
  R mv[3], A[9], Ab[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dp[3][3], dw[3][3], xb[3] = {0, 0, 0}, vb[3] = {0, 0, 0};
  if (on) {
    ad_p2g_terms<D, HF, R>(K, s, mv, A);
    ad_dweights<D, R>(K, fx, dw);
    ad_offsets<D, R>(K, fx, dp);
  }
  // per node (weight wt, adjoint (mbar, Pbar)): vbar, Abar and, through w and dpos, xbar
  const auto visit = [&](const R4& g, const R (&dpos)[3], R wt, const R (&gw)[3]) {
    const R P[3] = {g.y, g.z, g.w}, wm = wt * K.p_mass;
    R h[3], wb = K.p_mass * g.x;
    ad_affine<D, R>(mv, A, dpos, h);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      wb += P[d] * h[d];
      vb[d] += wm * P[d];
      const R wP = wt * P[d];
#pragma unroll
      for (int e = 0; e < D; ++e) {
        Ab[d * D + e] += wP * dpos[e];
        xb[e] -= wt * A[d * D + e] * P[d];  // through dpos = x_i - x_p
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) xb[d] += wb * gw[d];
  };
  if (box.fits) {
    ad_stage<D>(box, tile, node);
    const AdSrc<D, R, true, AdGridOpT<D, R>> src{tile + (on ? ad_local<D>(box, base) : 0),
                                                 box.sa, D == 3 ? box.e2 : 1, node, base};
    if (on) ad_visit<D, R, true>(src, w, dw, dp, visit);
  } else if (on) {
    const AdSrc<D, R, false, AdGridOpT<D, R>> src{nullptr, 0, 0, node, base};
    ad_visit<D, R, false>(src, w, dw, dp, visit);
  }
  if (on) {
    R sb[9];
#pragma unroll
    for (int k = 0; k < D * D; ++k) {
      bi[S::C + k] = K.p_mass * Ab[k];
      sb[k] = K.kst * Ab[k];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      bi[S::X + d] += xb[d];
      bi[S::V + d] = vb[d];
    }
    ad_sigma_bwd<D, HF, R>(K, s, sb, bi);
#pragma unroll
    for (int k = 0; k < NS; ++k) ab_in[ad_at<NS>(p, k)] = bi[k];
  }
  if (sens) {
    double sq[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) sq[k] = on ? (double)bi[k] * (double)bi[k] : 0.0;
    const double t = ad_warp_sums<NS>(sq);
    __shared__ double part[AD_T / 32][32];
    part[threadIdx.x >> 5][threadIdx.x & 31] = t;
    __syncthreads();
    if (threadIdx.x < NS) {
      double a = 0;
#pragma unroll
      for (int k = 0; k < AD_T / 32; ++k) a += part[k][threadIdx.x];
      atomicAdd(sens + (blockIdx.x % AD_SENS_COPIES) * NS + threadIdx.x, a);
    }
  }
}

// ------------------------------------------------------------- order
//
// Order of the particles inside the library, from their base cells at the
// start (they move little over an adjoint horizon): by cell block (4^3 or
// 8^2) along a serpentine, so that blocks that follow each other are
// neighbours; inside a block the first particle of every cell, then the
// second of every cell, and so on, so that a warp's lanes scatter from
// different cells.
constexpr int AD_RANK_BITS = 10;  // ranks beyond 2^10 - 1 share the last place

template <class R>
__global__ void k_ad_keys(const R* __restrict__ st, int64_t n, int ns, int D, int r0, int r1, int r2, R inv_dx,
                          int32_t* __restrict__ count, uint64_t* __restrict__ keys, int32_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int res[3] = {r0, r1, r2};
  const int bs = D == 3 ? 2 : 3;  // log2 of the block's edge
  int64_t cell = 0;
  int b[3] = {0, 0, 0};
  for (int d = 0; d < D; ++d) {
    const R t = st[i * ns + d] * inv_dx - (R)0.5;
    const int f = t == t ? (int)floor(t) : 0;
    b[d] = min(max(f, 0), res[d] - 1);
    cell = cell * res[d] + b[d];
  }
  const int rank = min(atomicAdd(count + cell, 1), (1 << AD_RANK_BITS) - 1);
  uint64_t blk = 0;
  int turn = 0;  // whether this axis runs backwards
  for (int d = 0; d < D; ++d) {
    const int nb = (res[d] + (1 << bs) - 1) >> bs, q = b[d] >> bs;
    const int at = turn ? nb - 1 - q : q;
    blk = blk * nb + at;
    turn ^= at & 1;
  }
  const int m = (1 << bs) - 1;
  // cells z fastest, then x, then y, as the simulator's binning
  const int c = D == 3 ? (((b[1] & m) << 2 | (b[0] & m)) << 2) | (b[2] & m) : ((b[0] & m) << 3) | (b[1] & m);
  keys[i] = ((blk << AD_RANK_BITS) | (uint64_t)rank) << 6 | (uint64_t)c;
  idx[i] = (int32_t)i;
}

// Between the caller's rows (n x ns, the caller's order) and the library's
// groups: a warp moves a group through shared memory, so that both sides are
// read and written in contiguous runs.  TO: rows -> groups.
template <class R, bool TO>
__global__ void __launch_bounds__(128) k_ad_permute(const R* __restrict__ in, R* __restrict__ out,
                                                    const int32_t* __restrict__ perm, int64_t n, int ns) {
  __shared__ R sh[4][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t g = (int64_t)blockIdx.x * 4 + warp;
  if (g * 32 >= n) return;
  const int cnt = (int)min((int64_t)32, n - g * 32);
  const int64_t row = lane < cnt ? (int64_t)perm[g * 32 + lane] * ns : 0;
  if (TO) {
    for (int r = 0; r < cnt; ++r) {
      const int64_t at = __shfl_sync(0xffffffffu, row, r);
      if (lane < ns) sh[warp][r][lane] = in[at + lane];
    }
    __syncwarp();
    for (int s = 0; s < ns; ++s)
      if (lane < cnt) out[(g * ns + s) * 32 + lane] = sh[warp][lane][s];
  } else {
    for (int s = 0; s < ns; ++s)
      if (lane < cnt) sh[warp][lane][s] = in[(g * ns + s) * 32 + lane];
    __syncwarp();
    for (int r = 0; r < cnt; ++r) {
      const int64_t at = __shfl_sync(0xffffffffu, row, r);
      if (lane < ns) out[at + lane] = sh[warp][r][lane];
    }
  }
}

// --------------------------------------------------------------- host

struct AdBase {
  virtual ~AdBase() {}
  virtual int setup() = 0;
  // t: index of the substep (the collider's angle and height depend on it)
  virtual int p2g(const void* in, cudaStream_t st) = 0;
  virtual int g2p(const void* in, void* out, int t, bool then_p2g, cudaStream_t st) = 0;
  virtual int step_bwd(const void* s_in, const void* ab_out, void* ab_in, int t, bool accumulate, cudaStream_t st) = 0;
  virtual int sort_keys(const void* s0, int32_t* count, uint64_t* keys, int32_t* idx, cudaStream_t st) = 0;
  virtual int permute(const void* in, void* out, bool gather, cudaStream_t st) = 0;
};

}  // namespace aq

struct aq_adjoint {
  aq_params P;
  int D = 0, NS = 0;
  int device = 0;  // where its memory is
  int64_t n = 0, ncell = 0;
  size_t rsz = 4;
  // three node grids in rotation: g[rot] takes (or holds) the current
  // state's sums (m, P); every kernel that fills one of the others clears
  // the one after, so that g[rot] is zero whenever a chain starts (unless
  // broken: a pass did not run to its end, or was only captured into a graph)
  void* g[3] = {nullptr, nullptr, nullptr};
  int rot = 0;
  bool broken = false;
  std::vector<void*> ckpt;  // states at multiples of the checkpoint interval (every > 0), or the initial state
  std::vector<void*> seg;   // states between two checkpoints; two ping-pong states (every == 0)
  std::vector<void*> stash;  // bisection checkpointing: one state per recursion level, plus a scratch state
  std::vector<void*> ab;     // the adjoints of two states, of the backward pass
  int T = 0, every = 0;
  int seg_of = -1;           // the segment whose states seg holds
  int32_t* perm = nullptr;  // sorted position -> caller's particle index (length n)
  int64_t recomputed = 0;   // forward substeps run again by the last backward pass
  double* dsens = nullptr;  // AD_SENS_COPIES x NS
  aq::AdBase* impl = nullptr;
  // SDF collider (aq_adjoint_set_collider): caller-owned volumes; at
  // substep t the angle is theta + omega dt t and the height
  // height + rate dt t (step_collider_difftaichi, mpm_solver.py:1554-1559)
  int col_on = 0, col_center = 0, col_dims[3] = {0, 0, 0}, col_off[3] = {0, 0, 0};
  const float* col_sdf = nullptr;
  const float* col_nrm = nullptr;
  double col_theta = 0, col_height = 0, col_omega = 0, col_rate = 0;

  size_t state_bytes() const { return rsz * NS * (size_t)aq::ad_padded(n); }
};

namespace aq {

// I < lb and I > ub of a node index against a wall in doubles, as integers
static int wall_lo(double lb) { return !(lb > -1e9) ? -1000000000 : lb > 1e9 ? 1000000000 : (int)ceil(lb); }
static int wall_hi(double ub) { return !(ub < 1e9) ? 1000000000 : ub < -1e9 ? -1000000000 : (int)floor(ub); }

template <int D, bool HF, class R>
struct AdImpl final : AdBase {
  typedef typename R4T<R>::type R4;
  aq_adjoint* a;
  AdK<R> K;
  static constexpr int G2P_BWD_SMEM = (AD_T / 32) * 2 * AdTile<D>::N * (int)sizeof(R4);
  explicit AdImpl(aq_adjoint* adj) : a(adj) {
    const aq_params& P = adj->P;
    memset(&K, 0, sizeof(K));
    for (int d = 0; d < 3; ++d) {
      K.res[d] = d < D ? P.res[d] : 1;
      K.wlo[d] = wall_lo(P.lb[d]);
      K.whi[d] = wall_hi(P.ub[d]);
    }
    K.mat = P.mat[0].kind;
    K.inv_dx = (R)(1.0 / P.dx);
    K.dx = (R)P.dx;
    K.dt = (R)P.dt;
    K.p_mass = (R)P.p_mass;
    K.kst = (R)(-(P.dt * P.p_vol * 4.0 * (1.0 / P.dx) * (1.0 / P.dx)));
    K.four_inv_dx2 = (R)(4.0 / (P.dx * P.dx));
    K.grav = (R)P.gravity;
    K.mu = (R)P.mat[0].mu;
    K.lam = (R)P.mat[0].lam;
  }
  int setup() override {
    AQ_CUDA_TRY(cudaFuncSetAttribute(k_ad_g2p_bwd<D, HF, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, G2P_BWD_SMEM));
    return AQ_OK;
  }
  void set_substep(int t) {
    K.col_on = a->col_on;
    if (!K.col_on) return;
    K.col_n = a->col_center;
    for (int d = 0; d < 3; ++d) {
      K.col_dims[d] = a->col_dims[d];
      K.col_off[d] = a->col_off[d];
      K.col_lo[d] = (int)a->P.lb[d];
      K.col_hi[d] = (int)a->P.ub[d];
    }
    K.col_sdf = a->col_sdf;
    K.col_nrm = a->col_nrm;
    K.col_omega = (R)a->col_omega;
    const double th = a->col_theta + a->col_omega * a->P.dt * t;
    const double h = a->col_height + a->col_rate * a->P.dt * t;
    K.pose.c = (R)cos(th);
    K.pose.s = (R)sin(th);
    K.pose.yshift = (int)(h / a->P.dx + 0.5);
  }
  R4* g(int k) const { return (R4*)a->g[(a->rot + k) % 3]; }
  unsigned blocks() const { return grid_for(a->n, AD_T); }
  // the same with enough CTAs for the clear (16 nodes a thread) where there
  // are few particles on a large grid (64 particles on 128^3 nodes, 8 substeps
  // forward and back: 13.3 ms with the particles' one CTA, 0.51 with these)
  unsigned clear_blocks() const { return std::max(blocks(), grid_for(a->ncell, 16 * AD_T)); }

  // the sums of state `in` into g[rot]
  int p2g(const void* in, cudaStream_t st) override {
    AQ_CUDA_TRY(launch_pdl(k_ad_pass<D, HF, R, false, true>, clear_blocks(), AD_T, 0, st, K, (const R*)in, (R*)nullptr, a->n,
                           (const R4*)nullptr, g(0), g(1), a->ncell));
    return AQ_OK;
  }
  // substep t from the state whose sums are in g[rot], and the new state's
  // sums, which g[rot] then names
  int g2p(const void* in, void* out, int t, bool then_p2g, cudaStream_t st) override {
    set_substep(t);
    if (then_p2g)
      AQ_CUDA_TRY(launch_pdl(k_ad_pass<D, HF, R, true, true>, clear_blocks(), AD_T, 0, st, K, (const R*)in, (R*)out, a->n,
                             (const R4*)g(0), g(1), g(2), a->ncell));
    else
      AQ_CUDA_TRY(launch_pdl(k_ad_pass<D, HF, R, true, false>, blocks(), AD_T, 0, st, K, (const R*)in, (R*)out, a->n,
                             (const R4*)g(0), (R4*)nullptr, (R4*)nullptr, (int64_t)0));
    a->rot = (a->rot + 1) % 3;
    return AQ_OK;
  }
  // reverse of substep t, whose old state's sums are in g[rot]
  int step_bwd(const void* s_in, const void* ab_out, void* ab_in, int t, bool accumulate, cudaStream_t st) override {
    set_substep(t);
    AQ_CUDA_TRY(launch_pdl(k_ad_g2p_bwd<D, HF, R>, clear_blocks(), AD_T, G2P_BWD_SMEM, st, K, (const R*)s_in,
                           (const R*)ab_out, (R*)ab_in, a->n, (const R4*)g(0), g(1), g(2), a->ncell));
    AQ_CUDA_TRY(launch_pdl(k_ad_p2g_bwd<D, HF, R>, blocks(), AD_T, 0, st, K, (const R*)s_in, (R*)ab_in, a->n,
                           (const R4*)g(0), (const R4*)g(1), accumulate ? a->dsens : (double*)nullptr));
    a->rot = (a->rot + 2) % 3;
    return AQ_OK;
  }
  int sort_keys(const void* s0, int32_t* count, uint64_t* keys, int32_t* idx, cudaStream_t st) override {
    k_ad_keys<R><<<grid_for(a->n, 256), 256, 0, st>>>((const R*)s0, a->n, a->NS, D, K.res[0], K.res[1], K.res[2],
                                                      K.inv_dx, count, keys, idx);
    AQ_CUDA_TRY(cudaGetLastError());
    return AQ_OK;
  }
  int permute(const void* in, void* out, bool gather, cudaStream_t st) override {
    const unsigned nb = grid_for(a->n, 128);
    if (gather)
      k_ad_permute<R, true><<<nb, 128, 0, st>>>((const R*)in, (R*)out, a->perm, a->n, a->NS);
    else
      k_ad_permute<R, false><<<nb, 128, 0, st>>>((const R*)in, (R*)out, a->perm, a->n, a->NS);
    AQ_CUDA_TRY(cudaGetLastError());
    return AQ_OK;
  }
};

// Sort the particles (k_ad_keys's order): a->perm[sorted position] = caller's index.
static int ad_make_perm(aq_adjoint* a, const void* d_s0, cudaStream_t st) {
  const int bs = a->D == 3 ? 4 : 8;
  int64_t nblk = 1;
  for (int d = 0; d < a->D; ++d) nblk *= (a->P.res[d] + bs - 1) / bs;
  int bits = AD_RANK_BITS + 6 + 1;
  while (bits < 64 && (int64_t(1) << (bits - AD_RANK_BITS - 6)) < nblk) ++bits;
  size_t tb = 0;
  uint64_t* nk = nullptr;
  AQ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, nk, nk, (int32_t*)nullptr, a->perm, (int)a->n, 0, bits, st));
  const size_t n8 = (sizeof(uint64_t) * (size_t)a->n + 255) & ~(size_t)255;
  char* tmp = nullptr;  // keys in, keys out, idx in, the sort's own
  if (pool_alloc((void**)&tmp, 3 * n8 + tb, st) != cudaSuccess) return AQ_E_NOMEM;
  uint64_t *kin = (uint64_t*)tmp, *kout = (uint64_t*)(tmp + n8);
  int32_t* iin = (int32_t*)(tmp + 2 * n8);
  // per-cell counts in the grid that takes the first state's sums: cleared
  // whole before them (a captured pass starts from what the one before left)
  // and again behind them
  void* count = a->g[a->rot];
  cudaError_t e = cudaMemsetAsync(count, 0, a->rsz * 4 * a->ncell, st);
  int rc = e == cudaSuccess ? a->impl->sort_keys(d_s0, (int32_t*)count, kin, iin, st) : AQ_E_CUDA;
  if (rc == AQ_OK &&
      cub::DeviceRadixSort::SortPairs(tmp + 3 * n8, tb, kin, kout, iin, a->perm, (int)a->n, 0, bits, st) != cudaSuccess)
    rc = AQ_E_CUDA;
  if (cudaMemsetAsync(count, 0, sizeof(int32_t) * a->ncell, st) != cudaSuccess && rc == AQ_OK) rc = AQ_E_CUDA;
  pool_free(tmp, st);
  return rc;
}

// Run substeps t0 .. t0 + k - 1 from the state in `in` (k >= 1), landing the
// state t0 + j in buf(j); with keep_sums, g[rot] then holds the last state's
// sums.
template <class F>
static int ad_chain(aq_adjoint* a, const void* in, int t0, int k, const F& buf, bool keep_sums, cudaStream_t st) {
  int rc = a->impl->p2g(in, st);
  for (int j = 1; j <= k && rc == AQ_OK; ++j) {
    rc = a->impl->g2p(in, buf(j), t0 + j - 1, j < k || keep_sums, st);
    in = buf(j);
  }
  return rc;
}

// Run substeps t0 .. t0 + k - 1 from the state in `in` (k >= 1), landing the
// state t0 + k in `dst` and using `tmp` as the other buffer; `in` is kept.
static int ad_run(aq_adjoint* a, const void* in, int t0, int k, void* dst, void* tmp, cudaStream_t st) {
  a->recomputed += k;
  return ad_chain(a, in, t0, k, [=](int j) { return (k - j) % 2 == 0 ? dst : tmp; }, false, st);
}

// Bisection checkpointing (the reference's logarithmic stash,
// run_forward_with_ad_nlogn / rerun_from / cnt_ending_zero,
// mpm_solver.py:1093-1137,1201-1207, restated as a recursion): to reverse
// substeps [t0, t1) from the state t0 in `buf`, run forward to the midpoint
// m, keep the state m in this level's stash, reverse [m, t1) with it, then
// reverse [t0, m) from `buf` (reusing the level's stash, which is free
// again).  Memory: one state per level (ceil(log2 T)); recomputation: about
// T log2(T) / 2 substeps.  ab[cur] holds the adjoint of state t1 on entry and
// of state t0 on return.
static int ad_reverse_bisect(aq_adjoint* a, int t0, int t1, const void* buf, int level, void** ab, int& cur,
                             cudaStream_t st) {
  if (t1 - t0 == 1) {
    int rc = a->impl->p2g(buf, st);
    if (rc == AQ_OK) rc = a->impl->step_bwd(buf, ab[cur], ab[1 - cur], t0, t0 >= 1, st);
    cur = 1 - cur;
    return rc;
  }
  const int m = t0 + (t1 - t0 + 1) / 2;
  void* mid = a->stash[level];
  int rc = ad_run(a, buf, t0, m - t0, mid, a->stash.back(), st);
  if (rc) return rc;
  if ((rc = ad_reverse_bisect(a, m, t1, mid, level + 1, ab, cur, st))) return rc;
  return ad_reverse_bisect(a, t0, m, buf, level, ab, cur, st);
}

// `want` state buffers in v; those it has are kept
static int ad_buffers(aq_adjoint* a, std::vector<void*>& v, int want, cudaStream_t st) {
  if ((int)v.size() > want) {
    cudaDeviceSynchronize();  // another stream may still use them
    for (; (int)v.size() > want; v.pop_back()) pool_free(v.back(), st);
  }
  while ((int)v.size() < want) {
    void* p = nullptr;
    AQ_CUDA_TRY(pool_alloc(&p, a->state_bytes(), st));
    v.push_back(p);
  }
  return AQ_OK;
}

// A pass begins: the grids zeroed if the last one broke off.
static int ad_begin(aq_adjoint* a, cudaStream_t st) {
  if (a->broken)
    for (void* g : a->g) AQ_CUDA_TRY(cudaMemsetAsync(g, 0, a->rsz * 4 * a->ncell, st));
  a->broken = true;  // until its last launch is queued
  return AQ_OK;
}

template <int D, class R>
static AdBase* make_ad(aq_adjoint* a) {
  if (a->P.has_F) return new (std::nothrow) AdImpl<D, true, R>(a);
  return new (std::nothrow) AdImpl<D, false, R>(a);
}

static void free_ad(aq_adjoint* a) {
  if (!a) return;
  delete a->impl;
  for (auto* v : {&a->ckpt, &a->seg, &a->stash, &a->ab})
    for (void* p : *v) pool_free(p, 0);
  pool_free(a->perm, 0);
  for (void* p : a->g) pool_free(p, 0);
  pool_free(a->dsens, 0);
  delete a;
}

}  // namespace aq

using namespace aq;

extern "C" {

int aq_adjoint_create(const aq_params* P, aq_adjoint** out) {
  if (!P || !out) return AQ_E_ARG;
  *out = nullptr;
  const int D = P->dim;
  if (D != 2 && D != 3) return AQ_E_ARG;
  if (P->has_mat) return AQ_E_LAYOUT;
  if (P->n_particles < 1 || P->n_particles > 0x7fffffffLL) return AQ_E_ARG;
  for (int d = 0; d < D; ++d)
    if (P->res[d] < 3 || P->res[d] > 8192) return AQ_E_ARG;
  const int mk = P->mat[0].kind;
  if (mk != AQ_MAT_FLUID && mk != AQ_MAT_ELASTIC) return AQ_E_ARG;  // reference materials only
  if (!P->has_F && mk != AQ_MAT_FLUID) return AQ_E_LAYOUT;
  if (P->use_friction) return AQ_E_ARG;  // the reference's AD scenes run without friction
  aq_adjoint* a = new (std::nothrow) aq_adjoint();
  if (!a) return AQ_E_NOMEM;
  a->P = *P;
  a->D = D;
  a->NS = 2 * D + D * D + (P->has_F ? D * D : 1);
  a->n = P->n_particles;
  a->rsz = P->precision ? sizeof(double) : sizeof(float);
  a->ncell = 1;
  for (int d = 0; d < D; ++d) a->ncell *= P->res[d];
  const size_t gbytes = a->rsz * 4 * a->ncell;
  cudaError_t e = cudaGetDevice(&a->device);
  for (int k = 0; k < 3; ++k) {
    if (e == cudaSuccess) e = pool_alloc(&a->g[k], gbytes, 0);
    if (e == cudaSuccess) e = cudaMemsetAsync(a->g[k], 0, gbytes, 0);
  }
  if (e == cudaSuccess) e = pool_alloc((void**)&a->dsens, sizeof(double) * AD_SENS_COPIES * a->NS, 0);
  if (e == cudaSuccess) e = pool_alloc((void**)&a->perm, sizeof(int32_t) * a->n, 0);
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);  // the memory is there for every stream
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "cudaMallocFromPoolAsync");
    free_ad(a);
    return AQ_E_NOMEM;
  }
  if (D == 3)
    a->impl = P->precision ? make_ad<3, double>(a) : make_ad<3, float>(a);
  else
    a->impl = P->precision ? make_ad<2, double>(a) : make_ad<2, float>(a);
  if (!a->impl) {
    free_ad(a);
    return AQ_E_NOMEM;
  }
  const int rc = a->impl->setup();
  if (rc != AQ_OK) {
    free_ad(a);
    return rc;
  }
  *out = a;
  return AQ_OK;
}

int aq_adjoint_set_collider(aq_adjoint* a, const float* d_sdf, const float* d_normal, const int32_t* dims,
                            const int32_t* offset, int32_t center, double theta, double height, double omega,
                            double height_rate) {
  if (!a) return AQ_E_ARG;
  if (!d_sdf) {
    a->col_on = 0;
    return AQ_OK;
  }
  if (a->D != 3 || !d_normal || !dims || !offset) return AQ_E_ARG;
  for (int k = 0; k < 3; ++k)
    if (dims[k] < 1) return AQ_E_ARG;
  a->col_on = 1;
  a->col_center = center;
  a->col_sdf = d_sdf;
  a->col_nrm = d_normal;
  for (int k = 0; k < 3; ++k) {
    a->col_dims[k] = dims[k];
    a->col_off[k] = offset[k];
  }
  a->col_theta = theta;
  a->col_height = height;
  a->col_omega = omega;
  a->col_rate = height_rate;
  return AQ_OK;
}

int aq_adjoint_destroy(aq_adjoint* a) {
  if (!a) return AQ_E_ARG;
  const OnDevice on(a->device);
  cudaDeviceSynchronize();
  free_ad(a);
  cudaStreamSynchronize(0);  // what the pool does not keep goes back to the device now
  return AQ_OK;
}

int aq_adjoint_forward(aq_adjoint* a, const void* d_s0, int32_t n_substeps, int32_t every, void* d_sT,
                       void* stream) {
  if (!a || !d_s0 || !d_sT || n_substeps < 1 || every < 0) return AQ_E_ARG;
  cudaStream_t st = as_stream(stream);
  const bool bisect = every == 0;
  int rc;
  a->T = 0;  // no valid run until this one is queued
  if ((rc = ad_buffers(a, a->ckpt, bisect ? 1 : (n_substeps + every - 1) / every, st))) return rc;
  if ((rc = ad_buffers(a, a->seg, bisect ? 2 : every, st))) return rc;
  if (!bisect && (rc = ad_buffers(a, a->stash, 0, st))) return rc;
  if ((rc = ad_begin(a, st))) return rc;
  // the state is kept in the library's order and layout; the caller's is
  // restored for d_sT here and for the gradients in aq_adjoint_backward
  if ((rc = ad_make_perm(a, d_s0, st))) return rc;
  if ((rc = a->impl->permute(d_s0, a->ckpt[0], true, st))) return rc;
  // state t goes to its checkpoint or to its place in the segment; the last
  // segment's states stay there for the backward pass
  const auto buf = [&](int t) -> void* {
    if (bisect) return a->seg[t & 1];
    if (t % every) return a->seg[t % every];
    return t < n_substeps ? a->ckpt[t / every] : a->seg[0];
  };
  if ((rc = ad_chain(a, a->ckpt[0], 0, n_substeps, buf, false, st))) return rc;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  AQ_CUDA_TRY(cudaStreamIsCapturing(st, &capturing));
  a->broken = capturing != cudaStreamCaptureStatusNone;
  a->T = n_substeps;
  a->every = every;
  a->seg_of = bisect ? -1 : (n_substeps - 1) / every;
  return a->impl->permute(buf(n_substeps), d_sT, false, st);
}

int aq_adjoint_backward(aq_adjoint* a, const void* d_seed, void* d_grad_s0, double* h_sens, void* stream) {
  if (!a || !d_seed || a->T < 1) return AQ_E_ARG;
  cudaStream_t st = as_stream(stream);
  const int T = a->T, every = a->every;
  int rc = AQ_OK, levels = 1;
  while ((1 << levels) < T) ++levels;
  // one stash per level, the last one is scratch
  if (every == 0 && (rc = ad_buffers(a, a->stash, levels + 1, st))) return rc;
  if ((rc = ad_buffers(a, a->ab, 2, st))) return rc;
  if ((rc = ad_begin(a, st))) return rc;
  void** ab = a->ab.data();
  rc = a->impl->permute(d_seed, ab[0], true, st);  // into the order of the forward pass
  const size_t sens_bytes = sizeof(double) * AD_SENS_COPIES * a->NS;
  if (rc == AQ_OK && cudaMemsetAsync(a->dsens, 0, sens_bytes, st) != cudaSuccess) rc = AQ_E_CUDA;
  int cur = 0;  // ab[cur] = adjoint of state t+1
  a->recomputed = 0;
  if (every == 0 && rc == AQ_OK) rc = ad_reverse_bisect(a, 0, T, a->ckpt[0], 0, ab, cur, st);
  for (int sgi = every == 0 ? -1 : (T - 1) / every; sgi >= 0 && rc == AQ_OK; --sgi) {
    const int t0 = sgi * every, t1 = std::min(T, t0 + every);
    const auto state = [&](int t) -> void* { return t == t0 ? a->ckpt[sgi] : a->seg[t - t0]; };
    bool sums = false;  // g[rot] holds the sums of state t1 - 1
    if (sgi != a->seg_of) {
      a->seg_of = -1;
      if (t1 - 1 > t0) {
        rc = ad_chain(a, a->ckpt[sgi], t0, t1 - 1 - t0, [&](int j) { return state(t0 + j); }, true, st);
        sums = true;
      }
      if (rc == AQ_OK) a->seg_of = sgi;
    }
    for (int t = t1 - 1; t >= t0 && rc == AQ_OK; --t) {
      if (!sums) rc = a->impl->p2g(state(t), st);
      sums = false;
      if (rc == AQ_OK) rc = a->impl->step_bwd(state(t), ab[cur], ab[1 - cur], t, t >= 1, st);
      cur = 1 - cur;  // ab[cur] = adjoint of state t
    }
  }
  if (rc == AQ_OK && d_grad_s0) rc = a->impl->permute(ab[cur], d_grad_s0, false, st);
  std::vector<double> part((size_t)AD_SENS_COPIES * a->NS);
  cudaError_t e = cudaSuccess;
  if (rc == AQ_OK && h_sens) e = cudaMemcpyAsync(part.data(), a->dsens, sens_bytes, cudaMemcpyDeviceToHost, st);
  const cudaError_t es = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) set_last_cuda_error(e, "aq_adjoint_backward");
  if (rc == AQ_OK && e != cudaSuccess) rc = AQ_E_CUDA;
  a->broken = rc != AQ_OK;
  if (rc == AQ_OK && h_sens)
    for (int s = 0; s < a->NS; ++s) {
      h_sens[s] = 0;
      for (int k = 0; k < AD_SENS_COPIES; ++k) h_sens[s] += part[(size_t)k * a->NS + s];
    }
  return rc;
}

}  // extern "C"
