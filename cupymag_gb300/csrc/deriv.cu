// Matrix-free derivative and coupling operators of the periodic hex grid (sm_103a).
//
// The three derivative matrices F_i (F_i[p, q] = integral of N_p dN_q/dx_i,
// cupymag/physics/assemble_demag.py:95-184) and the magnetoelastic coupling
// F_el = B^T C S (cupymag/physics/assemble_elasticity.py:268-459) are, on a
// grid of identical unit cells, 27-point periodic stencils: the coefficient
// between DOF p and DOF p + d is the same for every p.  These kernels apply
// them without the CSR matrices, which at 128^3 hold 1.6 GB (Fx, Fy, Fz) and
// 12.2 GB (F_el):
//
// * cpm_stencil_deriv  mode 0: Hd = alpha (Fx U, Fy U, Fz U)  (compute_derivatives.py:36-58)
//                      mode 1: b = alpha sum_i F_i (m_i - <m>_i), b[pin] = 0  (Micromagnetics.py:166-168)
// * cpm_stencil_strain  E (n,6) from u = [ux|uy|uz], optionally rotated by R
//                       (compute_derivatives.py:60-125)
// * cpm_stencil_fel     b_el = F_el E0, E0 node-interleaved (6n), b_el [x|y|z] (Micromagnetics.py:123),
//                       with the reference's empty anchor rows 0, n, 2n
//                       (assemble_elasticity.py:461-527)
//
// Every product is FP64 with the coefficients in the launch parameters
// (constant bank operands of the FMAs), so all three are bound by GB300's FP64
// pipe (about 2 FP64 operations per clock per SM); a few warps per SM keep it
// busy, so the kernels use the registers they need (no occupancy cap).
//
// On a cell with mirror symmetry (every hex cell here) the stencil of F_x is odd in dx and even in dy and dz, and
// likewise for F_y and F_z: 4 distinct coefficients each.  A block then holds a tile of columns and marches along x
// (mirror_kernel): differences along the odd axis first, sums along the even ones, and a plane's sums serve its own
// outputs and its x neighbours'.  FP64 operations per node: Hd 55 -> 30, demag right-hand side 79 -> 30 (the mean
// shift cancels in the differences), strain 186 -> 121 with the rotation.  F_el = B^T C S factors into the stress
// sigma = C E0 (6 x 6, once per node of the tile and its rim) and its divergence, b_a = sum_j F_j sigma_aj:
// 312 -> 143.  (The shape tables are rounded to 12 decimals, so the stencils are not products of 1-D stencils to
// rounding; the parities and the factor C are exact to 1e-16.)  Measured on GB300 at 128^3,
// us pairs / march: F_el 1248 / 653, strain 747 / 558, right-hand side 325 / 143, Hd 222 / 156; the FP64 pipe is
// 80 % busy.
//
// Other stencils: those odd in the offset, c(-d) = -c(d) with c(0) = 0, take each pair of opposite neighbours once,
// as the difference of the two gathered values times the odd part (c(d) - c(-d)) / 2, for every output; the rest
// sums all 27 neighbours in lexicographic offset order.  The host checks the caller's coefficients (mirror form and
// factor to 1e-15 of the largest, oddness to 1e-12).  Results agree with the CSR products to rounding.
#include <algorithm>
#include <cmath>

#include "stencil_ops.cuh"

namespace cpm {

constexpr int kDerivThreads = 256;

struct DerivArgs {
  int nx, ny, nz, n;
  const uint8_t *flags;  // unused (neighbours() takes any record with these fields)
  double f[3][27];
  double h[3][13];       // odd part (f[d] - f[26 - d]) / 2 of offsets d < 13 (the pair d, 26 - d)
};

struct FelArgs {
  int nx, ny, nz, n;
  const uint8_t *flags;
  int anchor;
  double c[3 * 6 * 27];
  double h[3 * 6 * 13];  // odd part, as DerivArgs::h, per (output, input)
};

// The neighbours d and 26 - d (opposite offsets) of a DOF with wrapped offsets b, d < 13.
__device__ __forceinline__ void pair_nodes(const Nbr &b, int d, int &qp, int &qm) {
  const int ia = d / 9, ib = (d / 3) % 3, ic = d % 3;
  qp = b.xi[ia] + b.yj[ib] + b.zk[ic];
  qm = b.xi[2 - ia] + b.yj[2 - ib] + b.zk[2 - ic];
}

static inline int64_t deriv_grid(int64_t n) {
  const int64_t cap = (int64_t)sm_count() * 8;
  return std::max<int64_t>(1, std::min<int64_t>((n + kDerivThreads - 1) / kDerivThreads, cap));
}

// ---------------------------------------------------------------- Hd and the demag right-hand side
template <int MODE, bool ODD>
__global__ void __launch_bounds__(kDerivThreads) deriv_kernel(const __grid_constant__ DerivArgs a,
                                                              const double *__restrict__ x, double *__restrict__ y,
                                                              double alpha, const double *shift, int64_t pin) {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  if (MODE == 1 && shift) {
    s0 = shift[0];
    s1 = shift[1];
    s2 = shift[2];
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < a.n; p += stride) {
    const Nbr b = neighbours(a, (int)p);
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    if (ODD) {
#pragma unroll
      for (int d = 0; d < 13; ++d) {
        int qp, qm;
        pair_nodes(b, d, qp, qm);
        if (MODE == 0) {
          const double v = __ldg(x + qp) - __ldg(x + qm);
          acc0 = fma(a.h[0][d], v, acc0);
          acc1 = fma(a.h[1][d], v, acc1);
          acc2 = fma(a.h[2][d], v, acc2);
        } else {
          acc0 = fma(a.h[0][d], __ldg(x + 3 * (int64_t)qp + 0) - __ldg(x + 3 * (int64_t)qm + 0), acc0);
          acc1 = fma(a.h[1][d], __ldg(x + 3 * (int64_t)qp + 1) - __ldg(x + 3 * (int64_t)qm + 1), acc1);
          acc2 = fma(a.h[2][d], __ldg(x + 3 * (int64_t)qp + 2) - __ldg(x + 3 * (int64_t)qm + 2), acc2);
        }
      }
    }
#pragma unroll
    for (int ia = 0; ia < 3; ++ia)
#pragma unroll
      for (int ib = 0; ib < 3; ++ib)
#pragma unroll
        for (int ic = 0; ic < 3; ++ic) {
          if (ODD) continue;
          const int q = b.xi[ia] + b.yj[ib] + b.zk[ic];
          const int d = (ia * 3 + ib) * 3 + ic;
          if (MODE == 0) {
            const double v = __ldg(x + q);
            acc0 = fma(a.f[0][d], v, acc0);
            acc1 = fma(a.f[1][d], v, acc1);
            acc2 = fma(a.f[2][d], v, acc2);
          } else {
            acc0 = fma(a.f[0][d], __ldg(x + 3 * (int64_t)q + 0) - s0, acc0);
            acc1 = fma(a.f[1][d], __ldg(x + 3 * (int64_t)q + 1) - s1, acc1);
            acc2 = fma(a.f[2][d], __ldg(x + 3 * (int64_t)q + 2) - s2, acc2);
          }
        }
    if (MODE == 0) {
      y[3 * p + 0] = alpha * acc0;
      y[3 * p + 1] = alpha * acc1;
      y[3 * p + 2] = alpha * acc2;
    } else {
      y[p] = p == pin ? 0.0 : alpha * ((acc0 + acc1) + acc2);
    }
  }
}

// ---------------------------------------------------------------- strain from u
// Voigt strain of the nine derivatives d_a u_b, rotated with the association of the reference's rotated strain
// (compute_derivatives.py:94-123); R[r][c] = R[3 r + c].
__device__ __forceinline__ void strain_voigt(bool rot, const double (&R)[9], double dxx, double dyx, double dzx,
                                             double dxy, double dyy, double dzy, double dxz, double dyz, double dzz,
                                             double (&out)[6]) {
  if (!rot) {
    out[0] = dxx;
    out[1] = dyy;
    out[2] = dzz;
    out[3] = dyx + dxy;
    out[4] = dzy + dyz;
    out[5] = dzx + dxz;
    return;
  }
  out[0] = (R[0] * dxx + R[3] * dyx) + R[6] * dzx;
  out[1] = (R[1] * dxy + R[4] * dyy) + R[7] * dzy;
  out[2] = (R[2] * dxz + R[5] * dyz) + R[8] * dzz;
  out[3] = ((R[1] * dxx + R[4] * dyx) + R[7] * dzx) + ((R[0] * dxy + R[3] * dyy) + R[6] * dzy);
  out[4] = ((R[2] * dxy + R[5] * dyy) + R[8] * dzy) + ((R[1] * dxz + R[4] * dyz) + R[7] * dzz);
  out[5] = ((R[2] * dxx + R[5] * dyx) + R[8] * dzx) + ((R[0] * dxz + R[3] * dyz) + R[6] * dzz);
}

template <bool ODD>
__global__ void __launch_bounds__(kDerivThreads) strain_stencil_kernel(const __grid_constant__ DerivArgs a,
                                                                       const double *__restrict__ u,
                                                                       const double *R9, double *__restrict__ E) {
  const int64_t n = a.n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double R[9];
  if (R9) {
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] = R9[k];
  }
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const Nbr b = neighbours(a, (int)p);
    double d[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};  // d[a][b] = (F_a u_b)_p
    if (ODD) {
#pragma unroll
      for (int s = 0; s < 13; ++s) {
        int qp, qm;
        pair_nodes(b, s, qp, qm);
        const double uu[3] = {__ldg(u + qp) - __ldg(u + qm), __ldg(u + n + qp) - __ldg(u + n + qm),
                              __ldg(u + 2 * n + qp) - __ldg(u + 2 * n + qm)};
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int c = 0; c < 3; ++c) d[k][c] = fma(a.h[k][s], uu[c], d[k][c]);
      }
    }
#pragma unroll
    for (int ia = 0; ia < 3 && !ODD; ++ia)
#pragma unroll
      for (int ib = 0; ib < 3; ++ib)
#pragma unroll
        for (int ic = 0; ic < 3; ++ic) {
          const int q = b.xi[ia] + b.yj[ib] + b.zk[ic];
          const int s = (ia * 3 + ib) * 3 + ic;
          const double uu[3] = {__ldg(u + q), __ldg(u + n + q), __ldg(u + 2 * n + q)};
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c) d[k][c] = fma(a.f[k][s], uu[c], d[k][c]);
        }
    double out[6];
    strain_voigt(R9 != nullptr, R, d[0][0], d[1][0], d[2][0], d[0][1], d[1][1], d[2][1], d[0][2], d[1][2], d[2][2],
                 out);
    double2 *e2 = reinterpret_cast<double2 *>(E + 6 * p);
    e2[0] = make_double2(out[0], out[1]);
    e2[1] = make_double2(out[2], out[3]);
    e2[2] = make_double2(out[4], out[5]);
  }
}

// ---------------------------------------------------------------- b_el = F_el E0
template <bool ODD>
__global__ void __launch_bounds__(kDerivThreads, 3) fel_stencil_kernel(const __grid_constant__ FelArgs a,
                                                                    const double *__restrict__ E0,
                                                                    double *__restrict__ y) {
  const int64_t n = a.n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    double acc[3] = {0.0, 0.0, 0.0};
    if (ODD && !(a.anchor && p == 0)) {
      const Nbr b = neighbours(a, (int)p);
#pragma unroll
      for (int d = 0; d < 13; ++d) {
        int qp, qm;
        pair_nodes(b, d, qp, qm);
        const double2 *ep = reinterpret_cast<const double2 *>(E0 + 6 * (int64_t)qp);
        const double2 *em = reinterpret_cast<const double2 *>(E0 + 6 * (int64_t)qm);
        const double2 p01 = __ldg(ep), p23 = __ldg(ep + 1), p45 = __ldg(ep + 2);
        const double2 m01 = __ldg(em), m23 = __ldg(em + 1), m45 = __ldg(em + 2);
        const double v[6] = {p01.x - m01.x, p01.y - m01.y, p23.x - m23.x, p23.y - m23.y, p45.x - m45.x, p45.y - m45.y};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int k = 0; k < 6; ++k) acc[r] = fma(a.h[(r * 6 + k) * 13 + d], v[k], acc[r]);
      }
    } else if (!(a.anchor && p == 0)) {
      const Nbr b = neighbours(a, (int)p);
#pragma unroll
      for (int ia = 0; ia < 3; ++ia)
#pragma unroll
        for (int ib = 0; ib < 3; ++ib)
#pragma unroll
          for (int ic = 0; ic < 3; ++ic) {
            const int q = b.xi[ia] + b.yj[ib] + b.zk[ic];
            const int d = (ia * 3 + ib) * 3 + ic;
            const double2 *e = reinterpret_cast<const double2 *>(E0 + 6 * (int64_t)q);
            const double2 v01 = __ldg(e), v23 = __ldg(e + 1), v45 = __ldg(e + 2);
            const double v[6] = {v01.x, v01.y, v23.x, v23.y, v45.x, v45.y};
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
              for (int k = 0; k < 6; ++k) acc[r] = fma(a.c[(r * 6 + k) * 27 + d], v[k], acc[r]);
          }
    }
    y[p] = acc[0];
    y[n + p] = acc[1];
    y[2 * n + p] = acc[2];
  }
}

// ---------------------------------------------------------------- mirror-symmetric stencils
// Fx at dx = +1: p[2 |dy| + |dz|]; Fy at dy = +1: q[2 |dx| + |dz|]; Fz at dz = +1: r[2 |dx| + |dy|].
struct Mirror {
  double p[4], q[4], r[4];
};

// A block of up to kTileThreads threads holds a ty x tz tile of columns and marches along x.
struct MirrorArgs {
  int nx, ny, nz, lx, ty, tz, ntz, anchor;
  Mirror c;
  double C[6][6];  // MODE 3: stress xx yy zz xy yz xz per unit eigenstrain component
};

constexpr int kTileThreads = 256;
constexpr double kPipeUs = 0.0096;  // of an SM's FP64 pipe per warp instruction: 16 cycles, at 80 to 90 % of them busy
constexpr int kTileRim = 350;  // nodes of a tile with its rim at most

// Parts of a field's derivatives from its values t (shared memory, z-lines of w): Fx from the x difference of
// the field, Fy and Fz at the node's own plane (c) and to both x neighbours (s).  Differences come first: on a
// field that is nearly constant (m, E0) sums first would lose what the difference keeps.
__device__ __forceinline__ double part_x(const Mirror &m, const double *t, int w) {
  const double u0 = t[w - 1] + t[-w - 1], u1 = t[w] + t[-w], u2 = t[w + 1] + t[-w + 1];
  return fma(m.p[3], u2 + u0, fma(m.p[2], u1, fma(m.p[1], t[1] + t[-1], m.p[0] * t[0])));
}
__device__ __forceinline__ void part_y(const Mirror &m, const double *t, int w, bool own, double &c, double &s) {
  const double d = t[w] - t[-w], e = (t[w + 1] - t[-w + 1]) + (t[w - 1] - t[-w - 1]);
  if (own) c = fma(m.q[1], e, fma(m.q[0], d, c));
  s = fma(m.q[3], e, fma(m.q[2], d, s));
}
__device__ __forceinline__ void part_z(const Mirror &m, const double *t, int w, bool own, double &c, double &s) {
  const double d = t[1] - t[-1], e = (t[w + 1] - t[w - 1]) + (t[-w + 1] - t[-w - 1]);
  if (own) c = fma(m.r[1], e, fma(m.r[0], d, c));
  s = fma(m.r[3], e, fma(m.r[2], d, s));
}

// MODE 0: y (n,3) = alpha (Fx x, Fy x, Fz x); 1: y (n) = alpha div x for x (n,3), 0 at pin; 2: E (n,6) from
// u (3n), rotated by R9 where that is set; 3: b_el = div (C E0).
// Per plane i the block publishes the fields' values and, for those that enter Fx, the differences
// W(i - 1) = v(i) - v(i - 2) of the tile and its rim (two buffers: one block barrier per plane), each formed once
// per node; a thread's outputs are those of plane i - 1.
template <int MODE>
struct MirrorShape {
  static constexpr int V = MODE == 0 ? 1 : MODE == 3 ? 6 : 3;   // fields
  static constexpr int W = MODE == 0 ? 1 : MODE == 1 ? 1 : 3;   // fields that enter Fx
  static constexpr int O = MODE == 0 ? 2 : MODE == 1 ? 1 : MODE == 2 ? 6 : 3;  // sums along the march
};

template <int MODE>
__global__ void __launch_bounds__(kTileThreads, 2) mirror_kernel(const __grid_constant__ MirrorArgs a,
                                                                 const double *__restrict__ x, double *__restrict__ y,
                                                                 double alpha, int64_t pin, const double *R9) {
  using Sh = MirrorShape<MODE>;
  // field slots: MODE 1 keeps m_y, m_z; MODE 3 the stresses yy zz xy yz xz; differences: x, m_x, u, (xx xy xz)
  constexpr int NF = MODE == 0 ? 1 : MODE == 1 ? 2 : MODE == 2 ? 3 : 5;
  __shared__ double sm[2][NF + Sh::W][kTileRim];
  const int nyz = a.ny * a.nz;
  const int64_t n = (int64_t)a.nx * nyz;
  const int tj = blockIdx.x / a.ntz, j0 = tj * a.ty, k0 = (blockIdx.x - tj * a.ntz) * a.tz;
  const int ty = min(a.ty, a.ny - j0), tz = min(a.tz, a.nz - k0), w = tz + 2, rim = (ty + 2) * w;
  const int x0 = blockIdx.y * a.lx, x1 = min(a.nx, x0 + a.lx), tid = threadIdx.x;
  const bool mine = tid < ty * tz;
  const int lj = tid / tz, lk = tid - lj * tz, f = (j0 + lj) * a.nz + k0 + lk, at = (lj + 1) * w + lk + 1;
  int node[2];  // the plane's nodes that this thread publishes
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int e = min(tid + h * kTileThreads, rim - 1), ej = e / w;
    int j = j0 + ej - 1, k = k0 + e - ej * w - 1;
    j = j < 0 ? a.ny - 1 : j >= a.ny ? 0 : j;
    k = k < 0 ? a.nz - 1 : k >= a.nz ? 0 : k;
    node[h] = j * a.nz + k;
  }
  double R[9];
  if (MODE == 2 && R9) {
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] = R9[k];
  }
  double v1[2][Sh::W], v2[2][Sh::W];  // the nodes' values at planes i - 1, i - 2
  double acc[Sh::O], side[Sh::O];
#pragma unroll
  for (int o = 0; o < Sh::O; ++o) acc[o] = side[o] = 0.0;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int k = 0; k < Sh::W; ++k) v1[h][k] = v2[h][k] = 0.0;
  for (int i = x0 - 1; i <= x1; ++i) {
    const int64_t plane = (int64_t)(i < 0 ? a.nx - 1 : i >= a.nx ? 0 : i) * nyz;
    double(*t)[kTileRim] = sm[i & 1];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = tid + h * kTileThreads;
      if (e >= rim) continue;
      const int64_t g = plane + node[h];
      double v[Sh::V], d[Sh::W];
      if (MODE == 0) {
        v[0] = __ldg(x + g);
      } else if (MODE == 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = __ldg(x + 3 * g + k);
      } else if (MODE == 2) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = __ldg(x + k * n + g);
      } else {
        const double2 *p = reinterpret_cast<const double2 *>(x + 6 * g);
        const double2 g01 = __ldg(p), g23 = __ldg(p + 1), g45 = __ldg(p + 2);
#pragma unroll
        for (int r = 0; r < 6; ++r)
          v[r] = fma(a.C[r][5], g45.y, fma(a.C[r][4], g45.x, fma(a.C[r][3], g23.y, fma(a.C[r][2], g23.x,
                 fma(a.C[r][1], g01.y, a.C[r][0] * g01.x)))));
      }
      constexpr int wf[3] = {0, MODE == 3 ? 3 : 1, MODE == 3 ? 5 : 2};  // the fields that enter Fx
#pragma unroll
      for (int k = 0; k < Sh::W; ++k) {
        d[k] = v[wf[k]] - v2[h][k];
        v2[h][k] = v1[h][k];
        v1[h][k] = v[wf[k]];
        t[NF + k][e] = d[k];
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) t[k][e] = v[MODE == 0 || MODE == 2 ? k : k + 1];
    }
    __syncthreads();
    if (!mine) continue;
    const bool own = i >= x0 && i < x1, out = i > x0;
    double c[Sh::O], s[Sh::O];
#pragma unroll
    for (int o = 0; o < Sh::O; ++o) c[o] = s[o] = 0.0;
    const int64_t o = (int64_t)(i - 1) * nyz + f;
    if (MODE == 0) {
      part_y(a.c, t[0] + at, w, own, c[0], s[0]);
      part_z(a.c, t[0] + at, w, own, c[1], s[1]);
      if (out) {
        double *q = y + 3 * o;
        q[0] = alpha * part_x(a.c, t[1] + at, w);
        q[1] = alpha * (acc[0] + s[0]);
        q[2] = alpha * (acc[1] + s[1]);
      }
    } else if (MODE == 1) {
      part_y(a.c, t[0] + at, w, own, c[0], s[0]);
      part_z(a.c, t[1] + at, w, own, c[0], s[0]);
      if (out) y[o] = o == pin ? 0.0 : alpha * ((acc[0] + s[0]) + part_x(a.c, t[2] + at, w));
    } else if (MODE == 2) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        part_y(a.c, t[k] + at, w, own, c[2 * k], s[2 * k]);
        part_z(a.c, t[k] + at, w, own, c[2 * k + 1], s[2 * k + 1]);
      }
      if (out) {
        double E[6];
        strain_voigt(R9 != nullptr, R, part_x(a.c, t[3] + at, w), acc[0] + s[0], acc[1] + s[1],
                     part_x(a.c, t[4] + at, w), acc[2] + s[2], acc[3] + s[3], part_x(a.c, t[5] + at, w),
                     acc[4] + s[4], acc[5] + s[5], E);
        double2 *e2 = reinterpret_cast<double2 *>(y + 6 * o);
        e2[0] = make_double2(E[0], E[1]);
        e2[1] = make_double2(E[2], E[3]);
        e2[2] = make_double2(E[4], E[5]);
      }
    } else {
      part_y(a.c, t[2] + at, w, own, c[0], s[0]);  // xy, xz
      part_z(a.c, t[4] + at, w, own, c[0], s[0]);
      part_y(a.c, t[0] + at, w, own, c[1], s[1]);  // yy, yz
      part_z(a.c, t[3] + at, w, own, c[1], s[1]);
      part_y(a.c, t[3] + at, w, own, c[2], s[2]);  // yz, zz
      part_z(a.c, t[1] + at, w, own, c[2], s[2]);
      if (out) {
        const bool zero = a.anchor && o == 0;
#pragma unroll
        for (int k = 0; k < 3; ++k)  // xx, xy, xz
          y[k * n + o] = zero ? 0.0 : (acc[k] + s[k]) + part_x(a.c, t[NF + k] + at, w);
      }
    }
#pragma unroll
    for (int k = 0; k < Sh::O; ++k) {
      acc[k] = c[k] + side[k];
      side[k] = s[k];
    }
  }
}

// Tile and planes per block.  Tile: the fewest FP64 warp instructions (`out` per output, `rim` per node of the tile
// and its rim).  Planes: the blocks of one SM run one after the other on its FP64 pipe, and the two rim planes of a
// range cost about 0.8 of an output plane.
// Returns the march's time by that model in us (see march_pays), negative where the grid has no tile.
static double mirror_shape(MirrorArgs &m, double out, double rim) {
  double best = 1e300, plane = 0.0;
  for (int nt = 1; nt <= m.nz; ++nt) {
    const int z = (m.nz + nt - 1) / nt;
    if (z > 128) continue;
    if (z < 3 && nt > 1) break;
    int t = std::min(std::min(kTileThreads / z, kTileRim / (z + 2) - 2), m.ny);
    if (t < 1) continue;
    t = (m.ny + (m.ny + t - 1) / t - 1) / ((m.ny + t - 1) / t);
    const double block = (t * z + 31) / 32 * out + ((t + 2) * (z + 2) + 31) / 32 * rim;
    const double cost = (double)((m.nz + z - 1) / z) * ((m.ny + t - 1) / t) * block;
    if (cost < best) {
      best = cost;
      plane = block;
      m.tz = z;
      m.ty = t;
    }
  }
  if (best >= 1e300) return -1.0;
  m.ntz = (m.nz + m.tz - 1) / m.tz;
  const int64_t tiles = (int64_t)m.ntz * ((m.ny + m.ty - 1) / m.ty);
  const int sms = sm_count();
  double us = 0.0;
  best = 1e300;
  for (int nr = 1; nr <= m.nx && nr <= 65535; ++nr) {
    const int l = (m.nx + nr - 1) / nr;
    const int64_t per = (tiles * ((m.nx + l - 1) / l) + sms - 1) / sms;
    const double cost = (double)per * (l + 0.8) + (per < 2 ? 0.5 * l : 0.0);
    if (cost < best) {
      best = cost;
      m.lx = l;
      us = kPipeUs * 1.07 * per * (l + 0.8) * plane + 0.4 * (l + 2);
    }
  }
  return tiles < (1ll << 31) ? us : -1.0;
}

// Whether a march of `us` (mirror_shape) and `start` us to begin with beats the pair kernel of `ops` FP64 operations
// per node: both wait on the FP64 pipe, the pair kernel in whole rounds of one 256-node block per SM, the march in
// blocks per SM times planes, plus 0.4 us a plane of latency.  Within 10 % of the times measured on GB300 on 70 grids
// from 8^3 to 128^3, among them films and bars (3x200x140, 600x600x4, 512x8x8), and never the slower form by more
// than 2 % there.  Us, pairs / march: F_el 25x27x29 25.2 / 27.9, 38^3 48.6 / 52.4, 40^3 48.6 / 33.2, 128^3 1248 / 653;
// strain 53^3 70.6 / 75.2, 64^3 98.1 / 91.7, 64x512x5 70.7 / 73.4, 256x4x256 98.1 / 75.1; right-hand side 20^3
// 7.7 / 7.2, 33x31x35 7.9 / 11.1, 128^3 325 / 143; Hd 53^3 22.2 / 23.9, 64^3 30.4 / 27.9, 128^3 222 / 156.
static bool march_pays(double us, double start, int64_t n, double ops) {
  const int64_t rounds = ((n + kDerivThreads - 1) / kDerivThreads + sm_count() - 1) / std::max(1, sm_count());
  const double warps = (double)std::min<int64_t>(kDerivThreads / 32, (n + 31) / 32);
  return us >= 0.0 && n >= kDerivThreads && us + start < kPipeUs * rounds * warps * ops + 1.0;
}

// The part of a 27-point stencil odd along `axis` and even along the other two, c[2 b + c] at the axis' +1
// (b, c: |offset| along the others in order); false unless that is all of it, to 1e-15 of `big`.
static bool mirror_part(const double *v, int axis, double big, double *out) {
  const double tol = 1e-15 * big;
  if (!std::isfinite(tol)) return false;
  double sum[4] = {0, 0, 0, 0};
  for (int d = 0; d < 27; ++d) {
    const int o[3] = {d / 9 - 1, (d / 3) % 3 - 1, d % 3 - 1};
    const int e1 = o[axis == 0 ? 1 : 0] != 0, e2 = o[axis == 2 ? 1 : 2] != 0;
    if (o[axis] == 0) {
      if (!(std::fabs(v[d]) <= tol)) return false;  // (not a number fails)
    } else {
      sum[2 * e1 + e2] += o[axis] * v[d] / (2.0 * (e1 ? 2 : 1) * (e2 ? 2 : 1));
    }
  }
  for (int d = 0; d < 27; ++d) {
    const int o[3] = {d / 9 - 1, (d / 3) % 3 - 1, d % 3 - 1};
    const int e1 = o[axis == 0 ? 1 : 0] != 0, e2 = o[axis == 2 ? 1 : 2] != 0;
    if (o[axis] != 0 && !(std::fabs(v[d] - o[axis] * sum[2 * e1 + e2]) <= tol)) return false;
  }
  for (int e = 0; e < 4; ++e) out[e] = sum[e];
  return true;
}

static double largest(const double *v, int count) {
  double big = 0.0;
  for (int d = 0; d < count; ++d) big = std::max(big, std::fabs(v[d]));
  return big;
}

static bool mirror_deriv(const cpm_deriv_stencil *D, MirrorArgs &m, double out, double rim, double start, double ops) {
  m = MirrorArgs{};
  m.nx = D->nx;
  m.ny = D->ny;
  m.nz = D->nz;
  return march_pays(mirror_shape(m, out, rim), start, (int64_t)D->nx * D->ny * D->nz, ops) &&
         mirror_part(D->fx, 0, largest(D->fx, 27), m.c.p) && mirror_part(D->fy, 1, largest(D->fy, 27), m.c.q) &&
         mirror_part(D->fz, 2, largest(D->fz, 27), m.c.r);
}

template <int MODE>
static void launch_mirror(const MirrorArgs &m, const double *x, double *y, double alpha, int64_t pin, const double *R9,
                          void *stream) {
  const dim3 grid((unsigned)(m.ntz * ((m.ny + m.ty - 1) / m.ty)), (unsigned)((m.nx + m.lx - 1) / m.lx));
  mirror_kernel<MODE><<<grid, kTileThreads, 0, (cudaStream_t)stream>>>(m, x, y, alpha, pin, R9);
}

// F_el as divergence of a stress: every (a, v) block is sum_j C[(a j)][v] F_j with the unit stencils F_j (1 at the
// axis' +1) and a stress symmetric in (a, j).
static bool mirror_fel(const cpm_fel_stencil *F, MirrorArgs &m) {
  m = MirrorArgs{};
  m.nx = F->nx;
  m.ny = F->ny;
  m.nz = F->nz;
  m.anchor = F->anchor ? 1 : 0;
  // one plane per block would form every stress three times
  if (!march_pays(mirror_shape(m, 87.0, 39.0), 2.5, (int64_t)m.nx * m.ny * m.nz, 312.0) || m.lx < 2) return false;
  const double big = largest(F->coef, 486);
  if (!(big > 0.0) || !std::isfinite(big)) return false;
  const double tol = 1e-15 * big;
  // parts of every block: odd along one axis, even along the others
  double part[3][3][6][4];  // [axis][a][v]
  for (int a = 0; a < 3; ++a)
    for (int v = 0; v < 6; ++v) {
      const double *c = F->coef + (a * 6 + v) * 27;
      double rest[27];
      for (int d = 0; d < 27; ++d) rest[d] = c[d];
      for (int ax = 0; ax < 3; ++ax) {
        double *q = part[ax][a][v];
        for (int e = 0; e < 4; ++e) q[e] = 0.0;
        for (int pass = 0; pass < 2; ++pass)
          for (int d = 0; d < 27; ++d) {
            const int o[3] = {d / 9 - 1, (d / 3) % 3 - 1, d % 3 - 1};
            const int e1 = o[ax == 0 ? 1 : 0] != 0, e2 = o[ax == 2 ? 1 : 2] != 0;
            if (o[ax] == 0) continue;
            if (pass == 0) q[2 * e1 + e2] += o[ax] * c[d] / (2.0 * (e1 ? 2 : 1) * (e2 ? 2 : 1));
            else rest[d] -= o[ax] * q[2 * e1 + e2];
          }
      }
      for (int d = 0; d < 27; ++d)
        if (!(std::fabs(rest[d]) <= tol)) return false;
    }
  const int voigt[3][3] = {{0, 3, 5}, {3, 1, 4}, {5, 4, 2}};
  double *unit[3] = {m.c.p, m.c.q, m.c.r};
  for (int ax = 0; ax < 3; ++ax) {
    int ba = 0, bv = 0;
    for (int a = 0; a < 3; ++a)
      for (int v = 0; v < 6; ++v)
        if (std::fabs(part[ax][a][v][0]) > std::fabs(part[ax][ba][bv][0])) ba = a, bv = v;
    const double lead = part[ax][ba][bv][0];
    if (lead == 0.0) return false;
    for (int e = 0; e < 4; ++e) unit[ax][e] = part[ax][ba][bv][e] / lead;
    for (int a = 0; a < 3; ++a)
      for (int v = 0; v < 6; ++v) {
        for (int e = 0; e < 4; ++e)
          if (!(std::fabs(part[ax][a][v][e] - part[ax][a][v][0] * unit[ax][e]) <= tol)) return false;
        double &c = m.C[voigt[a][ax]][v];
        if (a < ax) c = part[ax][a][v][0];                     // (a, ax) first seen from the smaller index
        else if (a == ax) c = part[ax][a][v][0];
        else if (!(std::fabs(part[ax][a][v][0] - part[a][ax][v][0]) <= tol)) return false;
      }
  }
  return true;
}

static bool grid_ok(int nx, int ny, int nz, int64_t parts) {
  return nx >= 3 && ny >= 3 && nz >= 3 && (int64_t)nx * ny * nz * parts < ((int64_t)1 << 31);
}

static DerivArgs deriv_args(const cpm_deriv_stencil *D) {
  DerivArgs a{};
  a.nx = D->nx;
  a.ny = D->ny;
  a.nz = D->nz;
  a.n = D->nx * D->ny * D->nz;
  a.flags = nullptr;
  for (int d = 0; d < 27; ++d) {
    a.f[0][d] = D->fx[d];
    a.f[1][d] = D->fy[d];
    a.f[2][d] = D->fz[d];
  }
  for (int k = 0; k < 3; ++k)
    for (int d = 0; d < 13; ++d) a.h[k][d] = 0.5 * (a.f[k][d] - a.f[k][26 - d]);
  return a;
}

// Whether each run of 27 coefficients is odd in the offset (to 1e-12 of its largest magnitude).
static bool stencils_odd(const double *c, int count) {
  for (int s = 0; s < count; ++s) {
    const double *v = c + 27 * s;
    double big = 0.0;
    for (int d = 0; d < 27; ++d) big = std::max(big, std::fabs(v[d]));
    const double tol = 1e-12 * big;
    if (std::fabs(v[13]) > tol) return false;
    for (int d = 0; d < 13; ++d)
      if (std::fabs(v[d] + v[26 - d]) > tol) return false;
  }
  return true;
}

}  // namespace cpm

extern "C" int cpm_stencil_deriv(const cpm_deriv_stencil *D, const double *x, double *y, double alpha, int mode,
                                 const double *shift, int64_t pin, void *stream) {
  using namespace cpm;
  if (!D || !x || !y || (mode != 0 && mode != 1) || !grid_ok(D->nx, D->ny, D->nz, 6)) {
    set_error("cpm_stencil_deriv: bad arguments (at least 3 cells per axis, mode 0 or 1)");
    return CPM_BAD_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  MirrorArgs m;
  if (mode == 0 ? mirror_deriv(D, m, 29.0, 1.0, 2.5, 55.0) : mirror_deriv(D, m, 28.0, 1.0, 1.5, 79.0)) {
    if (mode == 0) launch_mirror<0>(m, x, y, alpha, -1, nullptr, stream);
    else launch_mirror<1>(m, x, y, alpha, pin, nullptr, stream);
    return check_launch("cpm_stencil_deriv");
  }
  const DerivArgs a = deriv_args(D);
  const int g = (int)deriv_grid(a.n);
  const bool odd = stencils_odd(&a.f[0][0], 3);
  if (mode == 0) {
    if (odd) deriv_kernel<0, true><<<g, kDerivThreads, 0, st>>>(a, x, y, alpha, nullptr, -1);
    else deriv_kernel<0, false><<<g, kDerivThreads, 0, st>>>(a, x, y, alpha, nullptr, -1);
  } else {
    if (odd) deriv_kernel<1, true><<<g, kDerivThreads, 0, st>>>(a, x, y, alpha, shift, pin);
    else deriv_kernel<1, false><<<g, kDerivThreads, 0, st>>>(a, x, y, alpha, shift, pin);
  }
  return check_launch("cpm_stencil_deriv");
}

extern "C" int cpm_stencil_strain(const cpm_deriv_stencil *D, const double *u, const double *R9, double *E,
                                  void *stream) {
  using namespace cpm;
  if (!D || !u || !E || ((uintptr_t)E & 15) || !grid_ok(D->nx, D->ny, D->nz, 6)) {
    set_error("cpm_stencil_strain: bad arguments (at least 3 cells per axis, 16-byte aligned E)");
    return CPM_BAD_ARG;
  }
  MirrorArgs m;
  if (mirror_deriv(D, m, 117.0, 3.0, 2.5, 186.0)) {
    launch_mirror<2>(m, u, E, 1.0, -1, R9, stream);
    return check_launch("cpm_stencil_strain");
  }
  const DerivArgs a = deriv_args(D);
  const int g = (int)deriv_grid(a.n);
  if (stencils_odd(&a.f[0][0], 3))
    strain_stencil_kernel<true><<<g, kDerivThreads, 0, (cudaStream_t)stream>>>(a, u, R9, E);
  else
    strain_stencil_kernel<false><<<g, kDerivThreads, 0, (cudaStream_t)stream>>>(a, u, R9, E);
  return check_launch("cpm_stencil_strain");
}

extern "C" int cpm_stencil_fel(const cpm_fel_stencil *F, const double *E0, double *b_el, void *stream) {
  using namespace cpm;
  if (!F || !E0 || !b_el || ((uintptr_t)E0 & 15) || !grid_ok(F->nx, F->ny, F->nz, 6)) {
    set_error("cpm_stencil_fel: bad arguments (at least 3 cells per axis, 16-byte aligned E0)");
    return CPM_BAD_ARG;
  }
  MirrorArgs m;
  if (mirror_fel(F, m)) {
    launch_mirror<3>(m, E0, b_el, 1.0, -1, nullptr, stream);
    return check_launch("cpm_stencil_fel");
  }
  FelArgs a{};
  a.nx = F->nx;
  a.ny = F->ny;
  a.nz = F->nz;
  a.n = F->nx * F->ny * F->nz;
  a.flags = nullptr;
  a.anchor = F->anchor ? 1 : 0;
  for (int i = 0; i < 3 * 6 * 27; ++i) a.c[i] = F->coef[i];
  for (int s = 0; s < 18; ++s)
    for (int d = 0; d < 13; ++d) a.h[s * 13 + d] = 0.5 * (a.c[s * 27 + d] - a.c[s * 27 + 26 - d]);
  const int g = (int)deriv_grid(a.n);
  if (stencils_odd(a.c, 18))
    fel_stencil_kernel<true><<<g, kDerivThreads, 0, (cudaStream_t)stream>>>(a, E0, b_el);
  else
    fel_stencil_kernel<false><<<g, kDerivThreads, 0, (cudaStream_t)stream>>>(a, E0, b_el);
  return check_launch("cpm_stencil_fel");
}
