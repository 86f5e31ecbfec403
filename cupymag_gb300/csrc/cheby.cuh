// Chebyshev iteration on the scalar hex stencils of the projection solves
// (A1, A2), shared by the single-system solver (stencil.cu) and the
// block-diagonal one (batched.cu).
//
// The refinement form of the cupyx-semantics solve_cg
// (cupymag/solvers/linear_solvers.py:59-74): an outer loop decides
// ||b - A x|| <= tol ||b|| on an FP64 or proven double-float residual, and each
// of its cycles reduces that residual by FP32 steps with FP32 coefficients.
// Here the steps are Chebyshev's in place of CG's.  On the free DOFs A is a
// principal submatrix of the circulant stencil operator, so its eigenvalues lie
// between the minimum and the maximum of the symbol (both at corners of the
// torus for a stencil even along every axis): with that interval known, the
// three-term recurrence
//     x_{k+1} = x_k + w_k (x_k - x_{k-1}) + g_k (r - A x_k)
// needs no inner products.  One pass per step reads x_k (27 neighbours), x_{k-1}
// and r and writes x_{k+1} over x_{k-1}: 16 bytes per unknown and one grid
// barrier, where a CG iteration moves 44 bytes through three barriers and two
// grid reductions.  The number of steps of a cycle follows from the reduction
// it needs, ||r_k|| <= ||r_0|| / T_k; A1 and A2 (condition numbers 10.5 and
// 23.3) take 40 and 60 steps from a cold start to tol 1e-10, CG 28-36 and 41-55.
// Measured on GB300, us per cold solve, CG / this: A1 x 3 at 128^3 3500 / 960,
// at 112 x 96 x 90 3790 / 578; A2 x 3 at 128^3 5000 / 1350; A1 at 20^3 490 /
// 244 through solve_cg.  A 128^3 x 3 step takes 18.6 us (18.7 bytes per unknown
// with the overlaps: 6.3 TB/s out of the L2, 2 us of it the barrier).
//
// The even stencil has 8 distinct coefficients c[|dx|][|dy|][|dz|].  A thread holds
// a quad of a z-line and marches along x: per plane u = v(y-1) + v(y+1) and the
// sums over z +- 1 of v and u (shuffles; loads at the ends of a line and of the
// warp) give the plane's contribution to its own output and to its two x
// neighbours': 8 FMAs and 5 adds per unknown, three vector loads per quad.
//
// Vectors hold z-lines of `pitch` floats, element (i, s, j, k) of right-hand side s at
// ((i NR + s) ny + j) pitch + k, with copies of the line's first value at k = nz and of its last at k = -1, so a
// quad of a line is one aligned vector load for every nz and z neighbours need
// no wrapping.  r = -0.0f marks a pinned DOF (identity row, excluded column; its
// solution is x = b): the iterates stay zero there.  x is held as the
// unevaluated sum h + l of two float vectors until the end.  A right-hand side
// whose norm leaves the middle of the float range is solved as 2^-e b.
//
// The chunks of the passes that sum (runs of a plane times a range of planes) depend on the system alone, and its
// CTAs pass a grid barrier of their own: a system's iterates are the same bits on any number of CTAs.
#pragma once

#include "stencil_ops.cuh"

namespace cpm {

constexpr int kChebThreads = 256;
constexpr int kChebBlocks = 3;   // CTAs per SM (80 registers: the pass without spills)
constexpr int kChebPad = 8;      // floats before and after each vector
constexpr int kChebMaxSteps = 96;
constexpr int kChebSlot = 4;     // doubles per chunk partial

// The operator's part: coefficients and recurrence factors (launch parameters).
struct ChebOp {
  float c[8];                    // c[4 |dx| + 2 |dy| + |dz|]
  float cl[8];                   // the coefficients' rest: c + cl as a double-float value
  double c64[8];
  float w[kChebMaxSteps], g[kChebMaxSteps];  // factors of the step from x_k to x_{k+1}, k >= 1
  double itheta, acosh_s;        // 1 / centre of the interval; acosh of (centre / half width)
  double df_err;                 // error bound of a double-float residual as a multiple of ||b||
  double q32;                    // error bound of an FP32 residual r - A d as a multiple of |r| + |r - A d|
  int df;                        // double-float residuals (else FP64)
  unsigned long long timeout_ns;
};

// One system.
struct ChebSys {
  int nx, ny, nz, n;
  const uint8_t *flags;
  const double *b;
  double *x;
  const int *use_init_dev;
  int use_init_host;
  int maxiter;
  double tol;
  cpm_cg_info *info;
  float *v[5];                   // r and four iterate vectors
  double *part;                  // two halves of `half` doubles: kChebSlot per chunk of any pass
  int half;
  GridBarrier *bar;
  int pitch, nq;                      // floats and quads of a z-line
  int runs, tw, lx, ranges, chunks;   // step passes: runs of 32 quads per plane, runs per tile, planes per range
  int clx, cranges, cchunks;          // the check's passes, on the same tiles
  int rtiles, rlx, rranges, rchunks;  // residual passes: tiles of kChebThreads DOFs of a plane
  int lchunk, lchunks;                // pointwise passes: z-lines per chunk
  int cta0, ncta;
};

// Chunks of a pass at most, as the partials of cpm_cg_solve_stencil's workspace hold them.  Planes of more tiles
// than that (2.36 M nodes) have no such cut: their solves keep CG.
constexpr int64_t kChebMaxChunks = (int64_t)(kPartHalf / kChebSlot);

// Partition of a system's passes: enough chunks to fill the GPU when the system runs alone, as few
// planes of overlap as that allows.  `slots` CTAs are resident.
inline void cheb_split(int nx, int tiles, int sms, int slots, int &lx, int &ranges) {
  double best = 1e300;
  lx = nx;
  ranges = 1;
  for (int nr = 1; nr <= nx; ++nr) {
    const int l = (nx + nr - 1) / nr, r = (nx + l - 1) / l;
    const int64_t ch = (int64_t)tiles * r;
    if (nr > 1 && ch > kChebMaxChunks) break;
    const int64_t ctas = ch < slots ? ch : slots, loops = (ch + ctas - 1) / ctas;
    const int64_t per_sm = (ctas + sms - 1) / sms;
    // a tile-plane costs its SM about 400 cycles of L2 traffic and a plane about 500 of latency
    const double cost = (double)loops * (400.0 * per_sm + 500.0) * (l + 2);
    if (cost < best) {
      best = cost;
      lx = l;
      ranges = r;
    }
  }
}

// Floats of one vector.
inline size_t cheb_vec_floats(int nx, int ny, int nz, int nrhs) {
  return 2 * kChebPad + (size_t)nx * nrhs * ny * ((nz + 2 + 7) / 8 * 8);
}

inline void cheb_layout(ChebSys &S, int nrhs, int sms) {
  // Two CTAs per SM up to 2.5 M unknowns (the barrier costs more with more CTAs), three above.  Measured on GB300,
  // us per cold A1 solve on 2 / 3: 64^3 x 3 312 / 335, 128^3 451 / 467, 112 x 96 x 90 x 3 627 / 562,
  // 128^3 x 3 1084 / 980.
  const int slots = sms * ((int64_t)S.n * nrhs > 2500000 ? kChebBlocks : 2);
  S.nq = (S.nz + 3) / 4;
  S.pitch = (S.nz + 2 + 7) / 8 * 8;
  S.runs = (int)(((int64_t)nrhs * S.ny * S.nq + 31) / 32);
  constexpr int per = kChebThreads / 32;
  int tiles = (S.runs + per - 1) / per;
  S.tw = (S.runs + tiles - 1) / tiles;
  tiles = (S.runs + S.tw - 1) / S.tw;
  cheb_split(S.nx, tiles, sms, slots, S.lx, S.ranges);
  S.chunks = tiles * S.ranges;
  S.clx = S.lx;
  S.cranges = S.ranges;
  S.cchunks = S.chunks;
  S.rtiles = (int)(((int64_t)S.ny * S.nz + kChebThreads - 1) / kChebThreads);
  cheb_split(S.nx, S.rtiles, sms, slots, S.rlx, S.rranges);
  S.rchunks = S.rtiles * S.rranges;
  const int lines = S.nx * S.ny, lc = (lines + slots - 1) / slots;
  S.lchunk = lc < per ? per : lc;
  S.lchunks = (lines + S.lchunk - 1) / S.lchunk;
  const int most = S.rchunks > S.lchunks ? S.rchunks : S.lchunks;
  S.half = kChebSlot * (S.cchunks > most ? S.cchunks : most);
}

// Whether the iteration applies to a stencil at all, and its factors: scalar, even along every axis to
// rounding, symbol positive with a condition number of at most 64 (CG's iterations grow more slowly on
// wider spectra).
bool cheb_operator(const double *coef, int ncomp, ChebOp *op);
// Error bound of a double-float residual as a multiple of ||b|| (-1: none).
double df_error_bound(const cpm_stencil *s);
// Steps that the iteration takes from a cold start to tol (host estimate of the device's schedule).
int cheb_cold_steps(const ChebOp &op, double tol);

// Reduction of one cycle at most: FP32 iterates hold about 6 digits.
constexpr double kChebCycle = 1e6;
// The last cycle aims this factor below the threshold.
constexpr double kChebAim = 0.5;

// Steps of the cycle that starts at residual `res` and has to end below `goal`.
__host__ __device__ inline int cheb_steps(double res, double goal, double acosh_s) {
  const double ratio = res / goal, lr = ratio > 1.0 ? log(ratio < kChebCycle ? ratio : kChebCycle) : 0.0;
  // T_k(s) >= e^(k acosh s) / 2
  int k = (int)ceil((lr + 0.6931471805599453) / acosh_s);
  return k < 2 ? 2 : k > kChebMaxSteps ? kChebMaxSteps : k;
}

// ---------------------------------------------------------------- conversions without the FP64 pipe
// GB300 converts between float and double at its FP64 rate; these take integer instructions for values
// in the float range and the conversion instruction otherwise.
__device__ __forceinline__ double f2d(float f) {
  const uint32_t b = __float_as_uint(f);
  const uint32_t e = b & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return (double)f;
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// v = hi + lo to 2^-47 of v: hi the 24 leading bits of v (truncated), lo the rest rounded.
__device__ __forceinline__ void d2ff(double v, float &hi, float &lo) {
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  const uint32_t e = (h >> 20) & 0x7ffu;
  if (e < 1023u - 60u || e > 1023u + 120u) {
    hi = __double2float_rn(v);
    lo = isfinite(v) && fabsf(hi) <= 3.0e38f ? __double2float_rn(v - (double)hi) : 0.0f;
    return;
  }
  const uint32_t s = h & 0x80000000u;
  hi = __uint_as_float(s | ((e - 896u) << 23) | ((h & 0xfffffu) << 3) | (l >> 29));
  // the low 29 bits, in units of 2^(e - 1023 - 52)
  const float m = __uint2float_rn(l & 0x1fffffffu) * __uint_as_float((e - 896u - 52u) << 23);
  lo = __uint_as_float(__float_as_uint(m) | s);
}

// ---------------------------------------------------------------- double-float sums
__device__ __forceinline__ df::DF df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return df::DF(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t)));
}
// a + b, not renormalised: the high parts exactly, the low parts in FP32.
__device__ __forceinline__ df::DF df_add(const df::DF &a, const df::DF &b) {
  df::DF s = df_two_sum(a.hi, b.hi);
  s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  return s;
}

// ---------------------------------------------------------------- sums of a system
// Totals over the system's chunk partials, in chunk order, after a barrier.
template <int NV>
__device__ __forceinline__ bool cheb_totals(const ChebSys &S, unsigned long long tns, int chunks, int &par,
                                            double (&v)[NV], double (*sred)[kCGWarps]) {
  const double *half = S.part + (size_t)par * S.half;
  par ^= 1;
  if (!grid_sync(S.bar, S.ncta, tns)) return false;
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = 0.0;
  for (int c = threadIdx.x; c < chunks; c += kChebThreads)
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] += __ldcg(half + (size_t)c * kChebSlot + j);
  block_sum<NV, kCGWarps, kChebThreads>(v, sred);
  return true;
}

// ---------------------------------------------------------------- one step
// Pairs of floats: one packed instruction does both, which halves the issue slots of the pass's arithmetic.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
struct Quad {
  f32x2 a, b;
};
__device__ __forceinline__ Quad load_quad(const float *p) {
  const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p);
  return Quad{t.x, t.y};
}

// A thread's quad of a z-line, k = 4 k4 .. 4 k4 + 3 of line `row` of a plane.
struct ChebQuad {
  int off, om, od;    // the quad in its plane; offsets of the lines y - 1 and y + 1
  int valid, k4;      // unknowns inside the grid (0: the thread only takes part)
  bool nl, nr;        // the left / right neighbour is in no lane
  bool first, last;   // the line's ends
};

// The plane's contributions to its own output (cc) and to its two x neighbours' (ss).
__device__ __forceinline__ void cheb_plane(const ChebQuad &c, const f32x2 (&co)[8], const float *xp, const Quad &v,
                                           const Quad &m, const Quad &d, Quad &cc, Quad &ss) {
  const Quad u{add2(m.a, d.a), add2(m.b, d.b)};
  float v0, v1, v2, v3, u0, u1, u2, u3;
  unpack2(v.a, v0, v1);
  unpack2(v.b, v2, v3);
  unpack2(u.a, u0, u1);
  unpack2(u.b, u2, u3);
  float vl = __shfl_up_sync(0xffffffffu, v3, 1), ul = __shfl_up_sync(0xffffffffu, u3, 1);
  float vr = __shfl_down_sync(0xffffffffu, v0, 1), ur = __shfl_down_sync(0xffffffffu, u0, 1);
  if (c.nl) {
    vl = xp[-1];
    ul = xp[c.om - 1] + xp[c.od - 1];
  }
  if (c.nr) {
    vr = xp[4];
    ur = xp[c.om + 4] + xp[c.od + 4];
  }
  const Quad t{pack2(vl + v1, v0 + v2), pack2(v1 + v3, v2 + vr)};
  const Quad w{pack2(ul + u1, u0 + u2), pack2(u1 + u3, u2 + ur)};
  cc.a = fma2(co[3], w.a, fma2(co[2], u.a, fma2(co[1], t.a, mul2(co[0], v.a))));
  cc.b = fma2(co[3], w.b, fma2(co[2], u.b, fma2(co[1], t.b, mul2(co[0], v.b))));
  ss.a = fma2(co[7], w.a, fma2(co[6], u.a, fma2(co[5], t.a, mul2(co[4], v.a))));
  ss.b = fma2(co[7], w.b, fma2(co[6], u.b, fma2(co[5], t.b, mul2(co[4], v.b))));
}

// out = ca x + cb out + cg r - ch A x on the free DOFs, 0 on the pinned ones (out is not read where cb = 0), with ca
// and ch inside the coefficients.  CHECK: nothing is written; the chunk partials of |out|^2 times scale^2 per
// right-hand side go to `half` (cb = 0): the squares of a quad are added in FP32 (5 roundings), the quads in FP64.
template <int NR, bool CHECK>
__device__ __forceinline__ void cheb_pass(const ChebSys &S, const ChebOp &op, int l, const float *x, float *out,
                                          const float *r, float ca, float cb, float cg, float ch,
                                          const float (&scale)[NR], double *half, double (*sred)[kCGWarps]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = NR * S.ny, P = S.pitch, nq = S.nq, nx = S.nx;
  const int64_t plane = (int64_t)rows * P;
  f32x2 co[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float t = e == 0 ? fmaf(-ch, op.c[0], ca) : -ch * op.c[e];
    co[e] = pack2(t, t);
  }
  const f32x2 cb2 = pack2(cb, cb), cg2 = pack2(cg, cg);
  const int lx = CHECK ? S.clx : S.lx, ranges = CHECK ? S.cranges : S.ranges, chunks = CHECK ? S.cchunks : S.chunks;
  for (int chunk = l; chunk < chunks; chunk += S.ncta) {
    const int tile = chunk / ranges, x0 = (chunk - tile * ranges) * lx, x1 = min(nx, x0 + lx);
    const int run = tile * S.tw + warp;
    double sum = 0.0;
    int rhs = 0;
    if (warp < S.tw && run < S.runs) {
      ChebQuad c;
      {
        const int f = run * 32 + lane, fe = min(f, rows * nq - 1);
        const int row = fe / nq, j = row % S.ny;
        rhs = row / S.ny;
        c.k4 = fe - row * nq;
        c.off = row * P + 4 * c.k4;
        c.om = j == 0 ? (S.ny - 1) * P : -P;
        c.od = j == S.ny - 1 ? -(S.ny - 1) * P : P;
        c.nl = lane == 0 || c.k4 == 0;
        c.nr = lane == 31 || c.k4 == nq - 1;
        c.valid = f < rows * nq ? min(4, S.nz - 4 * c.k4) : 0;
        c.first = c.valid > 0 && c.k4 == 0;
        c.last = c.valid > 0 && c.k4 == nq - 1;
      }
      const float *xb = x + c.off;
      const float *xp = xb + (x0 == 0 ? nx - 1 : x0 - 1) * plane;
      Quad v = load_quad(xp), m = load_quad(xp + c.om), d = load_quad(xp + c.od), cc, ss, acc, sp;
      const float *xn = xb + x0 * plane;
      Quad nv = load_quad(xn), nm = load_quad(xn + c.om), nd = load_quad(xn + c.od);
      cheb_plane(c, co, xp, v, m, d, cc, sp);
      xp = xn;
      xn = x0 + 1 == nx ? xb : xn + plane;
      v = nv; m = nm; d = nd;
      nv = load_quad(xn);
      nm = load_quad(xn + c.om);
      nd = load_quad(xn + c.od);
      cheb_plane(c, co, xp, v, m, d, acc, ss);
      acc.a = add2(acc.a, sp.a);
      acc.b = add2(acc.b, sp.b);
      sp = ss;
      float *o = out + x0 * plane + c.off;
      const float *rp = r + x0 * plane + c.off;
  #pragma unroll 1
      for (int i = x0 + 1; i <= x1; ++i) {
        const Quad ro = load_quad(rp);
        Quad xo{0ull, 0ull};
        if (cb != 0.0f) xo = load_quad(o);
        xp = xn;
        v = nv; m = nm; d = nd;
        if (i < x1) {
          xn = i + 1 == nx ? xb : xn + plane;
          nv = load_quad(xn);
          nm = load_quad(xn + c.om);
          nd = load_quad(xn + c.od);
        }
        cheb_plane(c, co, xp, v, m, d, cc, ss);
        const f32x2 ra = fma2(cb2, xo.a, fma2(cg2, ro.a, add2(acc.a, ss.a)));
        const f32x2 rb = fma2(cb2, xo.b, fma2(cg2, ro.b, add2(acc.b, ss.b)));
        acc.a = add2(cc.a, sp.a);
        acc.b = add2(cc.b, sp.b);
        sp = ss;
        float q0, q1, q2, q3, r0, r1, r2, r3;
        unpack2(ra, q0, q1);
        unpack2(rb, q2, q3);
        unpack2(ro.a, r0, r1);
        unpack2(ro.b, r2, r3);
        if (__float_as_uint(r0) == 0x80000000u) q0 = 0.0f;
        if (__float_as_uint(r1) == 0x80000000u) q1 = 0.0f;
        if (__float_as_uint(r2) == 0x80000000u) q2 = 0.0f;
        if (__float_as_uint(r3) == 0x80000000u) q3 = 0.0f;
        if (CHECK) {
          if (c.valid < 4) q3 = 0.0f;
          if (c.valid < 3) q2 = 0.0f;
          if (c.valid < 2) q1 = 0.0f;
          if (c.valid < 1) q0 = 0.0f;
          float f = scale[0];
  #pragma unroll
          for (int s = 1; s < NR; ++s)
            if (rhs == s) f = scale[s];
          q0 *= f;
          q1 *= f;
          q2 *= f;
          q3 *= f;
          sum += f2d(fmaf(q0, q0, fmaf(q1, q1, fmaf(q2, q2, q3 * q3))));
          rp += plane;
          continue;
        }
        if (c.valid == 4) *reinterpret_cast<float4 *>(o) = make_float4(q0, q1, q2, q3);
        if (c.valid < 4 || c.first || c.last) {
          if (c.valid < 4) {
            if (c.valid > 0) o[0] = q0;
            if (c.valid > 1) o[1] = q1;
            if (c.valid > 2) o[2] = q2;
          }
          // the copies beyond the ends of the z-line
          if (c.first) o[S.nz] = q0;
          if (c.last) o[-4 * c.k4 - 1] = c.valid == 4 ? q3 : c.valid == 3 ? q2 : c.valid == 2 ? q1 : q0;
        }
        o += plane;
        rp += plane;
      }
    }
    if (CHECK) {
      double v[NR];
#pragma unroll
      for (int s = 0; s < NR; ++s) v[s] = rhs == s ? sum : 0.0;
      block_sum<NR, kCGWarps, kChebThreads>(v, sred);
#pragma unroll
      for (int s = 0; s < NR; ++s)
        if (threadIdx.x == s) half[(size_t)chunk * kChebSlot + s] = v[s];
    }
  }
}

// The value of column k of a z-line at p, with its copy beyond the line's other end.
__device__ __forceinline__ void cheb_put(float *p, int k, int nz, float v) {
  *p = v;
  if (k == 0) p[nz] = v;
  if (k == nz - 1) p[-nz] = v;
}

// ---------------------------------------------------------------- residual
// r = b - A (h + l) on the free DOFs in double-float arithmetic (l may be NULL), -0.0f on the pinned ones, and
// the chunk partials of |r|^2 per right-hand side, of the unrounded r in FP64 (the stopping test is on this norm);
// b times `down` where that is set.  Every value enters renormalised (h + l = hi + lo exactly, |lo| <= 2^-24 |hi|).  In units of 2^-48 of the sum of the terms'
// magnitudes: the z and y sums of a term are within 8 (df_add: 3 per sum, twice, and 2 for the dropped
// renormalisation), its product within 13 (df::fma), the 4 + 4 accumulations and two sums of planes within 3 each; the
// difference from b adds 3 and b's split 2, as |b| is at most that sum and |r|: 56, inside the 94 that the bound of
// df_error_bound allows.
template <int NR>
__device__ __forceinline__ void cheb_residual(const ChebSys &S, const ChebOp &op, int l, const double *down,
                                              const float *h, const float *lo, float *r, double *half,
                                              double (*sred)[kCGWarps]) {
  const int nyz = S.ny * S.nz, nz = S.nz, P = S.pitch, q = NR * S.ny * P;
  for (int chunk = l; chunk < S.rchunks; chunk += S.ncta) {
    const int tile = chunk / S.rranges, x0 = (chunk - tile * S.rranges) * S.rlx, x1 = min(S.nx, x0 + S.rlx);
    const int f = tile * kChebThreads + threadIdx.x;
    double nrm[NR];
#pragma unroll
    for (int s = 0; s < NR; ++s) nrm[s] = 0.0;
    if (f < nyz) {
      const int j = f / nz, k = f - j * nz;
      const int om = j == 0 ? (S.ny - 1) * P : -P, od = j == S.ny - 1 ? -(S.ny - 1) * P : P;
#pragma unroll
      for (int s = 0; s < NR; ++s) {  // one right-hand side at a time: 96 registers with all three
        df::DF acc, sp;
        const int at = (s * S.ny + j) * P + k;
        const float *hs = h + at, *ls = lo ? lo + at : nullptr;
        double sum = 0.0;
#pragma unroll 1
        for (int i = x0 - 1; i <= x1; ++i) {
          const int64_t p = (int64_t)(i < 0 ? S.nx - 1 : i >= S.nx ? 0 : i) * q;
          const float *hp = hs + p, *lp = ls + p;
          asm volatile("" : "+l"(hp), "+l"(lp));
          auto val = [&](int e) { return lo ? df_two_sum(hp[e], lp[e]) : df::DF(hp[e], 0.0f); };
          const df::DF v = val(0);
          const df::DF u = df_add(val(om), val(od));
          const df::DF t = df_add(val(-1), val(1));
          const df::DF w = df_add(df_add(val(om - 1), val(od - 1)), df_add(val(om + 1), val(od + 1)));
          const df::DF zero;
          auto cf = [&](int e) { return df::DF(op.c[e], op.cl[e]); };
          const df::DF cc = df::fma(cf(3), w, df::fma(cf(2), u, df::fma(cf(1), t, df::fma(cf(0), v, zero))));
          const df::DF ss = df::fma(cf(7), w, df::fma(cf(6), u, df::fma(cf(5), t, df::fma(cf(4), v, zero))));
          if (i > x0) {
            const int64_t dof = (int64_t)(i - 1) * nyz + f;
            const bool pin = S.flags && (S.flags[dof] & (kRowIdentity | kColExcluded)) != 0;
            const df::DF y = df_add(acc, ss);
            float bh, bl;
            d2ff(down ? S.b[dof * NR + s] * down[s] : S.b[dof * NR + s], bh, bl);
            const df::DF d = df_add(df::DF(bh, bl), df::DF(-y.hi, -y.lo));
            cheb_put(r + (int64_t)(i - 1) * q + at, k, nz, pin ? -0.0f : (d.hi + d.lo) + 0.0f);
            const double t = pin ? 0.0 : f2d(d.hi) + f2d(d.lo);
            sum = ::fma(t, t, sum);
          }
          acc = df_add(cc, sp);
          const float hi = __fadd_rn(acc.hi, acc.lo);
          acc.lo = __fsub_rn(acc.lo, __fsub_rn(hi, acc.hi));
          acc.hi = hi;
          sp = ss;
        }
        nrm[s] = sum;
      }
    }
    double v[NR];
#pragma unroll
    for (int s = 0; s < NR; ++s) v[s] = nrm[s];
    block_sum<NR, kCGWarps, kChebThreads>(v, sred);
#pragma unroll
    for (int s = 0; s < NR; ++s)
      if (threadIdx.x == s) half[(size_t)chunk * kChebSlot + s] = v[s];
  }
}

// The same in FP64 arithmetic.
template <int NR>
__device__ __noinline__ void cheb_residual64(const ChebSys &S, const ChebOp &op, int l, const double *down,
                                             const float *h, const float *lo, float *r, double *half,
                                             double (*sred)[kCGWarps]) {
  const int nyz = S.ny * S.nz, nz = S.nz, P = S.pitch, q = NR * S.ny * P;
  for (int chunk = l; chunk < S.rchunks; chunk += S.ncta) {
    const int tile = chunk / S.rranges, x0 = (chunk - tile * S.rranges) * S.rlx, x1 = min(S.nx, x0 + S.rlx);
    const int f = tile * kChebThreads + threadIdx.x;
    double nrm[NR];
#pragma unroll
    for (int s = 0; s < NR; ++s) nrm[s] = 0.0;
    if (f < nyz) {
      const int j = f / nz, k = f - j * nz;
      const int yo[3] = {j == 0 ? (S.ny - 1) * P : -P, 0, j == S.ny - 1 ? -(S.ny - 1) * P : P};
      for (int i = x0; i < x1; ++i) {
        const int xi[3] = {i == 0 ? S.nx - 1 : i - 1, i, i == S.nx - 1 ? 0 : i + 1};
        const int64_t dof = (int64_t)i * nyz + f;
        const bool pin = S.flags && (S.flags[dof] & (kRowIdentity | kColExcluded)) != 0;
#pragma unroll 1
        for (int s = 0; s < NR; ++s) {
          double y = 0.0;
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
#pragma unroll
              for (int c = 0; c < 3; ++c) {
                const int64_t p = (int64_t)xi[a] * q + (s * S.ny + j) * P + k + yo[b] + c - 1;
                const double xv = lo ? (double)h[p] + (double)lo[p] : (double)h[p];
                y = ::fma(op.c64[(a != 1) * 4 + (b != 1) * 2 + (c != 1)], xv, y);
              }
          const double t = pin ? 0.0 : (down ? S.b[dof * NR + s] * down[s] : S.b[dof * NR + s]) - y;
          cheb_put(r + (int64_t)i * q + (s * S.ny + j) * P + k, k, nz, pin ? -0.0f : (float)t + 0.0f);
#pragma unroll
          for (int e = 0; e < NR; ++e)
            if (e == s) nrm[e] = ::fma(t, t, nrm[e]);
        }
      }
    }
    double v[NR];
#pragma unroll
    for (int s = 0; s < NR; ++s) v[s] = nrm[s];
    block_sum<NR, kCGWarps, kChebThreads>(v, sred);
#pragma unroll
    for (int s = 0; s < NR; ++s)
      if (threadIdx.x == s) half[(size_t)chunk * kChebSlot + s] = v[s];
  }
}

// ---------------------------------------------------------------- the solve of one system
template <int NR>
struct ChebState {
  double bn[NR], res[NR], last[NR];  // ||b||, ||b - A x|| per right-hand side (of 2^-e b)
  double down[NR], up[NR];           // 2^-e, 2^e
  float scale[NR];
  int scaled, exp2[NR], active, pending, steps, fit, finite, check, proven;
};

// Steps of the next cycle, enough for every pending right-hand side, and whether its end may be proven by an
// FP32 residual (not where the caller asked for FP64 residuals).
template <int NR>
__device__ __forceinline__ int cheb_cycle(ChebState<NR> &st, const ChebSys &S, const ChebOp &op, int iters) {
  int steps = 2;
  st.check = op.df;
  for (int s = 0; s < NR; ++s) {
    if (!((st.pending >> s) & 1)) continue;
    const double goal = kChebAim * S.tol * st.bn[s];
    steps = max(steps, cheb_steps(st.res[s], goal, op.acosh_s));
    const double most = goal + op.q32 * (st.res[s] + goal) + op.df_err * st.bn[s];
    if (!(st.res[s] <= kChebCycle * goal && most <= 0.9 * S.tol * st.bn[s])) st.check = 0;
  }
  return min(steps, max(2, S.maxiter - iters));
}

// r = b (cold) or h + lo = x (warm), times `down` where that is set; with `sums` the chunk partials of |b|^2 and of
// the flagged rows that are not pinned (half 0).
template <int NR>
__device__ __noinline__ void cheb_start(const ChebSys &S, int l, bool use_init, const double *down, bool sums,
                                        double (*sred)[kCGWarps]) {
  const int q = NR * S.ny * S.pitch, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int chunk = l; chunk < S.lchunks; chunk += S.ncta) {
    double acc[NR + 1];
#pragma unroll
    for (int j = 0; j <= NR; ++j) acc[j] = 0.0;
    const int g1 = min(S.nx * S.ny, (chunk + 1) * S.lchunk);
    for (int g = chunk * S.lchunk + warp; g < g1; g += kChebThreads / 32) {
      const int i = g / S.ny, j = g - i * S.ny;
      for (int k = lane; k < S.nz; k += 32) {
        const int64_t dof = (int64_t)g * S.nz + k;
        int fr = 0;
        if (S.flags) fr = S.flags[dof] & (kRowIdentity | kRowZero | kColExcluded);
        if (fr && fr != (kRowIdentity | kColExcluded)) acc[NR] += 1.0;
#pragma unroll
        for (int s = 0; s < NR; ++s) {
          const int64_t e = (int64_t)i * q + (s * S.ny + j) * S.pitch + k;
          if (sums) acc[s] = fma(S.b[dof * NR + s], S.b[dof * NR + s], acc[s]);
          double t = use_init ? S.x[dof * NR + s] : S.b[dof * NR + s];
          if (down) t *= down[s];
          float hi, lw;
          d2ff(t, hi, lw);
          if (use_init) {
            cheb_put(S.v[3] + e, k, S.nz, fr ? 0.0f : hi);
            cheb_put(S.v[4] + e, k, S.nz, fr ? 0.0f : lw);
          } else {
            cheb_put(S.v[0] + e, k, S.nz, fr ? -0.0f : hi + 0.0f);
          }
        }
      }
    }
    if (!sums) continue;
    block_sum<NR + 1, kCGWarps, kChebThreads>(acc, sred);
#pragma unroll
    for (int j = 0; j <= NR; ++j)
      if (threadIdx.x == j) S.part[(size_t)chunk * kChebSlot + j] = acc[j];
  }
}

// Returns false (in every thread of the system's CTAs, before x is written) when the system is not one
// for this iteration: a flagged row that is not pinned, or a right-hand side or warm start that is not
// finite in floats.  Other CTAs may then still read S.part: its next user needs a barrier (or a launch) in front.
template <int NR>
__device__ __forceinline__ bool cheb_solve(const ChebSys &S, const ChebOp &op, int l, double (*sred)[kCGWarps]) {
  __shared__ ChebState<NR> st;  // thread 0 writes it after each reduction (FP64 scalars are slow in every thread)
  const unsigned long long tns = op.timeout_ns;
  const bool use_init = S.use_init_dev ? (__ldcg(S.use_init_dev) != 0) : (S.use_init_host != 0);
  const int q = NR * S.ny * S.pitch, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int par = 0;
  float *r = S.v[0];
  // ---- r = b (cold) or the split of x (warm); ||b||, flagged rows that are not pinned
  cheb_start<NR>(S, l, use_init, nullptr, true, sred);
  double v[NR + 1];
  if (!cheb_totals<NR + 1>(S, tns, S.lchunks, par, v, sred)) {
    set_status(S.info, CPM_BARRIER_TIMEOUT);
    return true;
  }
  if (threadIdx.x == 0) {
    st.fit = v[NR] == 0.0;
    st.active = st.scaled = 0;
    for (int s = 0; s < NR; ++s) {
      double bb = v[s];
      st.scale[s] = 1.0f;
      st.exp2[s] = 0;
      st.down[s] = st.up[s] = 1.0;
      if (bb != 0.0) {
        st.active |= 1 << s;
        if (!isfinite(bb)) st.fit = 0;
        else if (bb < 1e-30 || bb > 1e30) {
          const int e = ilogb(bb) / 2;
          st.down[s] = ldexp(1.0, -e);
          st.up[s] = ldexp(1.0, e);
          st.scaled = 1;
          bb = ldexp(bb, -2 * e);
        }
        if (st.fit) st.exp2[s] = ilogb(bb) / 2;  // the check squares in FP32 over r / 2^exp2, 2^exp2 near ||b||
        st.scale[s] = (float)ldexp(1.0, -st.exp2[s]);
      }
      st.bn[s] = st.res[s] = sqrt(bb);
    }
    st.pending = st.active;
    st.steps = st.fit ? cheb_cycle(st, S, op, 0) : 0;
  }
  __syncthreads();
  if (!st.fit) return false;
  const double *down = nullptr;
  if (st.scaled) {
    down = st.down;
    cheb_start<NR>(S, l, use_init, down, false, sred);
    if (!grid_sync(S.bar, S.ncta, tns)) {
      set_status(S.info, CPM_BARRIER_TIMEOUT);
      return true;
    }
  }
  const int active = st.active;
  float scale[NR];
#pragma unroll
  for (int s = 0; s < NR; ++s) scale[s] = st.scale[s];
  float *h = use_init ? S.v[3] : nullptr, *lo = use_init ? S.v[4] : nullptr;
  float *fr0 = S.v[1], *fr1 = S.v[2];
  int iters = 0, updates = 0, status = CPM_OK;
  int unconv = 0;
  bool first = true;
  if (active) {
    for (;;) {
      if (!first || use_init) {
        // ---- the residual of x = h + lo
        double *half = S.part + (size_t)par * S.half;
        if (op.df) cheb_residual<NR>(S, op, l, down, h, lo, r, half, sred);
        else cheb_residual64<NR>(S, op, l, down, h, lo, r, half, sred);
        double t[NR];
        if (!cheb_totals<NR>(S, tns, S.rchunks, par, t, sred)) { status = CPM_BARRIER_TIMEOUT; break; }
        if (!first) ++updates;
        if (threadIdx.x == 0) {
          st.finite = 1;
          for (int s = 0; s < NR; ++s) {
            st.res[s] = sqrt(t[s]);
            if (!((st.pending >> s) & 1)) continue;
            if (!isfinite(st.res[s])) st.finite = 0;
            // a double-float residual decides outside its error bound only; a warm start takes at least
            // one cycle, as CG takes one iteration
            const double at = S.tol * st.bn[s] - (op.df ? op.df_err * st.bn[s] : 0.0);
            if (!first && st.res[s] <= at) st.pending &= ~(1 << s);
          }
          st.steps = st.finite ? cheb_cycle(st, S, op, iters) : 0;
        }
        __syncthreads();
        if (!st.finite) {
          if (first) return false;
          status = CPM_NONFINITE;
          break;
        }
        if (!st.pending) break;
        if (iters >= S.maxiter) {
          unconv = 1;
          break;
        }
      }
      // ---- a cycle of steps on A d = r
      const int steps = st.steps;
      // the pass for x_2 reads r, as x_1 = r / theta; the one for x_3 takes its x_1 from r too
      float *d0 = fr1, *d1 = fr0;
      bool ok = true;
#pragma unroll 1
      for (int k = 1; ok && k < steps; ++k) {
        const float w = op.w[k - 1], g = op.g[k - 1], it = (float)op.itheta;
        const float ca = k == 1 ? (1.0f + w) * it + g : 1.0f + w, cb = k <= 2 ? 0.0f : -w;
        const float cg = k == 1 ? 0.0f : k == 2 ? g - w * it : g, ch = k == 1 ? g * it : g;
        cheb_pass<NR, false>(S, op, l, k == 1 ? r : d0, d1, r, ca, cb, cg, ch, scale, nullptr, sred);
        float *t = d0;
        d0 = d1;
        d1 = t;
        ok = grid_sync(S.bar, S.ncta, tns);
      }
      if (!ok) { status = CPM_BARRIER_TIMEOUT; break; }
      iters += steps;
      // ---- a last cycle: |r - A d| in FP32 proves the stopping test where its error bound leaves room.  Its
      // longest path has 10 roundings (the coefficient's, 2 sums over y and z, 4 FMAs, 2 planes, r), so the
      // error is at most 11 2^-24 sum|c| |d| + 3 2^-24 |r|, and |d| <= (|r| + |r - A d|) / sigma_min.
      bool proven = false;
      if (st.check) {
        double *half = S.part + (size_t)par * S.half;
        cheb_pass<NR, true>(S, op, l, d0, d1, r, 0.0f, 0.0f, 1.0f, 1.0f, scale, half, sred);
        double t[NR];
        if (!cheb_totals<NR>(S, tns, S.cchunks, par, t, sred)) { status = CPM_BARRIER_TIMEOUT; break; }
        if (threadIdx.x == 0) {
          int left = 0;
          for (int s = 0; s < NR; ++s) {
            if (!((st.pending >> s) & 1)) continue;
            const double res = 1.0001 * ldexp(sqrt(t[s]), st.exp2[s]);
            const double most = res + op.q32 * (st.res[s] + res) + op.df_err * st.bn[s];
            if (!(most <= S.tol * st.bn[s])) left = 1;
            else if (!left) st.last[s] = res;
          }
          st.proven = !left;
          if (!left)
            for (int s = 0; s < NR; ++s)
              if ((st.pending >> s) & 1) st.res[s] = st.last[s];
        }
        __syncthreads();
        proven = st.proven != 0;
      }
      // ---- x += d (d0): the first two corrections of a cold start are h and lo themselves
      if (!h) {
        h = d0;
        fr0 = d1;
        fr1 = S.v[3];
      } else if (!lo) {
        lo = d0;
        fr0 = d1;
        fr1 = S.v[4];
      } else {
        // the whole storage, copies included
        const int64_t all = (int64_t)S.nx * q + 1;
        for (int64_t e = (int64_t)l * kChebThreads + threadIdx.x; e < all; e += (int64_t)S.ncta * kChebThreads) {
          const df::DF c = df_add(df_two_sum(h[e - 1], lo[e - 1]), df::DF(d0[e - 1], 0.0f));
          const float hi = __fadd_rn(c.hi, c.lo);
          h[e - 1] = hi;
          lo[e - 1] = __fsub_rn(c.lo, __fsub_rn(hi, c.hi));
        }
        if (!grid_sync(S.bar, S.ncta, tns)) { status = CPM_BARRIER_TIMEOUT; break; }
      }
      first = false;
      if (proven) break;
    }
  }
  // ---- x = h + lo, b on the pinned DOFs and where b = 0
  if (status == CPM_OK || status == CPM_NONFINITE)
    for (int chunk = l; chunk < S.lchunks; chunk += S.ncta) {
      const int g1 = min(S.nx * S.ny, (chunk + 1) * S.lchunk);
      for (int g = chunk * S.lchunk + warp; g < g1; g += kChebThreads / 32) {
        const int i = g / S.ny, j = g - i * S.ny;
        for (int k = lane; k < S.nz; k += 32) {
          const int64_t dof = (int64_t)g * S.nz + k;
          const bool pin = S.flags && (S.flags[dof] & (kRowIdentity | kColExcluded)) != 0;
#pragma unroll
          for (int s = 0; s < NR; ++s) {
            const int64_t e = (int64_t)i * q + (s * S.ny + j) * S.pitch + k, o = dof * NR + s;
            double xv;
            if (pin || !((active >> s) & 1)) xv = S.b[o];
            else if (!h) xv = 0.0;
            else xv = lo ? f2d(h[e]) + f2d(lo[e]) : f2d(h[e]);
            if (down && !pin) xv *= st.up[s];
            S.x[o] = xv;
          }
        }
      }
    }
  if (threadIdx.x == 0) {
    if (l == 0) {
      for (int j = 0; j < 3; ++j) {
        S.info->iters[j] = j < NR && ((active >> j) & 1) ? iters : 0;
        S.info->resid[j] = j < NR ? st.res[j < NR ? j : 0] * st.up[j < NR ? j : 0] : 0.0;
        S.info->bnorm[j] = j < NR ? st.bn[j < NR ? j : 0] * st.up[j < NR ? j : 0] : 0.0;
      }
      S.info->outer = updates;
      S.info->df_updates = op.df ? updates : 0;
      set_status(S.info, status == CPM_OK && unconv ? CPM_NOT_CONVERGED : status);
    } else if (status != CPM_OK) {
      set_status(S.info, status);
    }
  }
  return true;
}

}  // namespace cpm
