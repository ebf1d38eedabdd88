// RPY mobility tensors on sm_100a: free space (src/bdsim/clib/diff_tensor.c:73-166,
// :483-549) and under Smith's Ewald summation (diff_tensor.c:170-266, :553-1087).
//
// One CTA owns a 16 x 16 tile of bead pairs on or below the block diagonal.
// Bead coordinates, radii and the beads' phase factors are staged in shared
// memory; each thread evaluates one pair block (real-space image sum +
// reciprocal sum) in registers, the 48 x 48 value tile and its transpose are
// assembled in shared memory and written out with row-contiguous 16-byte
// stores.
//
// The sums are bound by the arithmetic pipes (FP64 or FP32), so they are
// arranged to need few operations per pair:
//  - the Gaussians of the images factor by axis, exp(-a^2 |s + m|^2) =
//    E_x(m_x) E_y(m_y) E_z(m_z): 15 (FP32) or 9 (FP64) exponentials instead of
//    25 or, with those inside erfc, 50; erfc(x) = erfcx(x) e^{-x^2} in FP64
//    (erfcx_poly); one reciprocal square root gives l, 1/l and 1/l^2;
//  - the reciprocal vectors +-n_x, +-n_y, +-n_z have equal weights, so the sum
//    over the signs of cos(2 pi n.s) is 8 cos cos cos (4 or 2 where components
//    vanish), and that of n_x n_y cos(2 pi n.s) is -8 n_x n_y sin sin cos: a sum
//    over one octant (34 vectors at n_max = 4 instead of a half space of 64)
//    of products of per-axis factors, with the inner sum over n_z shared by the
//    six components.  The per-axis factors of a pair come from the two beads'
//    cos and sin of 2 pi s by angle addition: no per-vector phase tables.
// The minimum image does not enter the reciprocal part (the phase is
// periodic), only the real-space images.
// Measured (one B200, m_max = 2, n_max = 4), before these forms -> now: 1000 beads
// FP64 217 -> 100 us (FP64 pipe 67% busy), FP32 107 -> 53 us (75% of the issue
// slots; a quarter of it the compensated image sum); 1999 beads FP32 374 -> 192 us.
// Larger lattices (the rolled sums), 1000 beads, alpha = sqrt(pi), m_max = 3, n_max
// = 5: FP64 494 -> 275 us, FP32 193 -> 148 us.
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace pbg {

namespace {

constexpr int TB = 16;           // beads per tile edge
constexpr int TV = 3 * TB;       // values per tile edge
constexpr int THREADS = TB * TB;

// Constants of the pair terms, cO = 1/(8 pi L), cQ = (ai^2+aj^2)/(24 pi L^3).
template <typename T>
struct PairSums {
  T cO, cQ, alpha, alpha2;
  T o;       // 2 alpha / sqrt(pi)
  T q2;      // 4 alpha^3 / sqrt(pi)
};
template <typename T>
struct PairConst : PairSums<T> {};
template <>
struct PairConst<double> : PairSums<double> {
  double k1, k4;  // exp(-alpha^2), exp(-4 alpha^2)
};

struct RpyArgs {
  PairSource src;
  const double* pos;    // N x 3, for the phases
  const double* radii;
  const double* w;      // [n_max^2 + 1][4]: P, R, S, 0 by |n|^2
  const float* w_f;
  void* M;
  void* M_lower;        // or null: also receives the lower block triangle (tiles I >= J)
  double L, invL, scale, alpha;
  double cQ0;           // 1 / (24 pi L^3)
  double self_O[6], self_Q[6];
  PairConst<double> kd;  // cQ is the pair's own
  PairConst<float> kf;
  int n, ld, smith, m_max, n_max;
  int pad;              // also write the identity padding beyond 3n (rows and columns up to ld)
};

template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

// erfc(x) for x >= 0 in FP32 from e = exp(-x^2), by Abramowitz & Stegun,
// Handbook of Mathematical Functions, 7.1.26 (Hastings' rational
// approximation): erfc(x) = t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) e^{-x^2}
// with t = 1 / (1 + p x), absolute error below 1.5e-7 (a few FP32 ulps of
// erfc's values near 1).  The real-space Ewald sum needs exp(-x^2) anyway.
__device__ __forceinline__ float erfc_as(float x, float e) {
  float t;  // 1.0f / (1 + p x)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.3275911f, x, 1.0f)));
  float p = 1.061405429f;
  p = fmaf(p, t, -1.453152027f);
  p = fmaf(p, t, 1.421413741f);
  p = fmaf(p, t, -0.284496736f);
  p = fmaf(p, t, 0.254829592f);
  return p * t * e;
}

// erfcx(x) = e^{x^2} erfc(x) for x >= 0 in FP64: with t = (x - K) / (x + K), which
// maps [0, inf) to [-1, 1) (Shepherd & Laframboise, "Chebyshev approximation of
// (1 + 2x) exp(x^2) erfc(x) in 0 <= x < inf", Math. Comp. 36, 1981), the product
// (x + K) erfcx(x) is a polynomial in t; K = 3.5, degree 22, coefficients from
// the Chebyshev interpolation at 41 nodes in 50-digit arithmetic (remainder
// below 6e-17; measured <= 5.6e-16 relative over [0, 60] with the Horner
// evaluation).  One reciprocal serves the map and the quotient; the coefficients
// are constant-bank operands (as immediates each cost two more instructions).
__constant__ double c_erfcx[23] = {
    -9.77362109186586893e-10, 1.45206297924424880e-09, 1.17592366049743058e-08, -1.53343603491223697e-08,
    -8.65216924067200682e-08, 1.06340075357857900e-07, 5.52105671274727306e-07, -7.87790522611797210e-07,
    -3.39228192284693043e-06, 7.23940800259251787e-06, 1.86470501093057966e-05, -7.47753768750334476e-05,
    -4.20620746081935295e-05, 7.14531288364273669e-04, -1.30535471416713916e-03, -3.17705028603369353e-03,
    2.65186198844626665e-02, -9.23187066429999176e-02, 2.25738621647242677e-01, -4.35256026716721534e-01,
    6.94113646634648251e-01, -9.37799724567113913e-01, 1.08705558926225998e+00,
};
__device__ __forceinline__ double erfcx_poly(double x) {
  const double q = x + 3.5;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(q));
  const double h = fma(-q, r, 1.0);  // one third-order step
  r = fma(r, fma(h, h, h), r);
  const double t = (x - 3.5) * r;
  double p = c_erfcx[0];
#pragma unroll
  for (int i = 1; i < 23; ++i) p = fma(p, t, c_erfcx[i]);
  return p * r;
}
// 1 / sqrt(x) for normal x > 0: the PTX estimate and one third-order step (Householder's
// method) y <- y + y h (1/2 + 3/8 h), h = 1 - x y^2.
__device__ __forceinline__ double rsqrt_step(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = fma(-x * y, y, 1.0);
  return fma(y * h, fma(h, 0.375, 0.5), y);
}

// Free-space RPY pair block in FP64 (diff_tensor.c:490-549), three regimes.
__device__ void rpy_pair_fp64(double ai, double aj, double rx, double ry, double rz, double out[6]) {
  const double al = ai > aj ? ai : aj, as = ai > aj ? aj : ai;
  const double d2 = rx * rx + ry * ry + rz * rz, d = sqrt(d2), aij2 = ai * ai + aj * aj;
  double c1, cd, co;
  if (d > ai + aj) {
    c1 = 1.0 / (8 * PBG_PI * d);
    cd = 1.0 + aij2 / (3 * d2);
    co = (1.0 - aij2 / d2) / d2;
  } else if (d <= al - as) {
    c1 = 1.0 / (6 * PBG_PI * al);
    cd = 1.0;
    co = 0.0;
  } else {
    const double d3 = d2 * d;
    c1 = 1.0 / (6 * PBG_PI * ai * aj);
    double c3 = (ai - aj) * (ai - aj) + 3 * d2;
    c3 *= c3;
    cd = (16 * d3 * (ai + aj) - c3) / 32 / d3;
    double c5 = (ai - aj) * (ai - aj) - d2;
    c5 *= 3 * c5;
    co = c5 / (32 * d3) / d2;
  }
  out[0] = c1 * (cd + co * rx * rx);
  out[1] = c1 * (cd + co * ry * ry);
  out[2] = c1 * (cd + co * rz * rz);
  out[3] = c1 * co * rx * ry;
  out[4] = c1 * co * rx * rz;
  out[5] = c1 * co * ry * rz;
}

// Smith-Ewald pair block (diff_tensor.c:579-648) without the overlap fix:
// M = cO * O(sigma) + cQ * Q(sigma), as six outer-product components and a multiple of the unit matrix.
template <typename T>
struct Block6 {
  T c[6] = {0, 0, 0, 0, 0, 0}, d = 0;
};
// FP32: the sum of the images, with its rounding errors carried along (r): a plain
// sum's error grows with the images (|m|_1 <= 8 at alpha = 0.05: 3.0e-6 of the
// value, 2e-7 compensated).
struct ImageSum {
  float c[6] = {0, 0, 0, 0, 0, 0}, d = 0, r[7] = {0, 0, 0, 0, 0, 0, 0};
};

// s += a b with the sum's rounding error (of the larger s and the exact product) in r.
__device__ __forceinline__ void add_compensated(float a, float b, float& s, float& r) {
  const float t = __fmaf_rn(a, b, s);
  r = __fadd_rn(r, __fmaf_rn(a, b, -__fsub_rn(t, s)));
  s = t;
}

// Adds one image at (x, y, z), l2 = |(x, y, z)|^2, e = exp(-alpha^2 l2).
__device__ __forceinline__ void add_image(const PairConst<float>& k, float x, float y, float z, float l2, float e,
                                          ImageSum& acc) {
  float il;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(il) : "f"(l2));
  const float l = l2 * il, il2 = il * il;
  const float ec = erfc_as(k.alpha * l, e);
  const float u = ec * il, v = fmaf(k.o * l, e, ec) * (il * il2);
  const float oc = (k.cO * fmaf(k.o, e, u) - k.cQ * fmaf(3.0f, v, k.q2 * e)) * il2;
  const float ox = oc * x, oy = oc * y;
  add_compensated(1.0f, fmaf(k.cO, u, k.cQ * v), acc.d, acc.r[6]);
  add_compensated(ox, x, acc.c[0], acc.r[0]);
  add_compensated(oy, y, acc.c[1], acc.r[1]);
  add_compensated(oc * z, z, acc.c[2], acc.r[2]);
  add_compensated(ox, y, acc.c[3], acc.r[3]);
  add_compensated(ox, z, acc.c[4], acc.r[4]);
  add_compensated(oy, z, acc.c[5], acc.r[5]);
}
__device__ __forceinline__ void add_image(const PairConst<double>& k, double x, double y, double z, double l2,
                                          double e, Block6<double>& acc) {
  const double il = rsqrt_step(l2), l = l2 * il, il2 = il * il;
  const double ec = erfcx_poly(k.alpha * l) * e;
  const double u = ec * il, v = fma(k.o * l, e, ec) * (il * il2);
  acc.d += k.cO * u + k.cQ * v;
  const double oc = (k.cO * fma(k.o, e, u) - k.cQ * fma(3.0, v, k.q2 * e)) * il2;
  const double ox = oc * x, oy = oc * y;
  acc.c[0] = fma(ox, x, acc.c[0]);
  acc.c[1] = fma(oy, y, acc.c[1]);
  acc.c[2] = fma(oc * z, z, acc.c[2]);
  acc.c[3] = fma(ox, y, acc.c[3]);
  acc.c[4] = fma(ox, z, acc.c[4]);
  acc.c[5] = fma(oy, z, acc.c[5]);
}
// exp(-alpha^2 (s + m)^2), m = -2 .. 2.  FP32: one MUFU exponential each.  FP64:
// three exponentials, E(m) = E(0) exp(-2 alpha^2 s m) exp(-alpha^2 m^2) (the products
// taken in an order that cannot overflow for 2 alpha^2 |s| <= 700: every minimum-image
// vector for alpha <= 16; pair_sums takes the other pairs to real_sum).
__device__ __forceinline__ void gauss_axis(const PairConst<float>& k, float s, float (&e)[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const float x = s + (float)(m - 2);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e[m]) : "f"(-1.44269504f * k.alpha2 * (x * x)));
  }
}
__device__ __forceinline__ void gauss_axis(const PairConst<double>& k, double s, double (&e)[5]) {
  const double u = 2.0 * k.alpha2 * s, gp = exp(-u), gm = exp(u);
  e[2] = exp(-k.alpha2 * s * s);
  const double p = e[2] * gp, m = e[2] * gm;
  e[3] = p * k.k1;
  e[1] = m * k.k1;
  e[4] = p * (gp * k.k4);
  e[0] = m * (gm * k.k4);
}

// The images |m|_1 <= m_max <= 2 (25 at most), the nearest one (m = 0) first.
// FP64: it is returned apart from the others, which are summed among themselves.
// FP32: one compensated sum (main and rest are the same: the largest term comes
// first, as add_compensated wants it); unrolled, the per-axis values in registers.
// FP64: the loops stay rolled (an image is about 100 instructions) with the axis
// values selected by the uniform loop counters; images +-m_z run side by side.
template <typename T, typename A>
__device__ __forceinline__ void real_sum_small(const PairConst<T>& k, T sx, T sy, T sz, int m_max, A& main, A& rest) {
  T ex[5], ey[5], ez[5];
  gauss_axis(k, sx, ex);
  gauss_axis(k, sy, ey);
  gauss_axis(k, sz, ez);
  add_image(k, sx, sy, sz, sx * sx + sy * sy + sz * sz, ex[2] * ey[2] * ez[2], main);
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int mx = -2; mx <= 2; ++mx)
#pragma unroll
      for (int my = -2; my <= 2; ++my) {
        const int r = (mx < 0 ? -mx : mx) + (my < 0 ? -my : my);
        if (r > 2 || r > m_max) continue;
        const T x = sx + (T)mx, y = sy + (T)my, xy = x * x + y * y, e = ex[mx + 2] * ey[my + 2];
#pragma unroll
        for (int mz = -2; mz <= 2; ++mz) {
          const int q = r + (mz < 0 ? -mz : mz);
          if (q == 0 || q > 2 || q > m_max) continue;
          const T z = sz + (T)mz;
          add_image(k, x, y, z, fmaf(z, z, xy), e * ez[mz + 2], rest);
        }
      }
  } else {
    auto pick = [](const T (&v)[5], int m) { return m == -2 ? v[0] : m == -1 ? v[1] : m == 0 ? v[2] : m == 1 ? v[3] : v[4]; };
#pragma unroll 1
    for (int mx = -m_max; mx <= m_max; ++mx) {
      const int rx = m_max - (mx < 0 ? -mx : mx);
      const T x = sx + (T)mx, fx = pick(ex, mx);
#pragma unroll 1
      for (int my = -rx; my <= rx; ++my) {
        const int ry = rx - (my < 0 ? -my : my);
        const T y = sy + (T)my, xy = x * x + y * y, e = fx * pick(ey, my);
        if (mx != 0 || my != 0) add_image(k, x, y, sz, fma(sz, sz, xy), e * ez[2], rest);
#pragma unroll 1
        for (int mz = 1; mz <= ry; ++mz) {
          const T z0 = sz + (T)mz, z1 = sz - (T)mz;
          add_image(k, x, y, z0, fma(z0, z0, xy), e * (mz == 1 ? ez[3] : ez[4]), rest);
          add_image(k, x, y, z1, fma(z1, z1, xy), e * (mz == 1 ? ez[1] : ez[0]), rest);
        }
      }
    }
  }
}

// Any m_max: one exponential per image.
template <typename T, typename A>
__device__ __forceinline__ void real_sum(const PairConst<T>& k, T sx, T sy, T sz, int m_max, A& main, A& rest) {
  auto image = [&](int mx, int my, int mz, A& acc) {
    const T x = sx + (T)mx, y = sy + (T)my, z = sz + (T)mz, l2 = x * x + y * y + z * z;
    T e;
    if constexpr (sizeof(T) == 4) e = __expf(-k.alpha2 * l2);
    else e = exp(-k.alpha2 * l2);
    add_image(k, x, y, z, l2, e, acc);
  };
  image(0, 0, 0, main);
#pragma unroll 1
  for (int mx = -m_max; mx <= m_max; ++mx) {
    const int rx = m_max - (mx < 0 ? -mx : mx);
#pragma unroll 1
    for (int my = -rx; my <= rx; ++my) {
      const int ry = rx - (my < 0 ? -my : my);
#pragma unroll 1
      for (int mz = -ry; mz <= ry; ++mz)
        if (mx != 0 || my != 0 || mz != 0) image(mx, my, mz, rest);
    }
  }
}

// Per-axis factors of the octant sum: C(k) = 2 cos(k t), S(k) = 2 sin(k t) for
// k > 0, C(0) = 1 -- the factors 2 make the products the sums over the signs.
template <typename T>
__device__ __forceinline__ void axis_base(typename Vec2<T>::type pi, typename Vec2<T>::type pj, T& c, T& s) {
  c = pi.x * pj.x + pi.y * pj.y;
  s = pi.y * pj.x - pi.x * pj.y;
}

// Reciprocal vectors |n|_1 <= n_max <= 4, unrolled; w: [n^2][4] in shared memory.
template <typename T>
__device__ __forceinline__ void recip_sum_small(const PairConst<T>& k, const typename Vec2<T>::type* pi,
                                                const typename Vec2<T>::type* pj, const T* w, int n_max,
                                                Block6<T>& acc) {
  T C[3][5], S[3][5];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T c, s;
    axis_base<T>(pi[a], pj[a], c, s);
    const T c2 = (T)2 * c * c - (T)1, s2 = (T)2 * s * c;
    C[a][0] = (T)1;
    S[a][0] = (T)0;
    C[a][1] = (T)2 * c;
    S[a][1] = (T)2 * s;
    C[a][2] = (T)2 * c2;
    S[a][2] = (T)2 * s2;
    C[a][3] = (T)2 * (c2 * c - s2 * s);
    S[a][3] = (T)2 * (s2 * c + c2 * s);
    C[a][4] = (T)2 * ((T)2 * c2 * c2 - (T)1);
    S[a][4] = (T)4 * s2 * c2;
  }
  T G[17], P[17];
#pragma unroll
  for (int q = 1; q <= 16; ++q) {
    const bool used = q <= 6 || q == 8 || q == 9 || q == 10 || q == 16;
    if (used && q <= n_max * n_max) {
      P[q] = w[4 * q];
      G[q] = k.cQ * w[4 * q + 2] - k.cO * w[4 * q + 1];
    } else {
      P[q] = G[q] = (T)0;
    }
  }
  T dr = 0;
#pragma unroll
  for (int nx = 0; nx <= 4; ++nx)
#pragma unroll
    for (int ny = 0; ny <= 4; ++ny) {
      if (nx + ny > 4 || nx + ny > n_max) continue;
      T ad = 0, ag = 0, az = 0, bz = 0;
#pragma unroll
      for (int nz = 0; nz <= 4; ++nz) {
        const int q = nx * nx + ny * ny + nz * nz;
        if (q == 0 || nx + ny + nz > 4 || nx + ny + nz > n_max) continue;
        if (nz == 0) {
          ad += P[q];
          ag += G[q];
        } else {
          const T gc = G[q] * C[2][nz];
          ad += P[q] * C[2][nz];
          ag += gc;
          az += (T)(nz * nz) * gc;
          bz += (T)nz * (G[q] * S[2][nz]);
        }
      }
      const T cx = C[0][nx], cy = C[1][ny], cxy = nx == 0 ? cy : ny == 0 ? cx : cx * cy, g = cxy * ag;
      dr += cxy * ad;
      if (nx > 0) acc.c[0] += (T)(nx * nx) * g;
      if (ny > 0) acc.c[1] += (T)(ny * ny) * g;
      acc.c[2] += cxy * az;
      if (nx > 0 && ny > 0) acc.c[3] -= (T)(nx * ny) * (S[0][nx] * S[1][ny] * ag);
      if (nx > 0) acc.c[4] -= (T)nx * ((ny == 0 ? S[0][nx] : S[0][nx] * cy) * bz);
      if (ny > 0) acc.c[5] -= (T)ny * ((nx == 0 ? S[1][ny] : cx * S[1][ny]) * bz);
    }
  acc.d += k.cO * dr;
}

// Any n_max: the same sum with rolled loops, each axis stepped by angle addition.
template <typename T>
__device__ __forceinline__ void recip_sum(const PairConst<T>& k, const typename Vec2<T>::type* pi,
                                          const typename Vec2<T>::type* pj, const T* w, int n_max, Block6<T>& acc) {
  T c1[3], s1[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) axis_base<T>(pi[a], pj[a], c1[a], s1[a]);
  auto step = [](T& c, T& s, T cb, T sb) {
    const T t = c * cb - s * sb;
    s = s * cb + c * sb;
    c = t;
  };
  T dr = 0, cx = 1, sx = 0;
#pragma unroll 1
  for (int nx = 0; nx <= n_max; ++nx) {
    const T fx = nx ? (T)2 : (T)1;
    T cy = 1, sy = 0;
#pragma unroll 1
    for (int ny = 0; ny <= n_max - nx; ++ny) {
      const T f = ny ? (T)2 * fx : fx;
      T cz = 1, sz = 0, ad = 0, ag = 0, az = 0, bz = 0;
#pragma unroll 1
      for (int nz = 0; nz <= n_max - nx - ny; ++nz) {
        const int q = nx * nx + ny * ny + nz * nz;
        if (q) {
          const T fz = nz ? (T)2 * f : f, g = fz * (k.cQ * w[4 * q + 2] - k.cO * w[4 * q + 1]);
          ad += fz * w[4 * q] * cz;
          ag += g * cz;
          az += (T)(nz * nz) * (g * cz);
          bz += (T)nz * (g * sz);
        }
        step(cz, sz, c1[2], s1[2]);
      }
      const T g = cx * cy * ag;
      dr += cx * cy * ad;
      acc.c[0] += (T)(nx * nx) * g;
      acc.c[1] += (T)(ny * ny) * g;
      acc.c[2] += cx * cy * az;
      acc.c[3] -= (T)(nx * ny) * (sx * sy * ag);
      acc.c[4] -= (T)nx * (sx * cy * bz);
      acc.c[5] -= (T)ny * (cx * sy * bz);
      step(cy, sy, c1[1], s1[1]);
    }
    step(cx, sx, c1[0], s1[0]);
  }
  acc.d += k.cO * dr;
}

// (cos, sin)(2 pi f) of a bead coordinate in units of L.  FP32: the fraction
// rounded to float, and the rest of it (below 2^-25) by a first-order step, so
// both values are rounded once like the FP64 ones.
__device__ __forceinline__ double2 phase_of(double f, double) {
  double2 v;
  sincospi(2.0 * (f - rint(f)), &v.y, &v.x);
  return v;
}
__device__ __forceinline__ float2 phase_of(double f, float) {
  const double r = f - rint(f);
  const float h = (float)r, d = (float)((r - (double)h) * (2.0 * PBG_PI));
  float s, c;
  sincospif(2.0f * h, &s, &c);
  return make_float2(fmaf(-s, d, c), fmaf(c, d, s));
}

// pbg_min_image with at most one shift each way for |x| < 1.5 L (all of them for
// positions kept in the box); the same result otherwise, by its loops.
__device__ __forceinline__ double min_image_once(double x, double L) {
  const double h = L / 2.0;
  double y = x >= h ? x - L : x;
  y = y <= -h ? y + L : y;
  if (!(fabs(y) <= h)) y = pbg_min_image(x, L);
  return y;
}

// Row stride of the staged value tiles: rows start on 16-byte boundaries.
template <typename T> struct OutLd { static constexpr int v = sizeof(T) == 4 ? TV + 4 : TV + 2; };

// Rows row0 .. row0+47, columns col0 .. col0+47 of M from a staged tile, within
// the order n3: 16 bytes per store where M's rows allow it (vec).
template <typename T>
__device__ __forceinline__ void store_out(const T* s, T* M, int ld, int row0, int col0, int n3, bool vec) {
  constexpr int W = 16 / (int)sizeof(T), LDO = OutLd<T>::v;
#pragma unroll
  for (int q = 0; q < (TV * TV / W + THREADS - 1) / THREADS; ++q) {
    const int t = threadIdx.x + q * THREADS, r = t / (TV / W), c = (t % (TV / W)) * W;
    if (r >= TV || row0 + r >= n3) continue;
    T* g = M + (size_t)(row0 + r) * ld + col0 + c;
    if (vec && col0 + c + W <= n3) {
      *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(s + r * LDO + c);
    } else {
#pragma unroll
      for (int u = 0; u < W; ++u)
        if (col0 + c + u < n3) g[u] = s[r * LDO + c + u];
    }
  }
}

// Both sums of a pair: the nearest image, the other images, the reciprocal vectors.
template <bool SMALL, typename T, typename V2, typename A>
__device__ __forceinline__ void pair_sums(const PairConst<T>& k, const V2* pi, const V2* pj, const T* w,
                                          const RpyArgs& a, T sx, T sy, T sz, A& main, A& images, Block6<T>& recip) {
  if constexpr (SMALL) {
    recip_sum_small<T>(k, pi, pj, w, a.n_max, recip);
    // pair vectors of a caller can lie any number of boxes away (see gauss_axis)
    if (sizeof(T) == 8 && 2.0 * k.alpha2 * fmax(fmax(fabs(sx), fabs(sy)), fabs(sz)) > 700.0)
      real_sum<T>(k, sx, sy, sz, a.m_max, main, images);
    else
      real_sum_small<T>(k, sx, sy, sz, a.m_max, main, images);
  } else {
    recip_sum<T>(k, pi, pj, w, a.n_max, recip);
    real_sum<T>(k, sx, sy, sz, a.m_max, main, images);
  }
}

// One 16 x 16 bead tile (I, J), I >= J, of the tensor described by `a`.
// SMALL: m_max <= 2 and n_max <= 4 (the unrolled sums; the defaults' range).
template <typename T, bool SMALL>
__device__ __forceinline__ void rpy_tile_body(const RpyArgs& a, int I, int J, void* M_lower) {
  using V2 = typename Vec2<T>::type;
  constexpr int LDO = OutLd<T>::v;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // layout: tile and transposed tile [TV][LDO] T | weights [n_max^2 + 1][4] T
  T* s_out = reinterpret_cast<T*>(smem_raw);
  T* s_outT = s_out + TV * LDO;
  T* s_w = s_outT + TV * LDO;
  __shared__ V2 s_ph[2 * TB][3];
  __shared__ double s_pos[2 * TB][3], s_rad[2 * TB];

  const int tid = threadIdx.x;
  const int ti = tid / TB, tj = tid % TB;
  const int i = I * TB + ti, j = J * TB + tj;
  const int n = a.n;

  if (tid < 2 * TB * 3) {
    const int b = tid / 3, c = tid % 3, bead = b < TB ? I * TB + b : J * TB + (b - TB);
    if (bead < n) {
      if (a.src.pos) s_pos[b][c] = a.src.pos[3 * bead + c];
      if (a.smith) s_ph[b][c] = phase_of(a.pos[3 * bead + c] * a.invL, T());
    }
  } else if (tid >= 128 && tid < 128 + 2 * TB) {
    const int b = tid - 128, bead = b < TB ? I * TB + b : J * TB + (b - TB);
    if (bead < n) s_rad[b] = a.radii[bead];
  }
  if (a.smith) {
    const T* gsrc = sizeof(T) == 8 ? reinterpret_cast<const T*>(a.w) : reinterpret_cast<const T*>(a.w_f);
    for (int t = tid; t < 4 * (a.n_max * a.n_max + 1); t += THREADS) s_w[t] = gsrc[t];
  }
  __syncthreads();

  const bool active = (i < n) && (j < n) && !(I == J && ti < tj);
  if (active) {
    T v[6];
    const double ai = s_rad[ti], aj = s_rad[TB + tj];
    if (i == j) {
      // Self block (diff_tensor.c:553-575); the lattice sums are a-independent.
      double blk[6] = {0, 0, 0, 0, 0, 0};
      const double c1 = 1.0 / (6 * PBG_PI * ai);
      if (a.smith) {
        const double sqrt_pi = 1.7724538509055160273;
        const double c2 = 3 * ai / (4 * a.L);
        const double c3 = ai * ai * ai / (2 * a.L * a.L * a.L);
        const double so = 1.5 * a.alpha * ai / (sqrt_pi * a.L);
        const double sq = a.alpha * a.alpha * a.alpha * ai * ai * ai / (a.L * a.L * a.L * 3.0 * sqrt_pi);
        for (int c = 0; c < 3; ++c)
          blk[c] = c1 * (1.0 + c2 * (a.self_O[c] - so) + c3 * (a.self_Q[c] - sq));
        for (int c = 3; c < 6; ++c) blk[c] = c1 * (c2 * a.self_O[c] + c3 * a.self_Q[c]);
      } else {
        blk[0] = blk[1] = blk[2] = c1;
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) v[c] = (T)(blk[c] * a.scale);
    } else {
      // Pair vector handed to the reference kernels: -minimg(r_i - r_j).
      double rx, ry, rz;
      if (a.src.pairs) {
        get_pair_vector(a.src, i, j, rx, ry, rz);
      } else {
        rx = -min_image_once(s_pos[ti][0] - s_pos[TB + tj][0], a.src.L);
        ry = -min_image_once(s_pos[ti][1] - s_pos[TB + tj][1], a.src.L);
        rz = -min_image_once(s_pos[ti][2] - s_pos[TB + tj][2], a.src.L);
      }
      if (a.smith) {
        PairConst<T> k;
        if constexpr (sizeof(T) == 8) k = a.kd;
        else k = a.kf;
        k.cQ = (T)((ai * ai + aj * aj) * a.cQ0);
        const T sx = (T)(rx * a.invL), sy = (T)(ry * a.invL), sz = (T)(rz * a.invL);
        Block6<T> rest;
        double blk[6];
        if constexpr (sizeof(T) == 8) {
          Block6<T> main;
          pair_sums<SMALL>(k, s_ph[ti], s_ph[TB + tj], s_w, a, sx, sy, sz, main, rest, rest);
#pragma unroll
          for (int c = 0; c < 6; ++c) blk[c] = main.c[c] + (c < 3 ? rest.c[c] + (main.d + rest.d) : rest.c[c]);
        } else {
          // FP32 sums, added and scaled in FP64 and rounded once
          ImageSum im;
          pair_sums<SMALL>(k, s_ph[ti], s_ph[TB + tj], s_w, a, sx, sy, sz, im, im, rest);
          const double d = (double)(im.d + (im.r[6] + rest.d));
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const double o = (double)(im.c[c] + (im.r[c] + rest.c[c]));
            blk[c] = c < 3 ? o + d : o;
          }
        }
        const double d2 = rx * rx + ry * ry + rz * rz;
        if (d2 < (ai + aj) * (ai + aj)) {
          // Overlap fix (diff_tensor.c:614-643): swap far-field RPY for the
          // overlapping-regime RPY.
          double near[6], far[6];
          rpy_pair_fp64(ai, aj, rx, ry, rz, near);
          const double d = sqrt(d2), aij2 = ai * ai + aj * aj;
          const double f1 = 1.0 / (8 * PBG_PI * d), f2 = 1.0 + aij2 / (3 * d2);
          const double f3 = (1.0 - aij2 / d2) / d2;
          far[0] = f1 * (f2 + f3 * rx * rx);
          far[1] = f1 * (f2 + f3 * ry * ry);
          far[2] = f1 * (f2 + f3 * rz * rz);
          far[3] = f1 * f3 * rx * ry;
          far[4] = f1 * f3 * rx * rz;
          far[5] = f1 * f3 * ry * rz;
#pragma unroll
          for (int c = 0; c < 6; ++c) v[c] = (T)((blk[c] + (near[c] - far[c])) * a.scale);
        } else {
#pragma unroll
          for (int c = 0; c < 6; ++c) v[c] = (T)(blk[c] * a.scale);
        }
      } else {
        double blk[6];
        rpy_pair_fp64(ai, aj, rx, ry, rz, blk);
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = (T)(blk[c] * a.scale);
      }
    }
    const int comp[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        s_out[(3 * ti + r) * LDO + 3 * tj + c] = v[comp[r][c]];
        (I == J ? s_out : s_outT)[(3 * tj + r) * LDO + 3 * ti + c] = v[comp[r][c]];
      }
  }
  __syncthreads();

  T* M = reinterpret_cast<T*>(a.M);
  T* ML = reinterpret_cast<T*>(M_lower);
  const int n3 = 3 * n, row0 = TV * I, col0 = TV * J;
  const bool vec = a.ld % (16 / (int)sizeof(T)) == 0 && reinterpret_cast<uintptr_t>(M) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(ML) % 16 == 0;
  store_out(s_out, M, a.ld, row0, col0, n3, vec);
  if (ML) store_out(s_out, ML, a.ld, row0, col0, n3, vec);
  if (I != J) store_out(s_outT, M, a.ld, col0, row0, n3, vec);
  if (a.pad && (I + 1) * TB >= n) {
    // the last tile row also writes the identity padding beside its columns:
    // rows n3 .. ld-1 (and, in M, their transposes)
    const int c1 = I == J ? a.ld : col0 + TV, width = c1 - col0;
    for (int t = tid; t < (a.ld - n3) * width; t += THREADS) {
      const int r = n3 + t / width, c = col0 + t % width;
      const T v = r == c ? (T)1 : (T)0;
      M[(size_t)r * a.ld + c] = v;
      if (c < n3) M[(size_t)c * a.ld + r] = v;
      if (ML) ML[(size_t)r * a.ld + c] = v;
    }
  }
}

template <typename T, bool SMALL>
__global__ void __launch_bounds__(THREADS, sizeof(T) == 8 ? 2 : 3) rpy_tile_kernel(RpyArgs a) {
  // Tile (I, J), I >= J, from the linear lower-triangle block index.
  const int b = blockIdx.x;
  int I = (int)((sqrtf(8.0f * b + 1.0f) - 1.0f) * 0.5f);
  while ((I + 1) * (I + 2) / 2 <= b) ++I;
  while (I * (I + 1) / 2 > b) --I;
  const int J = b - I * (I + 1) / 2;
  rpy_tile_body<T, SMALL>(a, I, J, a.M_lower);
}

// Batched build: block b computes tile (work[b].y, work[b].z) of replica work[b].x;
// with fill_lower the lower block triangle also goes to the replica's M_lower.
template <typename T, bool SMALL>
__global__ void __launch_bounds__(THREADS, sizeof(T) == 8 ? 2 : 3) rpy_batch_kernel(const RpyArgs* __restrict__ args,
                                                            const int4* __restrict__ work, int fill_lower) {
  const int4 w = work[blockIdx.x];
  rpy_tile_body<T, SMALL>(args[w.x], w.y, w.z, fill_lower ? args[w.x].M_lower : nullptr);
}

__global__ void positions_from_pairs_kernel(const double* __restrict__ pairs, int n, double* __restrict__ pos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (i == 0) {
    pos[0] = pos[1] = pos[2] = 0.0;
    return;
  }
  const long long k = 3LL * (i - 1);  // pair (i, 0)
  pos[3 * i + 0] = -pairs[k];
  pos[3 * i + 1] = -pairs[k + 1];
  pos[3 * i + 2] = -pairs[k + 2];
}

// ---------------------------------------------------------------- host side

// Self-block lattice sums (diff_tensor.c:652-849) without the a-dependent
// self terms, in the reference's loop order.
void host_self_sums(double alpha, int m_max, int n_max, double O[6], double Q[6]) {
  const double sqrt_pi = std::sqrt(PBG_PI), alpha2 = alpha * alpha, alpha3 = alpha * alpha2;
  const double kexp = -PBG_PI * PBG_PI / alpha2;
  for (int c = 0; c < 6; ++c) O[c] = Q[c] = 0.0;
  auto outer = [](double x, double y, double z, double v[6]) {
    v[0] = x * x; v[1] = y * y; v[2] = z * z; v[3] = x * y; v[4] = x * z; v[5] = y * z;
  };
  double mm[6];
  for (int mx = -m_max; mx <= m_max; ++mx)
    for (int my = -(m_max - std::abs(mx)); my <= m_max - std::abs(mx); ++my)
      for (int mz = -(m_max - std::abs(mx) - std::abs(my)); mz <= m_max - std::abs(mx) - std::abs(my); ++mz) {
        if (!mx && !my && !mz) continue;
        const double l2 = mx * mx + my * my + mz * mz, l = std::sqrt(l2), l3 = l2 * l;
        outer(mx, my, mz, mm);
        const double ec = std::erfc(alpha * l);
        const double e = std::exp(-alpha2 * l2);
        // O: erfc * O(m) + (2 alpha / sqrt(pi)) exp(-alpha^2 m^2) / m^2 * m m
        const double o_fn[6] = {(1 + mm[0] / l2) / l, (1 + mm[1] / l2) / l, (1 + mm[2] / l2) / l,
                                mm[3] / l3, mm[4] / l3, mm[5] / l3};
        const double w_o = 2 * alpha / sqrt_pi * e / l2;
        for (int c = 0; c < 6; ++c) O[c] += ec * o_fn[c] + w_o * mm[c];
        // Q: (erfc + 2/sqrt(pi) alpha m e) * Q(m) - 4 alpha^3/sqrt(pi) e / m^2 * m m
        const double am = alpha * l, l5 = l3 * l2;
        const double q_fn[6] = {(1 - 3 * mm[0] / l2) / l3, (1 - 3 * mm[1] / l2) / l3, (1 - 3 * mm[2] / l2) / l3,
                                -3 * mm[3] / l5, -3 * mm[4] / l5, -3 * mm[5] / l5};
        const double w_q1 = std::erfc(am) + 2 / sqrt_pi * am * e;
        const double w_q2 = 2 / sqrt_pi * 2 * alpha3 * e / l2;
        for (int c = 0; c < 6; ++c) Q[c] += w_q1 * q_fn[c] - w_q2 * mm[c];
      }
  for (int nx = -n_max; nx <= n_max; ++nx)
    for (int ny = -(n_max - std::abs(nx)); ny <= n_max - std::abs(nx); ++ny)
      for (int nz = -(n_max - std::abs(nx) - std::abs(ny)); nz <= n_max - std::abs(nx) - std::abs(ny); ++nz) {
        if (!nx && !ny && !nz) continue;
        const double nl2 = nx * nx + ny * ny + nz * nz;
        outer(nx, ny, nz, mm);
        const double w = 2.0 / PBG_PI / nl2 * std::exp(kexp * nl2);
        const double t = 1.0 / nl2 - kexp;
        for (int c = 0; c < 3; ++c) O[c] += w * (1.0 - t * mm[c]);
        for (int c = 3; c < 6; ++c) O[c] += w * (-t * mm[c]);
        const double wq = 4 * PBG_PI * std::exp(kexp * nl2) / nl2;
        for (int c = 0; c < 6; ++c) Q[c] += wq * mm[c];
      }
}

std::mutex g_tables_mu;
std::map<std::tuple<double, int, int>, EwaldTables*> g_tables;

}  // namespace

long long lattice_points_l1(int m) {
  // integer points with |x| + |y| + |z| <= m: (2m + 1)(2m^2 + 2m + 3) / 3
  const long long mm = m;
  return (2 * mm + 1) * (2 * mm * mm + 2 * mm + 3) / 3;
}

void build_lattice_tables(double alpha, int m_max, int n_max, std::vector<double>& w, double self_O[6],
                          double self_Q[6]) {
  w.assign(4, 0.0);
  const double kk = PBG_PI * PBG_PI / (alpha * alpha);
  for (int q = 1; q <= n_max * n_max; ++q) {
    const double nl2 = q, e = std::exp(-kk * nl2);
    const double P = (2.0 / PBG_PI) / nl2 * e;  // O weight
    const double R = P * (1.0 + kk * nl2) / nl2;  // O weight * t
    const double S = 4 * PBG_PI * e / nl2;        // Q weight
    const double row[4] = {P, R, S, 0};
    w.insert(w.end(), row, row + 4);
  }
  host_self_sums(alpha, m_max, n_max, self_O, self_Q);
}

int get_ewald_tables(double alpha, int m_max, int n_max, const EwaldTables** out) {
  if (m_max < 0 || n_max < 0 || m_max > 16 || n_max > 16 || !(alpha > 0)) {
    pbg_set_error_message("invalid Ewald parameters alpha=%g m_max=%d n_max=%d", alpha, m_max, n_max);
    return PBG_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(g_tables_mu);
  auto key = std::make_tuple(alpha, m_max, n_max);
  auto it = g_tables.find(key);
  if (it != g_tables.end()) {
    *out = it->second;
    return PBG_OK;
  }
  auto* t = new EwaldTables();
  t->alpha = alpha;
  t->m_max = m_max;
  t->n_max = n_max;
  std::vector<double> w;
  build_lattice_tables(alpha, m_max, n_max, w, t->self_O, t->self_Q);
  const std::vector<float> w_f(w.begin(), w.end());
  if (cudaMalloc(&t->d_w, w.size() * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&t->d_w_f, w.size() * sizeof(float)) != cudaSuccess) {
    pbg_set_error_message("cudaMalloc failed for Ewald tables");
    return PBG_ERR_NOMEM;
  }
  PBG_CUDA_TRY(cudaMemcpy(t->d_w, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice));
  PBG_CUDA_TRY(cudaMemcpy(t->d_w_f, w_f.data(), w_f.size() * sizeof(float), cudaMemcpyHostToDevice));
  g_tables[key] = t;
  *out = t;
  return PBG_OK;
}

int launch_positions_from_pairs(const double* pairs, int n, double* pos, cudaStream_t st) {
  if (n <= 0) return PBG_OK;
  positions_from_pairs_kernel<<<(n + 127) / 128, 128, 0, st>>>(pairs, n, pos);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

// Shared memory beside the static arrays: the two value tiles and the weights.
static size_t rpy_smem_bytes(const EwaldTables* t, int precision, bool smith) {
  if (precision == PBG_PREC_FP64)
    return sizeof(double) * (2 * TV * OutLd<double>::v + (smith ? 4 * (t->n_max * t->n_max + 1) : 0));
  return sizeof(float) * (2 * TV * OutLd<float>::v + (smith ? 4 * (t->n_max * t->n_max + 1) : 0));
}

// The lattice sizes that the entry points take: images of 32 bytes and
// reciprocal half-vectors of 72 (FP64) or 36 (FP32) times 8 bytes within
// 227 KB beside a value tile.
static int check_lattice(const EwaldTables* t, int precision) {
  const size_t ts = precision == PBG_PREC_FP64 ? 8 : 4;
  const size_t images = (size_t)lattice_points_l1(t->m_max), half = ((size_t)lattice_points_l1(t->n_max) - 1) / 2;
  const size_t bytes = ts * TV * (TV + 1) + 32 * images + 72 * ts * half;
  if (bytes <= 227 * 1024) return PBG_OK;
  pbg_set_error_message("Ewald n-set too large (%zu bytes of tables)", bytes);
  return PBG_ERR_ARG;
}

// The unrolled sums cover ewald_real <= 2 and ewald_imag <= 4 (the usual
// parameters and everything below them): a pair costs about half of the rolled
// loops' instructions, which compute one exponential per image and step the
// phases by angle addition.
static bool small_lattice(const EwaldTables* t, bool smith) {
  return !smith || (t->m_max <= 2 && t->n_max <= 4 && t->alpha <= 16.0);  // alpha: see gauss_axis
}

static void fill_args(RpyArgs& a, const PairSource& src, const double* pos, const double* radii, bool smith,
                      const EwaldTables* t, double scale, void* M, void* M_lower, int ld, bool pad) {
  a.src = src;
  a.pos = pos;
  a.radii = radii;
  a.M = M;
  a.M_lower = M_lower;
  a.L = src.L;
  a.invL = 1.0 / src.L;
  a.cQ0 = 1.0 / (24 * PBG_PI * src.L * src.L * src.L);
  a.scale = scale;
  a.n = src.n;
  a.ld = ld;
  a.smith = smith ? 1 : 0;
  a.pad = pad ? 1 : 0;
  if (smith && t) {
    a.alpha = t->alpha;
    const double al = t->alpha, sqrt_pi = std::sqrt(PBG_PI);
    a.kd = PairConst<double>{{1.0 / (8 * PBG_PI * src.L), 0.0, al, al * al, 2 * al / sqrt_pi, 4 * al * al * al / sqrt_pi},
                             std::exp(-al * al), std::exp(-4 * al * al)};
    a.kf = PairConst<float>{{(float)a.kd.cO, 0.0f, (float)al, (float)a.kd.alpha2, (float)a.kd.o, (float)a.kd.q2}};
    a.w = t->d_w;
    a.w_f = t->d_w_f;
    a.m_max = t->m_max;
    a.n_max = t->n_max;
    for (int c = 0; c < 6; ++c) {
      a.self_O[c] = t->self_O[c];
      a.self_Q[c] = t->self_Q[c];
    }
  }
}

// Launches `kernel` with `smem` bytes, raising its limit where that is above
// the 48 KB default.
template <typename K, typename... A>
static int launch_tiles(K kernel, int blocks, size_t smem, cudaStream_t st, A... args) {
  if (smem > 40 * 1024)
    PBG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<blocks, THREADS, smem, st>>>(args...);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

int launch_rpy_tensor(const PairSource& src, const double* pos, const double* radii, bool smith,
                      const EwaldTables* t, double scale, int precision, void* M, int ld, cudaStream_t st,
                      void* M_lower, bool pad) {
  const int n = src.n;
  if (n <= 0) return PBG_OK;
  if (smith && !t) return PBG_ERR_ARG;
  if (smith)
    if (int rc = check_lattice(t, precision)) return rc;
  RpyArgs a{};
  fill_args(a, src, pos, radii, smith, t, scale, M, M_lower, ld, pad);
  const int tiles = (n + TB - 1) / TB, blocks = tiles * (tiles + 1) / 2;
  const size_t smem = rpy_smem_bytes(t, precision, smith);
  const bool small = small_lattice(t, smith);
  if (precision == PBG_PREC_FP64)
    return small ? launch_tiles(rpy_tile_kernel<double, true>, blocks, smem, st, a)
                 : launch_tiles(rpy_tile_kernel<double, false>, blocks, smem, st, a);
  return small ? launch_tiles(rpy_tile_kernel<float, true>, blocks, smem, st, a)
               : launch_tiles(rpy_tile_kernel<float, false>, blocks, smem, st, a);
}

size_t rpy_batch_arg_bytes() { return sizeof(RpyArgs); }

void rpy_batch_arg(const double* pos, const double* radii, int n, double L, bool smith, const EwaldTables* t,
                   double scale, void* M, void* M_lower, int ld, void* dst) {
  RpyArgs a{};
  const PairSource src{pos, nullptr, n, L};
  fill_args(a, src, pos, radii, smith, t, scale, M, M_lower, ld, true);
  std::memcpy(dst, &a, sizeof(a));
}

void rpy_batch_work(int replica, int n, std::vector<int4>& work) {
  const int tiles = (n + TB - 1) / TB;
  for (int I = 0; I < tiles; ++I)
    for (int J = 0; J <= I; ++J) work.push_back(make_int4(replica, I, J, 0));
}

// args: device array of the replicas' argument blocks (rpy_batch_arg).
// fill_lower: each replica's lower block triangle also goes to its M_lower
// (the matrix the step factors next).
int launch_rpy_batch(int precision, bool smith, const EwaldTables* t, const void* args, const int4* work,
                     int nwork, bool fill_lower, cudaStream_t st) {
  if (nwork <= 0) return PBG_OK;
  if (smith)
    if (int rc = check_lattice(t, precision)) return rc;
  const RpyArgs* a = static_cast<const RpyArgs*>(args);
  const size_t smem = rpy_smem_bytes(t, precision, smith);
  const bool small = small_lattice(t, smith);
  const int fill = fill_lower ? 1 : 0;
  if (precision == PBG_PREC_FP64)
    return small ? launch_tiles(rpy_batch_kernel<double, true>, nwork, smem, st, a, work, fill)
                 : launch_tiles(rpy_batch_kernel<double, false>, nwork, smem, st, a, work, fill);
  return small ? launch_tiles(rpy_batch_kernel<float, true>, nwork, smem, st, a, work, fill)
               : launch_tiles(rpy_batch_kernel<float, false>, nwork, smem, st, a, work, fill);
}

}  // namespace pbg
