// pair_math.cuh -- per-pair geometry, radial basis and angular moments.
//
// Radial functions H_k(r) = f_c(r) g_k(r) follow descriptor.cpp:51-138 and
// cutoff.cpp:20-37; the rational table follows ration.cu:27-69 (endpoint
// intervals forced to zero, ration.hpp:29).  Monomials are ordered as
// kernel.cu:1197-1232: 1, x, y, z, xx, xy, xz, yy, yz, zz, xxx, xxy, xxz,
// xyy, xyz, xzz, yyy, yyz, yzz, zzz.
#pragma once

#include "rcp.cuh"
#include "tmd_internal.h"

namespace tmd {

// Pair geometry computed by one lane and broadcast to the atom's group.
struct PairGeo {
  float r, rlo;         // distance as an FP32 hi/lo pair (r = hi + lo)
  float ux, uy, uz;     // unit vector (x_j - x_i) / r
  float fc, dfc;        // analytic cutoff and derivative
  float tq;             // table: offset inside the interval
  float rinv;           // 1 / (r + rlo)
  int ti;               // table interval (0 for analytic), -1 when inactive
};

__device__ inline double rsq_plain(double dx, double dy, double dz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                   __dmul_rn(dz, dz));
}

// Position of neighbor entry e, loaded early so the gather latency overlaps
// the previous chunk's arithmetic.
struct NbPos {
  double x, y, z;
  int code;  // shift code, -1 when the slot is empty
};

__device__ inline NbPos load_nb(const double *__restrict__ x, uint32_t e, bool valid) {
  NbPos p;
  if (valid) {
    int j = e & kAtomMask;
    p.x = __ldg(x + 3 * j);
    p.y = __ldg(x + 3 * j + 1);
    p.z = __ldg(x + 3 * j + 2);
    p.code = int(e >> kAtomBits);
  } else {
    p.x = p.y = p.z = 0.0;
    p.code = -1;
  }
  return p;
}

// Geometry of one pair (FP64 difference and cutoff test rij2 < rc^2 &&
// rij2 > 1e-10 as kernel.cu:1163).  g.ti = -1 if inactive.
// 1/r is that of r + rlo.  The shift is decoded for image entries only.
//
// The root, the cutoff's sine and cosine are the plain functions: an FP32
// root with one correction and polynomials of absolute accuracy gave 7 of
// 410 us of the fused descriptor at 128,000 atoms, and cost the relative
// accuracy of f_c and f_c' near rc (forces of rank-3 dimers at 0.98 to 0.998
// rc 2.6e-5 off, against 1.0e-5).
__device__ inline void pair_geometry(const KParams &kp, const BoxP &box, double xi,
                                     double yi, double zi, const NbPos &p,
                                     PairGeo &g) {
  constexpr int kNoShift = kShiftR + 7 * kShiftR + 49 * kShiftR;
  g.ti = -1;
  g.r = g.rlo = g.ux = g.uy = g.uz = g.fc = g.dfc = g.tq = g.rinv = 0.f;
  if (p.code < 0) return;
  double gx = p.x, gy = p.y, gz = p.z;
  if (p.code != kNoShift) {
    int sx, sy, sz;
    shift_decode(p.code, sx, sy, sz);
    image_of(box, p.x, p.y, p.z, sx, sy, sz, gx, gy, gz);
  }
  const double dx = gx - xi, dy = gy - yi, dz = gz - zi;
  const double r2 = rsq_plain(dx, dy, dz);
  if (!(r2 < kp.rcsq && r2 > 1e-10)) return;
  const double r = sqrt(r2);
  const float rf = float(r);
  g.r = rf;
  g.rlo = float(r - double(rf));
  g.rinv = rcp_sum(rf, g.rlo);
  g.ux = float(dx) * g.rinv;
  g.uy = float(dy) * g.rinv;
  g.uz = float(dz) * g.rinv;
  if (kp.radial == 1) {
    int ti = int(r * kp.tab_xdxd);
    if (ti > kp.tab_n - 2) ti = kp.tab_n - 2;
    g.ti = ti;
    g.tq = float(r - ti * kp.tab_dxd);
  } else {
    g.ti = 0;
    float z = rf * kp.inv_rc;
    if (kp.fctype == 0) {
      z = z > 1.f ? 1.f : z;
      float s, c;
      sincospif(z, &s, &c);
      g.fc = 0.5f + 0.5f * c;
      g.dfc = -0.5f * 3.14159265358979f * s * kp.inv_rc;
    } else {
      const float gm = 5.f;
      z = z > 3.14159265358979f ? 3.14159265358979f : z;
      float z4 = z * z * z * z, z5 = z4 * z;
      g.fc = 1.f + gm * z5 * z - (gm + 1.f) * z5;
      g.dfc = (gm + 1.f) * gm * kp.inv_rc * (z5 - z4);
    }
  }
}

// 2^x for x <= 0 by the ex2.approx.ftz instruction (one MUFU operation).  On
// the B200 it returns exp2f's value bit for bit for every FP32 x in
// [-126, 0] (all 1.1e9 inputs compared); below -126, where exp2f returns a
// subnormal, it returns 0.  The Gaussian radial basis takes it in place of
// exp2f's extra range handling.
__device__ __forceinline__ float exp2_nonpos(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Radial kinds the kernels are specialised on.
constexpr int kRadTable = 0;    // rational-interpolation table (FNN or tabulated)
constexpr int kRadGauss = 1;    // analytic Gaussian SF (descriptor::method 3)
constexpr int kRadGeneric = 2;  // analytic power-exponential / Morse / density

inline int radial_kind(const KParams &kp) {
  if (kp.radial == 1) return kRadTable;
  return kp.method == 3 ? kRadGauss : kRadGeneric;
}

// Radial parameters of a lane's 4 filters, loaded once per kernel.  For the
// Gaussian kind gc holds -2 gc and gl holds -gcl (signs and the factor 2
// applied once at load, exactly).
template <int RK>
struct Radial4 {
  float a[RK == kRadGeneric ? 4 : 1], b[RK == kRadTable ? 1 : 4],
      c[RK == kRadGeneric ? 4 : 1], blo[RK == kRadGauss ? 4 : 1],
      gc[RK == kRadGauss ? 4 : 1], gl[RK == kRadGauss ? 4 : 1];
  int k0;
};

template <int RK>
__device__ inline Radial4<RK> load_radial4(const KParams &kp, int k0) {
  Radial4<RK> R;
  R.k0 = k0;
#pragma unroll
  for (int t = 0; t < 4; t++) {
    if (RK == kRadGeneric) {
      R.a[t] = kp.p0[k0 + t];
      R.c[t] = kp.p2[k0 + t];
    }
    if (RK != kRadTable) R.b[t] = kp.p1[k0 + t];
    if (RK == kRadGauss) {
      R.blo[t] = kp.p1lo[k0 + t];
      R.gc[t] = -2.f * kp.gc[k0 + t];
      R.gl[t] = -kp.gcl[k0 + t];
    }
  }
  return R;
}

// Table coefficients (y, s, c1, c2) of filters k0..k0+3 of an interval.
struct TabRow {
  float4 y, s, c1, c2;
};
__device__ inline TabRow load_tab(const KParams &kp, int ti, int k0) {
  const int K = kp.K;
  const float4 *row = reinterpret_cast<const float4 *>(kp.table + (size_t)ti * 4 * K);
  return TabRow{__ldg(row + (k0 >> 2)), __ldg(row + ((K + k0) >> 2)),
                __ldg(row + ((2 * K + k0) >> 2)), __ldg(row + ((3 * K + k0) >> 2))};
}
__device__ inline void tab_eval4(const KParams &kp, const TabRow &T, float q, bool deriv, float H[4],
                                 float dH[4]) {
  const float ys[4] = {T.y.x, T.y.y, T.y.z, T.y.w};
  const float ss[4] = {T.s.x, T.s.y, T.s.z, T.s.w};
  const float c1s[4] = {T.c1.x, T.c1.y, T.c1.z, T.c1.w};
  const float c2s[4] = {T.c2.x, T.c2.y, T.c2.z, T.c2.w};
  const float dx = kp.tab_dx, rr = dx - q;
#pragma unroll
  for (int t = 0; t < 4; t++) {
    float c1 = c1s[t], c2 = c2s[t], s = ss[t];
    float c3 = fabsf(c2 * rr);
    float c4 = c3 + fabsf(c1 * q);
    if (c4 > 0.f) c3 = __fdividef(c3, c4);  // weight in [0, 1]: 2-ulp quotient
    c4 = c2 + c3 * (c1 - c2);
    H[t] = ys[t] + q * (s - rr * c4);
    if (deriv) dH[t] = s + (q - rr) * c4 + dx * (c4 - c2) * (1.f - c3);
  }
}

// H_k and (optionally) dH_k/dr for the lane's filters k0..k0+3.
template <int RK, bool DERIV>
__device__ inline void radial4(const KParams &kp, const Radial4<RK> &R, const PairGeo &g,
                               float H[4], float dH[4]) {
  if (RK == kRadTable) {
    if (g.ti <= 0 || g.ti >= kp.tab_n - 2) {
#pragma unroll
      for (int q = 0; q < 4; q++) { H[q] = 0.f; if (DERIV) dH[q] = 0.f; }
      return;
    }
    tab_eval4(kp, load_tab(kp, g.ti, R.k0), g.tq, DERIV, H, dH);
    return;
  }
  const float r = g.r;
#pragma unroll
  for (int t = 0; t < 4; t++) {
    float f, df;
    if (RK == kRadGauss) {
      // (r - omega) from the hi/lo pairs of both: no systematic rounding of
      // the Gaussian centre
      float d = (r - R.b[t]) + (g.rlo - R.blo[t]);
      f = exp2_nonpos(R.gl[t] * d * d);
      if (DERIV) {
        // dH = dfc f + fc (gc d f) = f (dfc + fc gc d): one FFMA and two FMULs
        H[t] = g.fc * f;
        dH[t] = f * fmaf(g.fc * R.gc[t], d, g.dfc);
        continue;
      }
      df = 0.f;
    } else {
      const float a = R.a[t], b = R.b[t], c = R.c[t];
      if (kp.method == 0) {
        float xr = r / a;
        float pw = powf(xr, b);
        f = expf(-pw);
        df = -f * b * powf(xr, b - 1.f) / a;
      } else if (kp.method == 1) {
        float gdr = b * (r - c);
        float e1 = expf(-gdr), e2 = expf(-2.f * gdr);
        f = a * (e2 - 2.f * e1);
        df = -a * b * 2.f * (e2 - e1);
      } else {
        float z = -b * ((r - c) / c);
        f = a * expf(z);
        df = -f * b / c;
      }
    }
    H[t] = g.fc * f;
    if (DERIV) dH[t] = g.dfc * f + g.fc * df;
  }
}

// Radial parameters of one filter k, loaded once per kernel by the lane that
// owns the filter (the wide-group descriptor form).
template <int RK>
struct Radial1 {
  float a, b, c, blo, gc, gl;
  int k;
};

template <int RK>
__device__ inline Radial1<RK> load_radial1(const KParams &kp, int k) {
  Radial1<RK> R{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, k};
  if (RK == kRadGeneric) { R.a = kp.p0[k]; R.c = kp.p2[k]; }
  if (RK != kRadTable) R.b = kp.p1[k];
  if (RK == kRadGauss) { R.blo = kp.p1lo[k]; R.gc = kp.gc[k]; R.gl = kp.gcl[k]; }
  return R;
}

// H_k of one filter: the expressions of radial4 for a single k.
template <int RK>
__device__ inline float radial1(const KParams &kp, const Radial1<RK> &R, const PairGeo &g) {
  if (RK == kRadTable) {
    if (g.ti <= 0 || g.ti >= kp.tab_n - 2) return 0.f;
    const int K = kp.K;
    const float *row = kp.table + (size_t)g.ti * 4 * K + R.k;
    const float y = __ldg(row), s = __ldg(row + K), c1 = __ldg(row + 2 * K),
                c2 = __ldg(row + 3 * K);
    const float q = g.tq, dx = kp.tab_dx, rr = dx - q;
    float c3 = fabsf(c2 * rr);
    float c4 = c3 + fabsf(c1 * q);
    if (c4 > 0.f) c3 = __fdividef(c3, c4);
    c4 = c2 + c3 * (c1 - c2);
    return y + q * (s - rr * c4);
  }
  float f;
  if (RK == kRadGauss) {
    float d = (g.r - R.b) + (g.rlo - R.blo);
    f = exp2_nonpos(-R.gl * d * d);
  } else {
    const float r = g.r, a = R.a, b = R.b, c = R.c;
    if (kp.method == 0) {
      float xr = r / a;
      float pw = powf(xr, b);
      f = expf(-pw);
    } else if (kp.method == 1) {
      float gdr = b * (r - c);
      float e1 = expf(-gdr), e2 = expf(-2.f * gdr);
      f = a * (e2 - 2.f * e1);
    } else {
      float z = -b * ((r - c) / c);
      f = a * expf(z);
    }
  }
  return g.fc * f;
}

template <int D>
__device__ inline void moments(float x, float y, float z, float M[D]) {
  M[0] = 1.f;
  if (D > 1) { M[1] = x; M[2] = y; M[3] = z; }
  if (D > 4) {
    float xx = x * x, xy = x * y, xz = x * z, yy = y * y, yz = z * y, zz = z * z;
    M[4] = xx; M[5] = xy; M[6] = xz; M[7] = yy; M[8] = yz; M[9] = zz;
    if (D > 10) {
      M[10] = xx * x; M[11] = xx * y; M[12] = xx * z; M[13] = xy * y;
      M[14] = xy * z; M[15] = xz * z; M[16] = yy * y; M[17] = yy * z;
      M[18] = yz * z; M[19] = zz * z;
    }
  }
}

// Rank 3: 16 functions in place of 20 monomials.  u is a unit vector, so
// xx + yy + zz = 1 and the 20 monomials span only 16 functions on the sphere:
// four of every five FMAs of the contractions and of the shared-memory reads
// that feed them, and rows of 64 bytes.  The descriptor accumulates P over the
// set {1, x, y, z, zz - c, xy, xz, xx - yy, yz, x (xx - s), x (yy - zz),
// y (yy - s), y (zz - xx), z (zz - s), z (xx - yy), xyz}, orthogonal for c = 1/3
// and s = 3/5: a monomial's sum, put together again from orthogonal parts,
// carries the rounding noise of its direct sum and no more (with xx - zz and the
// like, sums over xyy came out 1.5 times as noisy).  The pair force evaluates Q(u)
// with zz eliminated, over {1, x, y, z, xx, xy, xz, yy, yz, xxx, xxy, xxz,
// xyy, xyz, yyy, yyz}.
// c and s are the nearest numbers of 12 and 9 bits, so that the shares of P_0 and
// P_x in the other sums, (1 - c) / 2 and (1 - s) / 2, are FP32 numbers too: with
// fl(1/3) for both, xx and yy came out 4.5e-8 too large for every atom, twice
// that in rank 2 of G: total energies of W crystals off by 8e-9 and 1.8e-8 of
// themselves, virials by up to 2.1e-6 (1e-9, 3e-9 and 3.2e-7 with these).
template <int D>
constexpr int kBasis = basis_count(D);

constexpr float kC2 = 1365.f / 4096.f, kC2Rest = (1.f - kC2) / 2.f;
constexpr float kC3 = 307.f / 512.f, kC3Rest = (1.f - kC3) / 2.f;

template <int D>
__device__ inline void basis_p(float x, float y, float z, float M[kBasis<D>]) {
  if constexpr (D < 20) {
    moments<D>(x, y, z, M);
  } else {
    // explicit products: every kernel form rounds them alike, whatever else
    // the compiler would contract
    const float xx = __fmul_rn(x, x), yy = __fmul_rn(y, y), zz = __fmul_rn(z, z),
                xy = __fmul_rn(x, y);
    M[0] = 1.f; M[1] = x; M[2] = y; M[3] = z;
    M[4] = fmaf(z, z, -kC2); M[5] = xy; M[6] = __fmul_rn(x, z);
    M[7] = __fmul_rn(x - y, x + y); M[8] = __fmul_rn(y, z);
    M[9] = __fmul_rn(x, xx - kC3); M[10] = __fmul_rn(x, yy - zz);
    M[11] = __fmul_rn(y, yy - kC3); M[12] = __fmul_rn(y, zz - xx);
    M[13] = __fmul_rn(z, zz - kC3); M[14] = __fmul_rn(z, xx - yy);
    M[15] = __fmul_rn(xy, z);
  }
}

// The sums over monomials that the 16 sums stand for.
struct Rank3 {
  float xx, yy, zz, xxx, xyy, xzz, xxy, yyy, yzz, xxz, yyz, zzz;
};
__device__ inline Rank3 basis_expand(const float A[16]) {
  Rank3 r;
  r.zz = fmaf(kC2, A[0], A[4]);
  r.xx = fmaf(kC2Rest, A[0], 0.5f * (A[7] - A[4]));
  r.yy = fmaf(kC2Rest, A[0], -0.5f * (A[7] + A[4]));
  r.xxx = fmaf(kC3, A[1], A[9]);
  r.xyy = fmaf(kC3Rest, A[1], 0.5f * (A[10] - A[9]));
  r.xzz = fmaf(kC3Rest, A[1], -0.5f * (A[10] + A[9]));
  r.yyy = fmaf(kC3, A[2], A[11]);
  r.yzz = fmaf(kC3Rest, A[2], 0.5f * (A[12] - A[11]));
  r.xxy = fmaf(kC3Rest, A[2], -0.5f * (A[12] + A[11]));
  r.zzz = fmaf(kC3, A[3], A[13]);
  r.xxz = fmaf(kC3Rest, A[3], 0.5f * (A[14] - A[13]));
  r.yyz = fmaf(kC3Rest, A[3], -0.5f * (A[14] + A[13]));
  return r;
}

// G row of one (atom, block, filter): G_m = sum_d T[m][d] P_d^2, G_0 with the
// sign of P_0 under a square root (kernel_1_fused_device, kernel.cu:1028-1061).
// T depends on a monomial only through its exponents' partition (1; x; xx, xy;
// xxx, xxy, xyz), so rank 3 sums the squares of each class first.
template <int D, int M>
__device__ inline void invariants(const float A[kBasis<D>], const float *T, float G[M]) {
  if constexpr (D < 20) {
#pragma unroll
    for (int m = 0; m < M; m++) {
      float s = 0.f;
#pragma unroll
      for (int d = 0; d < D; d++) s = fmaf(T[m * D + d], A[d] * A[d], s);
      G[m] = s;
    }
  } else {
    const Rank3 p = basis_expand(A);
    const float c0 = A[0] * A[0];
    const float c1 = fmaf(A[3], A[3], fmaf(A[2], A[2], A[1] * A[1]));
    const float c4 = fmaf(p.zz, p.zz, fmaf(p.yy, p.yy, p.xx * p.xx));
    const float c5 = fmaf(A[8], A[8], fmaf(A[6], A[6], A[5] * A[5]));
    const float c10 = fmaf(p.zzz, p.zzz, fmaf(p.yyy, p.yyy, p.xxx * p.xxx));
    const float c11 = fmaf(p.xzz, p.xzz, fmaf(p.yzz, p.yzz, fmaf(p.xyy, p.xyy, fmaf(p.xxy, p.xxy,
                      fmaf(p.xxz, p.xxz, p.yyz * p.yyz)))));
    const float c14 = A[15] * A[15];
#pragma unroll
    for (int m = 0; m < M; m++) {
      const float *t = T + m * D;
      G[m] = fmaf(t[0], c0, fmaf(t[1], c1, fmaf(t[4], c4, fmaf(t[5], c5, fmaf(t[10], c10,
             fmaf(t[11], c11, t[14] * c14))))));
    }
  }
  G[0] = copysignf(1.f, A[0]) * sqrtf(G[0]);
}

// Coefficients of Q(u) for one filter: S_d = dE/dP_d = 2 P_d sum_m T[m][d]
// gp_m (kernel2_GPU, kernel.cu:730-848), for rank 3 folded to the 16
// functions that the force evaluates (zz = 1 - xx - yy).
template <int D>
__device__ inline void dedp_row(const float gp[4], const float *T, int M,
                                const float A[kBasis<D>], float F[kBasis<D>]) {
  auto t2 = [&](int d) {
    float t = 0.f;
#pragma unroll
    for (int m = 0; m < 4; m++)
      if (m < M) t = fmaf(gp[m], T[m * D + d], t);
    return 2.f * t;
  };
  if constexpr (D < 20) {
#pragma unroll
    for (int d = 0; d < D; d++) F[d] = t2(d) * A[d];
  } else {
    const Rank3 p = basis_expand(A);
    const float t0 = t2(0), t1 = t2(1), t4 = t2(4), t5 = t2(5), t10 = t2(10), t11 = t2(11),
                t14 = t2(14);
    F[0] = fmaf(t4, p.zz, t0 * A[0]);
    F[1] = fmaf(t11, p.xzz, t1 * A[1]);
    F[2] = fmaf(t11, p.yzz, t1 * A[2]);
    F[3] = fmaf(t10, p.zzz, t1 * A[3]);
    F[4] = t4 * fmaf(kC2Rest - kC2, A[0], fmaf(-1.5f, A[4], 0.5f * A[7]));  // xx - zz
    F[5] = t5 * A[5];
    F[6] = t5 * A[6];
    F[7] = t4 * fmaf(kC2Rest - kC2, A[0], fmaf(-1.5f, A[4], -0.5f * A[7]));  // yy - zz
    F[8] = t5 * A[8];
    F[9] = fmaf(t10, p.xxx, -t11 * p.xzz);
    F[10] = -t11 * A[12];
    F[11] = fmaf(t11, p.xxz, -t10 * p.zzz);
    F[12] = t11 * A[10];
    F[13] = t14 * A[15];
    F[14] = fmaf(t10, p.yyy, -t11 * p.yzz);
    F[15] = fmaf(t11, p.yyz, -t10 * p.zzz);
  }
}

// The functions of Q(u).
template <int D>
__device__ inline void basis_q(float x, float y, float z, float M[kBasis<D>]) {
  if constexpr (D < 20) {
    moments<D>(x, y, z, M);
  } else {
    const float xx = x * x, xy = x * y, xz = x * z, yy = y * y, yz = y * z;
    M[0] = 1.f; M[1] = x; M[2] = y; M[3] = z;
    M[4] = xx; M[5] = xy; M[6] = xz; M[7] = yy; M[8] = yz;
    M[9] = xx * x; M[10] = xx * y; M[11] = xx * z; M[12] = yy * x; M[13] = xy * z;
    M[14] = yy * y; M[15] = yy * z;
  }
}

// Gradient of Q(u) = sum_d V_d M_d(u) with respect to u, and u . grad Q.  Then
// dQ/dx_j = (gradQ - u (u . gradQ)) / r, which is sum_d V_d dM_d/dx_j
// (tensor_ops.cpp calculate_dM_{p,d,f}): only the tangential part counts, so
// Q may be any polynomial with the right values on the sphere.
template <int D>
__device__ inline void poly_grad(const float V[kBasis<D>], float x, float y, float z,
                                 float gq[3], float &nvm) {
  // Horner form: grad_a Q = V_a + x P_a + y Q_a + z R_a, with P, Q, R the
  // coefficients of x, y, z once the linear terms are taken out (three short
  // independent chains instead of one long sum per component)
  float gx = 0.f, gy = 0.f, gz = 0.f;
  if constexpr (D == 4) {
    gx = V[1]; gy = V[2]; gz = V[3];
  } else if constexpr (D == 10) {
    // xx, xy, xz, yy, yz, zz
    gx = fmaf(x, 2.f * V[4], fmaf(y, V[5], fmaf(z, V[6], V[1])));
    gy = fmaf(x, V[5], fmaf(y, 2.f * V[7], fmaf(z, V[8], V[2])));
    gz = fmaf(x, V[6], fmaf(y, V[8], fmaf(z, 2.f * V[9], V[3])));
  } else if constexpr (D == 20) {
    const float Px = fmaf(3.f * V[9], x, fmaf(2.f * V[10], y, fmaf(2.f * V[11], z, 2.f * V[4])));
    const float Qx = fmaf(V[12], y, fmaf(V[13], z, V[5]));
    const float Py = fmaf(V[10], x, fmaf(2.f * V[12], y, fmaf(V[13], z, V[5])));
    const float Qy = fmaf(3.f * V[14], y, fmaf(2.f * V[15], z, 2.f * V[7]));
    const float Pz = fmaf(V[11], x, fmaf(V[13], y, V[6]));
    const float Qz = fmaf(V[15], y, V[8]);
    gx = fmaf(x, Px, fmaf(y, Qx, fmaf(z, V[6], V[1])));
    gy = fmaf(x, Py, fmaf(y, Qy, fmaf(z, V[8], V[2])));
    gz = fmaf(x, Pz, fmaf(y, Qz, V[3]));
  }
  gq[0] = gx; gq[1] = gy; gq[2] = gz;
  nvm = fmaf(x, gx, fmaf(y, gy, z * gz));
}

}  // namespace tmd
