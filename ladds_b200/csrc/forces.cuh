// forces.cuh -- device acceleration set, FP64 and split precision.
//
// FP64:  every term in binary64 (third body in the direct difference form).
// SPLIT: central term, J2, the altitude used for the drag band and the shadow
//        edge in binary64; J3, C22/S22, Sun, Moon (Battin's f(q) form, free of
//        the cancellation of the direct form), SRP and drag in binary32, added
//        to the binary64 sum.  The Yoshida drift/kick accumulation stays
//        binary64.
//
// Both propagation kernels are bound by the instructions of these terms (FP64:
// the FP64 pipe; split: issue), so the terms share what they have in common:
//   - FP64: every gravity term of the Earth is  sr r + i5 (u, w, t), one radial
//     coefficient for central, J2, J3 and C22/S22 together and an extra of
//     three products; C22/S22 stay in inertial axes (ephemeris entry); in the
//     split form central + J2 are put together the same way;
//   - SRP acts along the Sun's direction: it takes the third-body term's
//     difference vector and reciprocal distance (FP64: it is a change of that
//     term's coefficient);
//   - FP64: the indirect third-body accelerations of both bodies are one
//     vector of the ephemeris entry;
//   - quotients are products with table reciprocals, square roots x rsqrt(x).
// Measured (1e6 objects, full set, 128 steps in a launch, per step; before: the
// terms one by one): FP64 47.7 -> 33.4 us by the sharing, 30.0 with the density
// table, 27.4 with the mask known at compile time; split 33.8 -> 30.2 -> 26.9 us
// (10,000 objects: 3.2 -> 2.2 and 2.4 -> 1.7 us).  Then rsqrtOf: 25.8 and 25.7 us
// (10,000 objects: 1.8 and 1.5 us).  The split form's binary32 terms
// keep their order of operations: evaluated with fewer operations they move an
// object by 1e-8 km in 128 steps; two objects at a time in paired binary32
// instructions were no gain (28.7 against 30.2 us before the mask was known).
#pragma once
#include <cfloat>

#include "physics.cuh"

namespace ladds {

constexpr double kJ2Coef = -1.5 * kJ2 * kMuEarth * kREarth * kREarth;
constexpr double kJ3Coef = -2.5 * kJ3 * kMuEarth * kREarth * kREarth * kREarth;
constexpr double kSrpCoef = kCR * kPSrp * kAU * kAU * 1.0e3;
constexpr uint32_t kPropTesseral = kPropC22 | kPropS22;

// Atmosphere tables.  Every band edge of the model is a multiple of 5 km.
//   FP64: per kilometre of altitude in [0, 8192) km the density at its middle
//     and 1 / H (one table per context, built by k_atm_table and read through the
//     L1 cache, which it fits): the exponential's argument is then within
//     1 / (2 H) <= 0.093 of zero and needs no range reduction.  1e6 objects, full
//     set, per step: 33.4 -> 30.0 us against a band search and exp((h0 - h) / H).
//   split: per 5 km (h0, 1 / H, rho0) of the band; 1000 km and above: the last.
//     In shared memory: a 16-byte read on the force evaluation's chain.
constexpr int kAtmFine = 8192, kAtmBand5 = 201;
struct AtmShared {
  float4 row5[kAtmBand5];
};
__constant__ AtmRow c_atm[kAtmBands] = LADDS_ATM_TABLE;

__device__ __forceinline__ int atmBandOf(double h) {  // largest k with h0[k] <= h (0 below the table, and for NaN)
  int k = 0;
  while (k + 1 < kAtmBands && c_atm[k + 1].h0 <= h) ++k;
  return k;
}
__global__ void k_atm_table(double2 *__restrict__ fine) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kAtmFine) return;
  const AtmRow r = c_atm[atmBandOf((double)i)];
  fine[i] = make_double2(r.rho0 * exp(-((double)i + 0.5 - r.h0) / r.H), 1.0 / r.H);
}
// stages the split form's table in shared memory (every thread of the block calls it)
__device__ __forceinline__ void loadAtmTable(AtmShared &atm) {
  for (int i = threadIdx.x; i < kAtmBand5; i += blockDim.x) {
    const AtmRow r = c_atm[atmBandOf(5.0 * i)];
    atm.row5[i] = make_float4((float)r.h0, 1.0f / (float)r.H, (float)r.rho0, 0.0f);
  }
}

// Altitudes outside the fine table, out of line: inlined, the exponential slows the
// path within the table (1e6 objects, default set, 128 iterations 19.66 ms, 19.61 so).
// Above it the last band's exponential has no search and no division: 200,000
// objects at 9000 km, full set, per step 6.8 us (10.1 by the search below; within
// the table 6.2), 4096 adjoint pairs there 1583 us a forward sweep of 1080 steps (3452;
// 1538).
constexpr AtmRow lastAtmRow() {
  const AtmRow t[kAtmBands] = LADDS_ATM_TABLE;
  return t[kAtmBands - 1];
}
constexpr AtmRow kAtmTop = lastAtmRow();
static_assert(kAtmTop.h0 <= kAtmFine, "above the fine table lies the last band only");
__device__ __forceinline__ double2 atmAbove(double h) {
  return make_double2(kAtmTop.rho0 * exp((kAtmTop.h0 - h) * (1.0 / kAtmTop.H)), 1.0 / kAtmTop.H);
}
// altitudes below it, and NaN
__device__ __forceinline__ double2 atmBelow(double h) {
  const AtmRow r = c_atm[atmBandOf(h)];
  return make_double2(r.rho0 * exp(-(h - r.h0) / r.H), 1.0 / r.H);
}

__device__ __noinline__ double2 atmOutside(double h) { return h >= (double)kAtmFine ? atmAbove(h) : atmBelow(h); }

// density [kg/m^3] and 1 / H [1/km] at altitude h.  The kilometre is floor(h):
// the low word of h + 3 * 2^51 rounded down, so a band begins exactly at its
// edge.  exp of |x| <= 0.093 by its Taylor polynomial of degree 9 (remainder
// x^10 / 10! < 1.4e-17), even and odd parts side by side.
__device__ __forceinline__ double2 atmDensity(const double2 *__restrict__ fine, double h) {
  if ((uint32_t)__double2hiint(h) >= 0x40c00000u) return atmOutside(h);  // >= 8192 km, negative, NaN
  const double m = __dadd_rd(h, 6755399441055744.0);
  const double2 t = __ldg(&fine[__double2loint(m)]);
  const double x = ((m - 6755399441055744.0) + 0.5 - h) * t.y, x2 = x * x;
  const double even = 1.0 + x2 * (1.0 / 2 + x2 * (1.0 / 24 + x2 * (1.0 / 720 + x2 * (1.0 / 40320))));
  const double odd = 1.0 + x2 * (1.0 / 6 + x2 * (1.0 / 120 + x2 * (1.0 / 5040 + x2 * (1.0 / 362880))));
  return make_double2(t.x * (even + x * odd), t.y);
}

// 1 / sqrt(x) of a normal x > 0: the hardware's approximation y (its low word
// is zero, so y y is exact; relative error below 2^-20) and three terms of the
// binomial series of (1 - e)^(-1/2), e = 1 - x y^2.  What the series leaves out
// is below 2^-77; measured within 0.5000 ulp (the library's function: 0.508).
// Without that function's branch for special arguments the reciprocal roots of a
// force evaluation run side by side: three of them, one warp, 212 -> 91 cycles; 16
// warps on one SM 280 -> 201 (one alone 79 -> 68).
// NaN at 0 and infinity, where an acceleration is NaN either way.
__device__ __forceinline__ double rsqrtOf(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(fma(fma(5.0 / 16, e, 3.0 / 8), e, 0.5), e * y, y);
}

// sqrt(x) of a normal x; x itself below, and for NaN
__device__ __forceinline__ double sqrtOf(double x) { return x >= DBL_MIN ? x * rsqrtOf(x) : x; }

// the Earth's gravity terms of the mask: acceleration sr r + (ax, ay, az),
// added to sr and a; r2 = |r|^2, rinv = 1 / |r|
__device__ __forceinline__ void earthGravity(uint32_t mask, double x, double y, double z, double rinv,
                                             const EphEntry &e, double &sr, double a[3]) {
  const double i2 = rinv * rinv, i3 = i2 * rinv;
  if (mask & kPropKEP) sr += -kMuEarth * i3;
  if (mask & (kPropJ2 | kPropJ3 | kPropTesseral)) {
    const double i5 = i3 * i2, q = z * z * i2;
    const double c2 = (mask & kPropJ2) ? kJ2Coef : 0.0;
    double t = 2.0 * c2 * z, b = c2 * (1.0 - 5.0 * q);
    if (mask & (kPropJ3 | kPropTesseral)) {
      const double c3 = (mask & kPropJ3) ? kJ3Coef : 0.0;
      const double p = (mask & kPropTesseral) ? e.p : 0.0, s = (mask & kPropTesseral) ? e.q : 0.0;
      const double u = p * x + s * y, w = s * x - p * y, g = x * u + y * w;
      b += i2 * (c3 * z * (3.0 - 7.0 * q) - 2.5 * g);
      t += c3 * (3.0 * q - 0.6);
      a[0] += i5 * u;
      a[1] += i5 * w;
    }
    sr += i5 * b;
    a[2] += i5 * t;
  }
}

// the object lies in the Earth's (cylindrical) shadow
__device__ __forceinline__ bool inShadow(double x, double y, double z, double r2, const double sunHat[3]) {
  const double proj = x * sunHat[0] + y * sunHat[1] + z * sunHat[2];
  return proj < 0.0 && (r2 - proj * proj) < kREarth * kREarth;
}

// FP64 acceleration of the terms of the mask
__device__ __forceinline__ void accel(uint32_t mask, const double r[3], const double v[3], double aom, double bcInv,
                                      const EphEntry &e, const double2 *fine, double a[3]) {
  const double x = r[0], y = r[1], z = r[2];
  const double r2 = x * x + y * y + z * z;
  const double rinv = rsqrtOf(r2);
  double c[3] = {0.0, 0.0, 0.0}, sr = 0.0;
  if (mask & (kPropSOL | kPropLUN)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = -e.indirect[k];
  }
  if (mask & (kPropSOL | kPropSRP)) {
    const double dx = e.sun[0] - x, dy = e.sun[1] - y, dz = e.sun[2] - z;
    const double di = rsqrtOf(dx * dx + dy * dy + dz * dz);
    double k = (mask & kPropSOL) ? kMuSun : 0.0;
    if ((mask & kPropSRP) && !inShadow(x, y, z, r2, e.sunHat)) k -= kSrpCoef * aom;
    k *= di * di * di;
    c[0] += k * dx;
    c[1] += k * dy;
    c[2] += k * dz;
  }
  if (mask & kPropLUN) {
    const double dx = e.moon[0] - x, dy = e.moon[1] - y, dz = e.moon[2] - z;
    const double di = rsqrtOf(dx * dx + dy * dy + dz * dz);
    const double k = kMuMoon * di * di * di;
    c[0] += k * dx;
    c[1] += k * dy;
    c[2] += k * dz;
  }
  if (mask & kPropDRAG) {
    const double wx = v[0] + kOmegaEarth * y, wy = v[1] - kOmegaEarth * x, wz = v[2];
    const double wn = sqrtOf(wx * wx + wy * wy + wz * wz);
    const double k = -0.5e3 * atmDensity(fine, r2 * rinv - kREarth).x * bcInv * wn;
    c[0] += k * wx;
    c[1] += k * wy;
    c[2] += k * wz;
  }
  if (mask & (kPropKEP | kPropJ2 | kPropJ3 | kPropTesseral)) {
    earthGravity(mask, x, y, z, rinv, e, sr, c);
    c[0] += sr * x;
    c[1] += sr * y;
    c[2] += sr * z;
  }
  a[0] = c[0];
  a[1] = c[1];
  a[2] = c[2];
}

// The binary32 terms of the split form are written with explicitly rounded
// operations (a product fused into a sum only where it says so): their rounding,
// not the binary64 part's, decides where an object is after some hundred steps,
// and it does not depend on which terms a kernel has side by side.
__device__ __forceinline__ float mulf(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float addf(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float subf(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmaf_(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Battin's f(q) = (1+q)^{3/2} - 1 written without cancellation.  The
// binary32 terms use the approximate square root (s * rsqrtOf(s)) and division
// of the hardware: their few-ulp errors are far below the split form's
// binary32 rounding of the perturbations themselves.
__device__ __forceinline__ float battinF(float q) {
  const float s = addf(1.0f, q);
  const float num = mulf(q, fmaf_(q, addf(3.0f, q), 3.0f));
  return __fdividef(num, fmaf_(s, mulf(s, rsqrtf(s)), 1.0f));
}

// third body at p: adds -mu / |d|^3 (r + f(q) p) to b, with d = p - r and
// q = r.(r - 2 p) / |p|^2; di = 1 / |d|
__device__ __forceinline__ void thirdBody(const float r[3], const float *p, float invP2, float mu, float di,
                                          float b[3]) {
  const float q = mulf(fmaf_(r[2], fmaf_(-2.0f, p[2], r[2]),
                             fmaf_(r[0], fmaf_(-2.0f, p[0], r[0]), mulf(r[1], fmaf_(-2.0f, p[1], r[1])))),
                       invP2);
  const float k = mulf(mulf(mulf(-mu, di), di), di);
  const float f = battinF(q);
#pragma unroll
  for (int i = 0; i < 3; ++i) b[i] = fmaf_(k, fmaf_(f, p[i], r[i]), b[i]);
}

// Split-precision acceleration of the terms of the mask.
__device__ __forceinline__ void accel(uint32_t mask, const double r[3], const double v[3], float aom, float bcInv,
                                      const EphEntryF &e, const AtmShared &atm, double a[3]) {
  const double x = r[0], y = r[1], z = r[2];
  const double r2 = x * x + y * y + z * z;
  const double rinv = rsqrtOf(r2);
  const double rinv2 = rinv * rinv;
  const float rf[3] = {(float)x, (float)y, (float)z};
  float b[3] = {0.f, 0.f, 0.f};
  if (mask & (kPropJ3 | kPropTesseral)) {
    const float rinvf = (float)rinv, rinv2f = (float)rinv2;
    if (mask & kPropJ3) {
      const float k = mulf((float)kJ3Coef, mulf(mulf(mulf(rinv2f, rinv2f), rinv2f), rinvf));
      const float z2 = mulf(rf[2], rf[2]);
      const float f = fmaf_(3.0f, rf[2], -mulf(mulf(mulf(7.0f, z2), rf[2]), rinv2f));
      b[0] = mulf(mulf(k, rf[0]), f);
      b[1] = mulf(mulf(k, rf[1]), f);
      // 6 z^2 - 7 z^4 / r^2 - 0.6 r^2 == z^2 (6 - 7 z^2/r^2) - 0.6 r^2
      b[2] = mulf(k, fmaf_(z2, fmaf_(-7.0f, mulf(z2, rinv2f), 6.0f), -mulf(0.6f, (float)r2)));
    }
    if (mask & kPropTesseral) {
      const float C = (mask & kPropC22) ? (float)kC22 : 0.0f;
      const float S = (mask & kPropS22) ? (float)kS22 : 0.0f;
      const float c = e.cosT, s = e.sinT;
      const float xe = fmaf_(c, rf[0], mulf(s, rf[1])), ye = fmaf_(c, rf[1], -mulf(s, rf[0]));
      const float g = fmaf_(mulf(2.0f * S, xe), ye, mulf(C, fmaf_(xe, xe, -mulf(ye, ye))));
      const float k = mulf((float)(3.0 * kMuEarth * kREarth * kREarth), mulf(mulf(rinv2f, rinv2f), rinvf));
      const float g5 = mulf(5.0f, g);
      const float axe = mulf(k, fmaf_(-mulf(g5, xe), rinv2f, mulf(2.0f, fmaf_(C, xe, mulf(S, ye)))));
      const float aye = mulf(k, fmaf_(-mulf(g5, ye), rinv2f, mulf(2.0f, fmaf_(S, xe, -mulf(C, ye)))));
      b[0] = addf(b[0], fmaf_(c, axe, -mulf(s, aye)));
      b[1] = addf(b[1], fmaf_(s, axe, mulf(c, aye)));
      b[2] = fmaf_(k, -mulf(mulf(g5, rf[2]), rinv2f), b[2]);
    }
  }
  float srp = 0.f, d[3] = {0.f, 0.f, 0.f};  // radiation pressure: -srp d, d towards the Sun
  if (mask & (kPropSOL | kPropSRP)) {
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = subf(e.sun[i], rf[i]);
    const float di = rsqrtf(fmaf_(d[2], d[2], fmaf_(d[0], d[0], mulf(d[1], d[1]))));
    if (mask & kPropSOL) thirdBody(rf, e.sun, e.sunInvS2, (float)kMuSun, di, b);
    // the shadow edge in binary64: it switches the whole SRP term, and a
    // binary32 edge (~0.4 m) flips stage evaluations near it, which moved
    // single objects by up to 0.3 m per day against the FP64 path
    if ((mask & kPropSRP) && !inShadow(x, y, z, r2, e.sunHat)) {
      // (AU * di)^2 * di keeps every factor inside binary32 range
      const float au = mulf((float)kAU, di);
      srp = mulf(mulf((float)(kCR * kPSrp * 1.0e3), aom), mulf(mulf(au, au), di));
    }
  }
  if (mask & kPropLUN) {
    const float m[3] = {subf(e.moon[0], rf[0]), subf(e.moon[1], rf[1]), subf(e.moon[2], rf[2])};
    const float di = rsqrtf(fmaf_(m[2], m[2], fmaf_(m[0], m[0], mulf(m[1], m[1]))));
    thirdBody(rf, e.moon, e.moonInvS2, (float)kMuMoon, di, b);
  }
  if (mask & kPropSRP) {
#pragma unroll
    for (int i = 0; i < 3; ++i) b[i] = fmaf_(-srp, d[i], b[i]);
  }
  if (mask & kPropDRAG) {
    const float w[3] = {fmaf_((float)kOmegaEarth, rf[1], (float)v[0]), fmaf_(-(float)kOmegaEarth, rf[0], (float)v[1]),
                        (float)v[2]};
    const float w2 = fmaf_(w[2], w[2], fmaf_(w[0], w[0], mulf(w[1], w[1])));
    const float wn = w2 > 0.0f ? mulf(w2, rsqrtf(w2)) : 0.0f;
    // an altitude within binary32 rounding of a band edge may take the
    // neighbouring band, whose density agrees there to the table's continuity
    const float h = (float)(r2 * rinv - kREarth);
    const float4 row = atm.row5[min(max((int)mulf(h, 0.2f), 0), kAtmBand5 - 1)];
    const float rho = mulf(row.z, __expf(mulf(-subf(h, row.x), row.y)));
    const float k = mulf(mulf(mulf(-0.5e3f, rho), bcInv), wn);
#pragma unroll
    for (int i = 0; i < 3; ++i) b[i] = fmaf_(k, w[i], b[i]);
  }
  double sr = 0.0, az = 0.0;
  if (mask & (kPropKEP | kPropJ2)) {
    const double i3 = rinv2 * rinv;
    if (mask & kPropKEP) sr = -kMuEarth * i3;
    if (mask & kPropJ2) {
      const double k = kJ2Coef * (i3 * rinv2);
      sr += k * (1.0 - 5.0 * (z * z * rinv2));
      az = 2.0 * k;
    }
  }
  a[0] = sr * x + (double)b[0];
  a[1] = sr * y + (double)b[1];
  a[2] = (sr + az) * z + (double)b[2];
}

}  // namespace ladds
