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
// Measured (1e6 objects, 128 steps in a launch, per step; before: the terms one
// by one): full set FP64 47.7 -> 33.5 us, split 33.8 -> 30.2 us; the default
// set (without the third bodies) 35.0 -> 29.5 and 22.6 -> 20.6 us.  The split
// form's binary32 terms keep their order of operations: evaluated with fewer
// operations (23.5 us) they move an object by 1e-8 km in 128 steps.
#pragma once
#include "physics.cuh"

namespace ladds {

constexpr double kJ2Coef = -1.5 * kJ2 * kMuEarth * kREarth * kREarth;
constexpr double kJ3Coef = -2.5 * kJ3 * kMuEarth * kREarth * kREarth * kREarth;
constexpr double kSrpCoef = kCR * kPSrp * kAU * kAU * 1.0e3;
constexpr uint32_t kPropTesseral = kPropC22 | kPropS22;

// The band is found without a search: every band edge of the table is a
// multiple of 5 km, so the band of h in [0, 1000) km is a function of
// floor(h / 5) (a 200-entry table; 1000 km and above: the last band).
constexpr int kAtmBand5 = 201;
template <bool SPLIT>
struct AtmShared;
template <>
struct AtmShared<false> {
  double h0[kAtmBands], rho0[kAtmBands], invH[kAtmBands];
  uint8_t band5[kAtmBand5 + 3];  // band of the altitudes [5 i, 5 i + 5) km
};
// split precision: the band's constants themselves per 5 km,
// (h0, 1 / H, rho0): one 16-byte read per evaluation
template <>
struct AtmShared<true> {
  float4 row5[kAtmBand5];
};

__device__ __forceinline__ int atmBandOf5(const AtmRow *rows, int i) {  // largest k with h0[k] <= 5 i
  int k = 0;
  while (k + 1 < kAtmBands && rows[k + 1].h0 <= 5.0 * i) ++k;
  return k;
}

// stages the atmosphere table in shared memory (every thread of the block calls it)
__device__ __forceinline__ void loadAtmTable(AtmShared<false> &atm, const AtmRow *rows) {
  for (int i = threadIdx.x; i < kAtmBands; i += blockDim.x) {
    atm.h0[i] = rows[i].h0;
    atm.rho0[i] = rows[i].rho0;
    atm.invH[i] = 1.0 / rows[i].H;
  }
  for (int i = threadIdx.x; i < kAtmBand5; i += blockDim.x) atm.band5[i] = (uint8_t)atmBandOf5(rows, i);
}
__device__ __forceinline__ void loadAtmTable(AtmShared<true> &atm, const AtmRow *rows) {
  for (int i = threadIdx.x; i < kAtmBand5; i += blockDim.x) {
    const AtmRow r = rows[atmBandOf5(rows, i)];
    atm.row5[i] = make_float4((float)r.h0, 1.0f / (float)r.H, (float)r.rho0, 0.0f);
  }
}

// band index: largest k with h0[k] <= h (0 below the table).  The 5 km table
// gives it up to the rounding of h / 5 at a band edge (every band is at least
// 5 km wide), which one comparison with each neighbouring edge corrects: the
// result equals a search of h0 for every h (NaN: band 0).
__device__ __forceinline__ int atmBand(const AtmShared<false> &t, double h) {
  int k = t.band5[min(max((int)(h * 0.2), 0), kAtmBand5 - 1)];
  if (h < t.h0[k])
    k = max(k - 1, 0);
  else if (k + 1 < kAtmBands && h >= t.h0[k + 1])
    k = k + 1;
  return k;
}

// x sqrt(1 / x), 0 at 0
__device__ __forceinline__ double sqrtOf(double x) { return x > 0.0 ? x * rsqrt(x) : x; }

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
                                      const EphEntry &e, const AtmShared<false> &atm, double a[3]) {
  const double x = r[0], y = r[1], z = r[2];
  const double r2 = x * x + y * y + z * z;
  const double rinv = rsqrt(r2);
  double c[3] = {0.0, 0.0, 0.0}, sr = 0.0;
  if (mask & (kPropSOL | kPropLUN)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = -e.indirect[k];
  }
  if (mask & (kPropSOL | kPropSRP)) {
    const double dx = e.sun[0] - x, dy = e.sun[1] - y, dz = e.sun[2] - z;
    const double di = rsqrt(dx * dx + dy * dy + dz * dz);
    double k = (mask & kPropSOL) ? kMuSun : 0.0;
    if ((mask & kPropSRP) && !inShadow(x, y, z, r2, e.sunHat)) k -= kSrpCoef * aom;
    k *= di * di * di;
    c[0] += k * dx;
    c[1] += k * dy;
    c[2] += k * dz;
  }
  if (mask & kPropLUN) {
    const double dx = e.moon[0] - x, dy = e.moon[1] - y, dz = e.moon[2] - z;
    const double di = rsqrt(dx * dx + dy * dy + dz * dz);
    const double k = kMuMoon * di * di * di;
    c[0] += k * dx;
    c[1] += k * dy;
    c[2] += k * dz;
  }
  if (mask & kPropDRAG) {
    const double wx = v[0] + kOmegaEarth * y, wy = v[1] - kOmegaEarth * x, wz = v[2];
    const double wn = sqrtOf(wx * wx + wy * wy + wz * wz);
    const double h = r2 * rinv - kREarth;
    const int b = atmBand(atm, h);
    const double rho = atm.rho0[b] * exp((atm.h0[b] - h) * atm.invH[b]);
    const double k = -0.5e3 * rho * bcInv * wn;
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

// Battin's f(q) = (1+q)^{3/2} - 1 written without cancellation.  The
// binary32 terms use the approximate square root (s * rsqrt(s)) and division
// of the hardware: their few-ulp errors are far below the split form's
// binary32 rounding of the perturbations themselves.
__device__ __forceinline__ float battinF(float q) {
  const float s = 1.0f + q;
  const float s32 = s * (s * rsqrtf(s));
  return __fdividef(q * (3.0f + q * (3.0f + q)), 1.0f + s32);
}

// Split-precision acceleration of the terms of the mask.  The binary32 terms
// keep one order of operations and of summation: their rounding, not the
// binary64 part's, decides where an object is after some hundred steps.
__device__ __forceinline__ void accel(uint32_t mask, const double r[3], const double v[3], float aom, float bcInv,
                                      const EphEntryF &e, const AtmShared<true> &atm, double a[3]) {
  const double x = r[0], y = r[1], z = r[2];
  const double r2 = x * x + y * y + z * z;
  const double rinv = rsqrt(r2);
  const double rinv2 = rinv * rinv;
  const float xf = (float)x, yf = (float)y, zf = (float)z;
  float bx = 0.f, by = 0.f, bz = 0.f;
  if (mask & (kPropJ3 | kPropTesseral)) {
    const float rinvf = (float)rinv, rinv2f = (float)rinv2;
    if (mask & kPropJ3) {
      const float k = (float)kJ3Coef * (rinv2f * rinv2f * rinv2f * rinvf);
      const float z2 = zf * zf;
      const float f = 3.0f * zf - 7.0f * z2 * zf * rinv2f;
      const float z2r2 = z2 * rinv2f;
      bx += k * xf * f;
      by += k * yf * f;
      // 6 z^2 - 7 z^4 / r^2 - 0.6 r^2 == z^2 (6 - 7 z^2/r^2) - 0.6 r^2
      bz += k * (z2 * (6.0f - 7.0f * z2r2) - 0.6f * (float)r2);
    }
    if (mask & kPropTesseral) {
      const float C = (mask & kPropC22) ? (float)kC22 : 0.0f;
      const float S = (mask & kPropS22) ? (float)kS22 : 0.0f;
      const float c = e.cosT, s = e.sinT;
      const float xe = c * xf + s * yf, ye = -s * xf + c * yf;
      const float g = C * (xe * xe - ye * ye) + 2.0f * S * xe * ye;
      const float k = (float)(3.0 * kMuEarth * kREarth * kREarth) * (rinv2f * rinv2f * rinvf);
      const float axe = k * (2.0f * (C * xe + S * ye) - 5.0f * g * xe * rinv2f);
      const float aye = k * (2.0f * (S * xe - C * ye) - 5.0f * g * ye * rinv2f);
      bx += c * axe - s * aye;
      by += s * axe + c * aye;
      bz += k * (-5.0f * g * zf * rinv2f);
    }
  }
  float srp = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;  // radiation pressure: srp (sx, sy, sz) towards the Sun
  if (mask & (kPropSOL | kPropSRP)) {
    const float *sp = e.sun;
    sx = sp[0] - xf, sy = sp[1] - yf, sz = sp[2] - zf;
    const float di = rsqrtf(sx * sx + sy * sy + sz * sz);
    if (mask & kPropSOL) {
      // q = r.(r - 2s) / |s|^2 ;  a = -mu / |d|^3 (r + f(q) s),  d = s - r
      const float q = (xf * (xf - 2.0f * sp[0]) + yf * (yf - 2.0f * sp[1]) + zf * (zf - 2.0f * sp[2])) * e.sunInvS2;
      const float k = -(float)kMuSun * di * di * di;
      const float f = battinF(q);
      bx += k * (xf + f * sp[0]);
      by += k * (yf + f * sp[1]);
      bz += k * (zf + f * sp[2]);
    }
    // the shadow edge in binary64: it switches the whole SRP term, and a
    // binary32 edge (~0.4 m) flips stage evaluations near it, which moved
    // single objects by up to 0.3 m per day against the FP64 path
    if ((mask & kPropSRP) && !inShadow(x, y, z, r2, e.sunHat)) {
      // (AU * di)^2 * di keeps every factor inside binary32 range
      const float au = (float)kAU * di;
      srp = (float)(kCR * kPSrp * 1.0e3) * aom * (au * au * di);
    }
  }
  if (mask & kPropLUN) {
    const float *sp = e.moon;
    const float q = (xf * (xf - 2.0f * sp[0]) + yf * (yf - 2.0f * sp[1]) + zf * (zf - 2.0f * sp[2])) * e.moonInvS2;
    const float dx = sp[0] - xf, dy = sp[1] - yf, dz = sp[2] - zf;
    const float di = rsqrtf(dx * dx + dy * dy + dz * dz);
    const float k = -(float)kMuMoon * di * di * di;
    const float f = battinF(q);
    bx += k * (xf + f * sp[0]);
    by += k * (yf + f * sp[1]);
    bz += k * (zf + f * sp[2]);
  }
  if (mask & kPropSRP) {
    bx -= srp * sx;
    by -= srp * sy;
    bz -= srp * sz;
  }
  if (mask & kPropDRAG) {
    const float wx = (float)v[0] + (float)kOmegaEarth * yf, wy = (float)v[1] - (float)kOmegaEarth * xf,
                wz = (float)v[2];
    const float w2 = wx * wx + wy * wy + wz * wz;
    const float wn = w2 > 0.0f ? w2 * rsqrtf(w2) : 0.0f;
    // an altitude within binary32 rounding of a band edge may take the
    // neighbouring band, whose density agrees there to the table's continuity
    const float h = (float)(r2 * rinv - kREarth);
    const float4 row = atm.row5[min(max((int)(h * 0.2f), 0), kAtmBand5 - 1)];
    const float rho = row.z * __expf(-(h - row.x) * row.y);
    const float k = -0.5e3f * rho * bcInv * wn;
    bx += k * wx;
    by += k * wy;
    bz += k * wz;
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
  a[0] = sr * x + (double)bx;
  a[1] = sr * y + (double)by;
  a[2] = (sr + az) * z + (double)bz;
}

}  // namespace ladds
