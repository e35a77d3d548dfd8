// adjoint.cuh -- FP64 adjoint of the Yoshida-4 step for conjunction pairs.
//
// Loss of a batch of pairs (A_p, B_p):
//   L = sum_p min_{s = 1..S} dl2_p(s),
// dl2_p(s) = squared closest approach of the two straight segments over the
// step ending at s (utils::distanceByLinearInterpolation,
// DistanceApproximation.cpp:13-58, the miss distance of CollisionFunctor.cpp:
// 94-129), evaluated on the states after step s.  Gradients: dL/d(r, v) of
// both initial states and dL/dbcInv of both objects (bcInv = Cd A / m enters
// the drag term).
//
// Forward (k_adj_forward): one lane per object in each of the block's warps
// that share out its force terms, the two objects of a pair in adjacent lanes
// (states exchanged by shuffles after every step).  It stores, per step, the
// start state and the velocities of the second and third kick (12 doubles: the
// records) or, where those would be too large, the state every `ck` steps.
// Backward (k_adj_backward): the records in reverse order; from checkpoints, segment by
// segment, each after a forward sweep of the segment that stores its records:
//   adjoint of a drift  r' = r + c h v:          lv += c h lr
//   adjoint of a kick   v' = v + d h a(r, v):    g = d h lv;
//       lr += (da/dr)^T g,  lv += (da/dv)^T g,  lbc += (da/dbc)^T g.
// Every term but drag is the gradient of a potential (central, zonal J2/J3,
// tesseral C22/S22 in the rotating frame, third body, cannonball SRP), so its
// Jacobian is symmetric.  The SRP
// shadow switch and the atmosphere band are piecewise constant and contribute
// nothing.  Drag, a = K(|r|) |w| w with w = v + Omega r (co-rotating
// atmosphere) and K = -0.5e3 rho(h) bcInv, has its transposed Jacobian
// written out:
//   q = K (|w| g + w (w.g) / |w|);  lv += q;  lr += M^T q - K |w| (w.g) / H r_hat;
//   lbc += -0.5e3 rho |w| (w.g).
// The seed of a pair is the gradient of dl2 at its argmin step s*; with the
// clamped closest-approach time t* (envelope theorem, t* constant at the
// clamps): d dl2 / d r_A = 2 dr*, d dl2 / d v_A = 2 dr* (t* - dt), B negated.
#pragma once
#include "forces.cuh"
#include "propagate.cuh"

namespace ladds {

// Jacobian of the FP64 acceleration at (r, v), as the reverse of a kick applies
// it to g: lr += P g with P = (da/dr)^T, lv += D g with D = (da/dv)^T (symmetric),
// lbc += b . g with b = da/dbcInv.  One item: m[k * 32] for the lane's object,
// k = 0..8 P by rows, 9..14 D as xx, xy, xz, yy, yz, zz, 15..17 b (9 and up
// only where the mask has drag).
//   Earth: a = s r + i5 (u, w, t) (earthGravity); with f, q, b, t as there,
//     grad s = A r + B z^ + G (u, w, 0), G = -5 / |r|^7,
//     A = i2 (-3 s_central + i5 (-5 b + 2 E q - 2 i2 in)),  E = 5 c2 + 7 c3 z i2,
//     B = G t - 6 c3 q / |r|^7, and J = s I + A r r^T + B (r z^T + z r^T)
//     + G (r (u, w, 0)^T + (u, w, 0) r^T) + i5 (p, h; h, -p; 2 c2 + 6 c3 z i2).
//   Sun (with radiation pressure) and Moon: k (3 d d^T / |d|^2 - I).
//   Drag: D = K (|w| I + w w^T / |w|), P = M^T D - K |w| / (H |r|) r w^T.
constexpr int kJacWords = 18;
__device__ __forceinline__ void accelJacobian(uint32_t mask, const double r[3], const double v[3], double aom,
                                              double bcInv, const EphEntry &e, const double2 *atm, double *m) {
  const double x = r[0], y = r[1], z = r[2];
  const double r2 = x * x + y * y + z * z, rinv = rsqrtOf(r2);
  double xx = 0.0, xy = 0.0, xz = 0.0, yy = 0.0, yz = 0.0, zz = 0.0;
  if (mask & (kPropKEP | kPropJ2 | kPropJ3 | kPropTesseral)) {
    const double i2 = rinv * rinv, i3 = i2 * rinv, i5 = i3 * i2, i7 = i5 * i2, q = z * z * i2;
    double s = (mask & kPropKEP) ? -kMuEarth * i3 : 0.0, A = -3.0 * s;
    if (mask & (kPropJ2 | kPropJ3 | kPropTesseral)) {
      const double c2 = (mask & kPropJ2) ? kJ2Coef : 0.0;
      double b = c2 * (1.0 - 5.0 * q), eq = 5.0 * c2 * q, d = 2.0 * c2;  // b, E q, the zz extra
      double B = -10.0 * c2 * z, in = 0.0;                              // B |r|^7
      if (mask & (kPropJ3 | kPropTesseral)) {
        const double c3 = (mask & kPropJ3) ? kJ3Coef : 0.0, zi = c3 * z * i2;
        const double p = (mask & kPropTesseral) ? e.p : 0.0, h = (mask & kPropTesseral) ? e.q : 0.0;
        const double u = p * x + h * y, w = h * x - p * y;
        in = c3 * z * (3.0 - 7.0 * q) - 2.5 * (x * u + y * w);
        b += i2 * in;
        eq += 7.0 * zi * q;
        B += c3 * (3.0 - 21.0 * q);
        d += 6.0 * zi;
        const double G = -5.0 * i7, gu = G * u, gw = G * w, pi = i5 * p;
        xx += 2.0 * gu * x + pi;
        yy += 2.0 * gw * y - pi;
        xy += gw * x + gu * y + i5 * h;
        xz += gu * z;
        yz += gw * z;
      }
      s += i5 * b;
      A += i5 * (2.0 * (eq - i2 * in) - 5.0 * b);
      B *= i7;
      xz += B * x;
      yz += B * y;
      zz += 2.0 * B * z + i5 * d;
    }
    A *= i2;
    const double ax = A * x, ay = A * y, az = A * z;
    xx += s + ax * x;
    yy += s + ay * y;
    zz += s + az * z;
    xy += ax * y;
    xz += ax * z;
    yz += ay * z;
  }
  if (mask & (kPropSOL | kPropSRP)) {
    const double dx = e.sun[0] - x, dy = e.sun[1] - y, dz = e.sun[2] - z;
    const double di = rsqrtOf(dx * dx + dy * dy + dz * dz), di2 = di * di;
    double k = (mask & kPropSOL) ? kMuSun : 0.0;
    if ((mask & kPropSRP) && !inShadow(x, y, z, r2, e.sunHat)) k -= kSrpCoef * aom;
    k *= di2 * di;
    const double k3 = 3.0 * k * di2, tx = k3 * dx, ty = k3 * dy, tz = k3 * dz;
    xx += tx * dx - k;
    yy += ty * dy - k;
    zz += tz * dz - k;
    xy += tx * dy;
    xz += tx * dz;
    yz += ty * dz;
  }
  if (mask & kPropLUN) {
    const double dx = e.moon[0] - x, dy = e.moon[1] - y, dz = e.moon[2] - z;
    const double di = rsqrtOf(dx * dx + dy * dy + dz * dz), di2 = di * di;
    const double k = kMuMoon * (di2 * di);
    const double k3 = 3.0 * k * di2, tx = k3 * dx, ty = k3 * dy, tz = k3 * dz;
    xx += tx * dx - k;
    yy += ty * dy - k;
    zz += tz * dz - k;
    xy += tx * dy;
    xz += tx * dz;
    yz += ty * dz;
  }
  double yx = xy, zx = xz, zy = yz;
  if (mask & kPropDRAG) {
    const double wx = v[0] + kOmegaEarth * y, wy = v[1] - kOmegaEarth * x, wz = v[2];
    const double w2 = wx * wx + wy * wy + wz * wz, winv = w2 >= DBL_MIN ? rsqrtOf(w2) : 0.0, wn = w2 * winv;
    const double2 air = atmDensity(atm, r2 * rinv - kREarth);
    const double c4 = -0.5e3 * air.x * wn, c1 = c4 * bcInv, c2 = -0.5e3 * air.x * bcInv * winv;
    const double ex = c2 * wx, ey = c2 * wy;
    const double dxx = c1 + ex * wx, dxy = ex * wy, dxz = ex * wz, dyy = c1 + ey * wy, dyz = ey * wz;
    m[9 * 32] = dxx;
    m[10 * 32] = dxy;
    m[11 * 32] = dxz;
    m[12 * 32] = dyy;
    m[13 * 32] = dyz;
    m[14 * 32] = c1 + c2 * wz * wz;
    m[15 * 32] = c4 * wx;
    m[16 * 32] = c4 * wy;
    m[17 * 32] = c4 * wz;
    // w = (vx + W y, vy - W x, vz): M^T q = (-W qy, W qx, 0); K depends on |r| through rho(h)
    const double kr = -c1 * (air.y * rinv), kx = kr * wx, ky = kr * wy, kz = kr * wz;
    xx += kx * x - kOmegaEarth * dxy;
    xy += ky * x - kOmegaEarth * dyy;
    xz += kz * x - kOmegaEarth * dyz;
    yx += kx * y + kOmegaEarth * dxx;
    yy += ky * y + kOmegaEarth * dxy;
    yz += kz * y + kOmegaEarth * dxz;
    zx += kx * z;
    zy += ky * z;
    zz += kz * z;
  }
  m[0] = xx;
  m[1 * 32] = xy;
  m[2 * 32] = xz;
  m[3 * 32] = yx;
  m[4 * 32] = yy;
  m[5 * 32] = yz;
  m[6 * 32] = zx;
  m[7 * 32] = zy;
  m[8 * 32] = zz;
}

// One FP64 Yoshida step (the expression forms of k_propagate).  e3 = the step's three stage entries.
__device__ __forceinline__ void adjStep(uint32_t mask, double r[3], double v[3], double aom, double bc,
                                        const EphEntry *e3, const double2 *atm, const PropConsts &pc) {
  double a[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] += pc.hc1 * v[k];
  accel(mask, r, v, aom, bc, e3[0], atm, a);
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] += pc.hd1 * a[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] += pc.hc2 * v[k];
  accel(mask, r, v, aom, bc, e3[1], atm, a);
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] += pc.hd2 * a[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] += pc.hc2 * v[k];
  accel(mask, r, v, aom, bc, e3[2], atm, a);
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] += pc.hd1 * a[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] += pc.hc1 * v[k];
}

constexpr int kAdjObjs = 32;   // objects per block: lane = object, a pair in adjacent lanes
constexpr int kAdjForce = 3;   // warps of the forward sweep that share the force terms out
constexpr int kAdjFwdThreads = (kAdjForce + 1) * 32;
template <int W>
__device__ __forceinline__ constexpr uint32_t adjTerms() {
  return W == 0 ? kPropDRAG
                : W == 1 ? (kPropKEP | kPropJ2 | kPropJ3 | kPropTesseral) : (kPropSOL | kPropLUN | kPropSRP);
}

// The ephemeris of 16 steps (3 stage entries each) staged in shared memory:
// the terms' reads of the Sun, the Moon and the rotation angle at every stage
// would otherwise be L2 reads on the chain right after a block barrier.  The
// next chunk is loaded into registers while the current one is in use, and
// stored to shared memory at the switch, between two block barriers.  Every
// thread of the block calls use() with the same arguments.
constexpr int kEphChunkSteps = 16;
static_assert(sizeof(EphEntry) % 16 == 0, "ephemeris entries are staged as 16-byte words");
constexpr int kEphChunkWords = kEphChunkSteps * 3 * (int)(sizeof(EphEntry) / 16);
constexpr int kEphSlots = (kEphChunkWords + kAdjFwdThreads - 1) / kAdjFwdThreads;
struct EphStage {
  uint4 pre[kEphSlots];

  // issues the loads of steps [first, last)
  __device__ __forceinline__ void fetch(const EphEntry *__restrict__ eph, int first, int last) {
    const int words = min(max(last - first, 0), kEphChunkSteps) * 3 * (int)(sizeof(EphEntry) / 16);
    const uint4 *src = reinterpret_cast<const uint4 *>(eph + 3 * (size_t)first);
#pragma unroll
    for (int i = 0; i < kEphSlots; ++i) {
      const int w = (int)threadIdx.x + i * kAdjFwdThreads;
      if (w < words) pre[i] = __ldg(src + w);
    }
  }
  // makes the fetched steps current, then fetches the steps from `next`
  __device__ __forceinline__ void use(uint4 *buf, const EphEntry *__restrict__ eph, int next, int last) {
    __syncthreads();  // no warp reads the previous chunk any more
#pragma unroll
    for (int i = 0; i < kEphSlots; ++i) {
      const int w = (int)threadIdx.x + i * kAdjFwdThreads;
      if (w < kEphChunkWords) buf[w] = pre[i];
    }
    __syncthreads();
    fetch(eph, next, last);
  }
};

// Steps s0 + 1 .. s1 of the pairs from the states st (st[c * nObj + j],
// c = x, y, z, vx, vy, vz; objects 2p (A) and 2p + 1 (B) form pair p).
//   ckpt (or null): the state after step k ck at ckpt[(k * 6 + c) * nObj + j]
//   rec (or null): of each step the start state and the velocities of the
//     second and third kick, rec[((s - s0 - 1) * 12 + c) * nObj + j] -- all that
//     the reverse of the step needs
//   miss, argStep, seed (or all null): the pair's smallest squared miss distance,
//     its step, and d dl2 / d(r, v) there, seed[c * nObj + j]
//
// A few thousand objects leave most of the chip idle: the dependent chain of a
// step bounds the sweep, not its instructions.  So a block's 32 objects have
// four warps (lane = object): three hold the whole state and evaluate a third
// of the terms each, known at compile time (MASK, 0: from pc.mask); the partial
// accelerations meet in shared memory, one block barrier per stage, and every
// warp adds them in the same order.  The fourth warp follows the state and takes
// what is not part of the chain: the miss distances of the step before, and the
// stores.  The exchange buffer alternates between two halves, so a warp that
// has passed the barrier of stage n + 1 cannot overwrite the half that a slower
// warp still reads for stage n.  Lanes past the last object step a copy of it
// (every warp reaches every barrier) and write nothing.  4096 pairs, full set, per
// step: 2.56 us with four warps that share the terms by the runtime mask and
// all take the miss distance (2.24 of it with the terms of forces.cuh), 1.41 like
// this; 512 pairs 2.43 -> 1.33.
template <uint32_t MASK>
__global__ void __launch_bounds__(kAdjFwdThreads) k_adj_forward(
    const double *__restrict__ st, const double *__restrict__ bc, const double *__restrict__ aom, int nObj, int s0,
    int s1, const EphEntry *__restrict__ eph, PropConsts pc, double dt, int ck, double *__restrict__ ckpt,
    double *__restrict__ rec, double *__restrict__ miss, int *__restrict__ argStep, double *__restrict__ seed) {
  __shared__ double ex[2][kAdjForce][3][kAdjObjs];
  __shared__ uint4 ephBuf[kEphChunkWords];
  const uint32_t mask = MASK ? MASK : pc.mask;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j0 = blockIdx.x * kAdjObjs + lane;
  const bool live = j0 < nObj;
  const int j = live ? j0 : nObj - 1;
  EphStage es;
  es.fetch(eph, s0, s1);
  double r[3] = {st[j], st[nObj + j], st[2 * nObj + j]};
  double v[3] = {st[3 * nObj + j], st[4 * nObj + j], st[5 * nObj + j]};
  const double myBc = bc[j], myAom = aom[j];
  const bool isA = (lane & 1) == 0, writer = live && w == kAdjForce;
  double best = INFINITY, sd[6] = {0, 0, 0, 0, 0, 0};
  int arg = 0, half = 0;
  // the miss distance of the step that has ended with (r, v); NaN never wins
  auto missOf = [&](int s) {
    double a[6], o[6], dr[3], p2[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double pr = __shfl_xor_sync(0xffffffffu, r[c], 1), pv = __shfl_xor_sync(0xffffffffu, v[c], 1);
      a[c] = isA ? r[c] : pr;
      a[3 + c] = isA ? v[c] : pv;
      o[c] = isA ? pr : r[c];
      o[3 + c] = isA ? pv : v[c];
    }
    const double t = interpolate(a, a + 3, o, o + 3, dt, dr, p2), d2 = dot3rn(dr, dr);
    if (d2 < best) {
      best = d2;
      arg = s;
      const double sign = isA ? 2.0 : -2.0, tv = t - dt;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sd[c] = sign * dr[c];
        sd[3 + c] = sign * dr[c] * tv;
      }
    }
  };
  const double hc[3] = {pc.hc1, pc.hc2, pc.hc2}, hd[3] = {pc.hd1, pc.hd2, pc.hd1};
  for (int s = s0; s < s1; ++s) {
    const int inChunk = (s - s0) % kEphChunkSteps;
    if (inChunk == 0) es.use(ephBuf, eph, s + kEphChunkSteps, s1);
    const EphEntry *e3 = reinterpret_cast<const EphEntry *>(ephBuf) + 3 * inChunk;
    double *q = rec + (size_t)(s - s0) * 12 * nObj + j;
    if (w == kAdjForce) {
      if (miss && s > s0) missOf(s);
      if (writer && ckpt && s % ck == 0) {
        double *k = ckpt + (size_t)(s / ck) * 6 * nObj + j;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          k[(size_t)c * nObj] = r[c];
          k[(size_t)(3 + c) * nObj] = v[c];
        }
      }
      if (writer && rec) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          q[(size_t)c * nObj] = r[c];
          q[(size_t)(3 + c) * nObj] = v[c];
        }
      }
    }
#pragma unroll
    for (int g = 0; g < 3; ++g) {
#pragma unroll
      for (int k = 0; k < 3; ++k) r[k] += hc[g] * v[k];
      double a[3];
      if (w == 0) accel(mask & adjTerms<0>(), r, v, myAom, myBc, e3[g], pc.atm, a);
      if (w == 1) accel(mask & adjTerms<1>(), r, v, myAom, myBc, e3[g], pc.atm, a);
      if (w == 2) accel(mask & adjTerms<2>(), r, v, myAom, myBc, e3[g], pc.atm, a);
      if (w < kAdjForce) {
#pragma unroll
        for (int k = 0; k < 3; ++k) ex[half][w][k][lane] = a[k];
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double sum = ex[half][0][k][lane] + ex[half][1][k][lane] + ex[half][2][k][lane];
        v[k] += hd[g] * sum;
      }
      half ^= 1;
      if (g < 2 && writer && rec) {
#pragma unroll
        for (int c = 0; c < 3; ++c) q[(size_t)(6 + 3 * g + c) * nObj] = v[c];
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] += pc.hc1 * v[k];
  }
  if (w != kAdjForce || !miss) return;
  missOf(s1);
  if (!live) return;
#pragma unroll
  for (int c = 0; c < 6; ++c) seed[(size_t)c * nObj + j] = sd[c];
  if (isA) {
    miss[j >> 1] = best;
    argStep[j >> 1] = arg;
  }
}

// Reverse of steps s1 .. s0 + 1 from their records (of k_adj_forward), grad[c * nObj + j]: c = 0..5
// dL/d(r, v), c = 6 dL/dbcInv; `first`: the adjoint starts at zero, else from grad.
//
// What depends on the step after is little: a 3 x 3 product or two per kick.
// The Jacobians do not -- every stage position is in the records -- so nine warps
// evaluate those of three steps side by side (warp = stage of a step, lane =
// object) into shared memory, while a tenth takes the adjoint through the three
// steps before; one block barrier per three steps, two buffers.  The producers'
// loads are issued one batch ahead.  4096 pairs, full set, per step: 6.17 us with the
// products of each kick formed on the chain (and the segments' states again; 4.28
// with the terms of forces.cuh), 0.79 like this (FP64 pipe 51 % busy); 512 pairs 5.07 ->
// 0.46.
constexpr int kAdjBatchSteps = 3;
constexpr int kAdjProducers = 3 * kAdjBatchSteps;
constexpr int kAdjBwdThreads = (kAdjProducers + 1) * 32;
constexpr int kEphWords = (int)(sizeof(EphEntry) / sizeof(double));
struct AdjBackShared {
  double m[2][kAdjProducers][kJacWords][kAdjObjs];
  double eph[kAdjProducers][kEphWords];
};
static_assert(kEphWords <= 32, "a warp stages an ephemeris entry with one load");

template <uint32_t MASK>
__global__ void __launch_bounds__(kAdjBwdThreads, 2) k_adj_backward(
    const double *__restrict__ bc, const double *__restrict__ aom, int nObj, int s0, int s1,
    const EphEntry *__restrict__ eph, PropConsts pc, const double *__restrict__ rec, const int *__restrict__ argStep,
    const double *__restrict__ seed, bool first, double *__restrict__ grad) {
  extern __shared__ __align__(16) unsigned char adjSmem[];
  AdjBackShared &sh = *reinterpret_cast<AdjBackShared *>(adjSmem);
  const uint32_t mask = MASK ? MASK : pc.mask;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j0 = blockIdx.x * kAdjObjs + lane;
  const bool live = j0 < nObj;
  const int j = live ? j0 : nObj - 1;
  const int batches = (s1 - s0 + kAdjBatchSteps - 1) / kAdjBatchSteps;
  // batch b: steps s1 - 3 b, one less, two less, each with its third stage first
  if (w < kAdjProducers) {
    const int stage = 2 - w % 3;
    const double myBc = bc[j], myAom = aom[j];
    double in[12], en = 0.0;
    auto load = [&](int b) {
      const int s = s1 - b * kAdjBatchSteps - w / 3;
      if (s <= s0) return;
      const double *q = rec + (size_t)(s - s0 - 1) * 12 * nObj + j;
#pragma unroll
      for (int c = 0; c < 6; ++c) in[c] = __ldg(q + (size_t)c * nObj);
      if (stage > 0) {
#pragma unroll
        for (int c = 6; c < 9; ++c) in[c] = __ldg(q + (size_t)c * nObj);
      }
      if (stage > 1) {
#pragma unroll
        for (int c = 9; c < 12; ++c) in[c] = __ldg(q + (size_t)c * nObj);
      }
      if (lane < kEphWords)
        en = __ldg(reinterpret_cast<const double *>(eph + 3 * (size_t)(s - 1) + stage) + lane);
    };
    load(0);
    for (int b = 0; b <= batches; ++b) {
      if (b < batches && s1 - b * kAdjBatchSteps - w / 3 > s0) {
        double r[3], v[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          r[k] = in[k];
          r[k] += pc.hc1 * in[3 + k];
          v[k] = in[3 + k];
          if (stage > 0) {
            r[k] += pc.hc2 * in[6 + k];
            v[k] = in[6 + k];
          }
          if (stage > 1) {
            r[k] += pc.hc2 * in[9 + k];
            v[k] = in[9 + k];
          }
        }
        __syncwarp();
        if (lane < kEphWords) sh.eph[w][lane] = en;
        __syncwarp();
        if (b + 1 < batches) load(b + 1);
        accelJacobian(mask, r, v, myAom, myBc, reinterpret_cast<const EphEntry &>(sh.eph[w]), pc.atm,
                      &sh.m[b & 1][w][0][lane]);
      }
      __syncthreads();
    }
    return;
  }
  double lr[3] = {0, 0, 0}, lv[3] = {0, 0, 0}, lbc = 0.0;
  if (!first) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      lr[c] = grad[(size_t)c * nObj + j];
      lv[c] = grad[(size_t)(3 + c) * nObj + j];
    }
    lbc = grad[(size_t)6 * nObj + j];
  }
  const int sStar = argStep[j >> 1];
  double sd[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) sd[c] = seed[(size_t)c * nObj + j];
  const double hd[3] = {pc.hd1, pc.hd2, pc.hd1}, hc[3] = {pc.hc2, pc.hc2, pc.hc1};
  for (int b = 0; b <= batches; ++b) {
    if (b > 0) {
      const int sTop = s1 - (b - 1) * kAdjBatchSteps;
#pragma unroll
      for (int i = 0; i < kAdjBatchSteps; ++i) {
        const int s = sTop - i;
        if (s <= s0) break;
        if (s == sStar) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            lr[c] += sd[c];
            lv[c] += sd[3 + c];
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) lv[c] += pc.hc1 * lr[c];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double *m = &sh.m[(b - 1) & 1][3 * i + k][0][lane];
          const double gx = hd[k] * lv[0], gy = hd[k] * lv[1], gz = hd[k] * lv[2];
#pragma unroll
          for (int c = 0; c < 3; ++c) lr[c] += m[(3 * c) * 32] * gx + m[(3 * c + 1) * 32] * gy + m[(3 * c + 2) * 32] * gz;
          if (mask & kPropDRAG) {
            lv[0] += m[9 * 32] * gx + m[10 * 32] * gy + m[11 * 32] * gz;
            lv[1] += m[10 * 32] * gx + m[12 * 32] * gy + m[13 * 32] * gz;
            lv[2] += m[11 * 32] * gx + m[13 * 32] * gy + m[14 * 32] * gz;
            lbc += m[15 * 32] * gx + m[16 * 32] * gy + m[17 * 32] * gz;
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) lv[c] += hc[k] * lr[c];
        }
      }
    }
    __syncthreads();
  }
  if (!live) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    grad[(size_t)c * nObj + j] = lr[c];
    grad[(size_t)(3 + c) * nObj + j] = lv[c];
  }
  grad[(size_t)6 * nObj + j] = lbc;
}

// Synthetic conjunction pairs: A forward tca[p] steps, B = A + (dr, dv), then
// B backward tca[p] steps (stage entries of each step in reverse order: the
// composition is symmetric, so the stage times of a backward step are those
// of the forward step it retraces).  st: object SoA as above, B slots
// (2p + 1) receive the back-propagated state.
__global__ void __launch_bounds__(128) k_adj_make_pairs(double *__restrict__ st, const double *__restrict__ bc,
                                                        const double *__restrict__ aom, int nPairs,
                                                        const int *__restrict__ tca, const double *__restrict__ off,
                                                        const EphEntry *__restrict__ eph, PropConsts pc,
                                                        PropConsts back) {
  const double2 *atm = pc.atm;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nPairs) return;
  const int nObj = 2 * nPairs, a = 2 * p, b = 2 * p + 1;
  double r[3] = {st[a], st[nObj + a], st[2 * nObj + a]};
  double v[3] = {st[3 * nObj + a], st[4 * nObj + a], st[5 * nObj + a]};
  const int n = tca[p];
  for (int s = 0; s < n; ++s) adjStep(pc.mask, r, v, aom[a], bc[a], eph + 3 * s, atm, pc);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    r[c] += off[6 * p + c];
    v[c] += off[6 * p + 3 + c];
  }
  for (int s = n - 1; s >= 0; --s) {
    const EphEntry e3[3] = {eph[3 * s + 2], eph[3 * s + 1], eph[3 * s]};
    adjStep(back.mask, r, v, aom[b], bc[b], e3, atm, back);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    st[(size_t)c * nObj + b] = r[c];
    st[(size_t)(3 + c) * nObj + b] = v[c];
  }
}

}  // namespace ladds
