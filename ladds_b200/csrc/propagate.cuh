// propagate.cuh -- Yoshida-4 propagation kernels (+ the input of the scan that follows).
//
// Replaces YoshidaIntegrator::integrate(false) (called at Simulation.cpp:297;
// the integrator itself is in the non-vendored OrbitPropagator).  Form: DKD
// composition of Yoshida (1990): drift c1, kick d1, drift c2, kick d2,
// drift c2, kick d1, drift c1 -- three force evaluations per step at the
// stage times t + c1 dt, t + (c1+c2) dt, t + (c1+2 c2) dt.
//
// One thread per object, state held in registers across `nSteps` steps, so
// a multi-step launch touches HBM once (read 64 B + write 48 B per object).
// Ephemeris entries of all stages of the launch live in __constant__ memory
// (uniform across the warp).
#pragma once
#include "bulk_copy.cuh"
#include "cell_sort.cuh"
#include "conjunction.cuh"
#include "forces.cuh"
#include "state.cuh"

#include <type_traits>

namespace ladds {

constexpr int kMaxEphSteps = 128;  // 3 * 128 entries * 112 B (FP64) or 88 B (split): up to 43 KB of constant memory
template <bool SPLIT>
using EphOf = typename std::conditional<SPLIT, EphEntryF, EphEntry>::type;
static_assert(sizeof(EphEntryF) <= sizeof(EphEntry), "the stage table holds entries of either form");
__constant__ __align__(256) unsigned char c_eph[3 * kMaxEphSteps * sizeof(EphEntry)];
template <bool SPLIT>
__device__ __forceinline__ const EphOf<SPLIT> *stageTable() {
  return reinterpret_cast<const EphOf<SPLIT> *>(c_eph);
}
// the atmosphere table that a force evaluation reads
template <bool SPLIT>
using AtmOf = typename std::conditional<SPLIT, AtmShared, const double2 *>::type;

struct PropConsts {
  double hc1, hc2, hd1, hd2;  // Yoshida coefficients * dt
  uint32_t mask;
  const double2 *atm;  // the fine atmosphere table
};

// floor((v - lo) * inv) with exactly these two roundings; NaN -> 0; clamped to
// [0, n).  The floor of a value below 2^31 is the low word of its sum with
// 3 * 2^51 rounded down; larger values, infinities and NaN are told by the high word.
__device__ __forceinline__ uint32_t cellCoord(double v, double lo, double inv, int32_t n) {
  const double u = __dmul_rn(__dsub_rn(v, lo), inv);
  const int hi = __double2hiint(u);
  if (hi < 0) return 0u;  // negative (or -0)
  if (hi >= 0x41e00000) return u >= 2147483648.0 ? (uint32_t)(n - 1) : 0u;
  return (uint32_t)min(__double2loint(__dadd_rd(u, 6755399441055744.0)), n - 1);
}

struct CellOf {
  uint32_t row, key;
};
__device__ __forceinline__ CellOf cellOf(double x, double y, double z, const GridDesc &g) {
  const uint32_t ix = cellCoord(x, g.boxMin[0], g.invCell, g.n[0]);
  const uint32_t iy = cellCoord(y, g.boxMin[1], g.invCell, g.n[1]);
  const uint32_t iz = cellCoord(z, g.boxMin[2], g.invCell, g.n[2]);
  const uint32_t row = iz * (uint32_t)g.n[1] + iy;
  return {row, row * (uint32_t)g.n[0] + ix};
}

// What a scan needs of an object that has just been propagated (or is
// scanned as it is), in slot order: its cell key, its arrival index in its
// cell row, and its 32-byte scan record (ScanRec).
struct ScanInput {
  uint32_t *keys, *rowCount, *arrival;
  ScanRec *rec;
  const double *radius;
};
// every lane of the warp calls it (inRange = false for lanes without an object)
__device__ __forceinline__ void writeScanInput(const ScanInput &o, const GridDesc &g, int j, bool inRange,
                                               const double r[3], const double v[3], uint32_t tag) {
  const CellOf c = cellOf(r[0], r[1], r[2], g);
  const uint32_t a = countRowArrival(c.row, inRange, o.rowCount);
  if (!inRange) return;
  o.keys[j] = c.key;
  o.arrival[j] = a;
  o.rec[j] = scanRec(r, v, o.radius[j], tagDummy(tag));
}

// nSteps Yoshida-4 steps of one object (stage ephemerides ephBase ... of the
// stage table); a non-finite end state sets bit 1 of *status.
template <bool SPLIT>
__device__ __forceinline__ void yoshidaLoop(uint32_t mask, double r[3], double v[3], double aom, double bc,
                                            int nSteps, int ephBase, const PropConsts &pc,
                                            const AtmOf<SPLIT> &atm) {
  using C = typename std::conditional<SPLIT, float, double>::type;
  const C aomC = (C)aom, bcC = (C)bc;
  const EphOf<SPLIT> *e = stageTable<SPLIT>() + ephBase;
  double a[3];
  for (int st = 0; st < nSteps; ++st, e += 3) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] += pc.hc1 * v[k];
    accel(mask, r, v, aomC, bcC, e[0], atm, a);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += pc.hd1 * a[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] += pc.hc2 * v[k];
    accel(mask, r, v, aomC, bcC, e[1], atm, a);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += pc.hd2 * a[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] += pc.hc2 * v[k];
    accel(mask, r, v, aomC, bcC, e[2], atm, a);
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += pc.hd1 * a[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] += pc.hc1 * v[k];
  }
}
// MASK: the launch's component mask where it is known at compile time, else 0.
// evasive-preserving objects (Keplerian forces only, Particle.h:48-52) take a loop of
// their own, so that in the other one the mask is the launch's and its branches are
// uniform.  A warp that holds both kinds goes through both loops, which a mask known
// at compile time pays back; without it the warp takes one loop with each object's own
// mask (200,000 objects, every third of them such, per step: central + J2 3.0 -> 2.4 us,
// central alone 2.7 -> 1.7, central + drag split 3.9 -> 3.4).
template <bool SPLIT, uint32_t MASK>
__device__ __forceinline__ void yoshidaSteps(double r[3], double v[3], double aom, double bc, uint32_t tag,
                                             int nSteps, int ephBase, const PropConsts &pc,
                                             const AtmShared &atmS, unsigned *__restrict__ status) {
  const AtmOf<SPLIT> &atm = [&]() -> const AtmOf<SPLIT> & {
    if constexpr (SPLIT)
      return atmS;
    else
      return pc.atm;
  }();
  const bool keplerian = tagAct(tag) == kEvasivePreserving && (pc.mask & ~kPropKEP) != 0u;
  if (MASK ? keplerian : __any_sync(__activemask(), keplerian))
    yoshidaLoop<SPLIT>(MASK || keplerian ? pc.mask & kPropKEP : pc.mask, r, v, aom, bc, nSteps, ephBase, pc, atm);
  else
    yoshidaLoop<SPLIT>(MASK ? MASK : pc.mask, r, v, aom, bc, nSteps, ephBase, pc, atm);
  if (!(isfinite(r[0]) && isfinite(r[1]) && isfinite(r[2]) && isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2])))
    atomicOr(status, 1u);
}

// Propagation without a scan: nSteps steps in place, one object per thread.
template <bool SPLIT, uint32_t MASK>
__global__ void __launch_bounds__(256, 4) k_propagate(DevState s, int n, int nSteps, int ephBase, PropConsts pc,
                                                   unsigned *__restrict__ status) {
  __shared__ AtmShared atmS;
  if (SPLIT) {
    loadAtmTable(atmS);
    __syncthreads();
  }
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t tag = s.tag[j];
  if (tagDummy(tag)) return;
  double r[3] = {s.x[j], s.y[j], s.z[j]}, v[3] = {s.vx[j], s.vy[j], s.vz[j]};
  yoshidaSteps<SPLIT, MASK>(r, v, s.aom[j], s.bc[j], tag, nSteps, ephBase, pc, atmS, status);
  s.x[j] = r[0];
  s.y[j] = r[1];
  s.z[j] = r[2];
  s.vx[j] = v[0];
  s.vy[j] = v[1];
  s.vz[j] = v[2];
}

// The propagation that ends at a scan (nSteps steps: those since the scan
// before it), over a persistent grid.  CTA b takes the tiles b, b + gridDim.x,
// ... of kStageObjects consecutive slots.  While a tile is propagated, the
// state of the CTA's next tile is already on its way into shared memory: one
// thread issues nine bulk copies (x, y, z, vx, vy, vz, aom, bc: 2 KB each;
// tags: 1 KB) completed on an mbarrier, so no warp stalls on its loads after
// the first tile.  The partial tile at the end (n % kStageObjects
// objects) is read directly.  The new state goes to `to`, which may be s
// itself: the state before it stays readable for the pair scan that is still
// running on it.  Per-object arithmetic and results are k_propagate's.  A wait
// that runs out (it cannot, unless a copy is lost) sets bit 8 of *status.
constexpr int kStageObjects = 256;
constexpr int kStageArrays = 8;
constexpr uint32_t kStageTxBytes = kStageArrays * kStageObjects * 8 + kStageObjects * 4;
constexpr uint32_t kStageWaitPolls = 1u << 22;

template <bool SPLIT, bool SCAN, uint32_t MASK>
__global__ void __launch_bounds__(kStageObjects, 4) k_propagate_staged(DevState s, DevState to, int n, int nSteps,
                                                                      int ephBase, PropConsts pc, GridDesc g,
                                                                      ScanInput scan, unsigned *__restrict__ status) {
  __shared__ AtmShared atmS;
  __shared__ __align__(16) double sv[kStageArrays][kStageObjects];
  __shared__ __align__(16) uint32_t stag[kStageObjects];
  __shared__ __align__(8) unsigned long long sbar;
  const int tid = threadIdx.x;
  const int nFull = n / kStageObjects, nTiles = (n + kStageObjects - 1) / kStageObjects;
  // one thread: the copies of full tile t into the stage
  auto issue = [&](int t) {
    const size_t base = (size_t)t * kStageObjects;
    const double *src[kStageArrays] = {s.x, s.y, s.z, s.vx, s.vy, s.vz, s.aom, s.bc};
    asyncProxyFence();
    mbarArriveExpectTx(&sbar, kStageTxBytes);
#pragma unroll
    for (int a = 0; a < kStageArrays; ++a) bulkLoad(sv[a], src[a] + base, kStageObjects * 8, &sbar);
    bulkLoad(stag, s.tag + base, kStageObjects * 4, &sbar);
  };
  if (tid == 0) {
    mbarInit(&sbar, 1);
    mbarInitFence();
  }
  if (SPLIT) loadAtmTable(atmS);
  __syncthreads();
  int t = blockIdx.x;
  if (tid == 0 && t < nFull) issue(t);
  for (uint32_t it = 0; t < nTiles; t += gridDim.x) {  // t is the same in every thread of the CTA
    const int j = t * kStageObjects + tid;
    const bool inRange = j < n;
    double r[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0}, aom = 0.0, bc = 0.0;
    uint32_t tag = kTagDummy;
    if (t < nFull) {
      if (!mbarWait(&sbar, it & 1u, kStageWaitPolls)) atomicOr(status, 8u);
      ++it;
      r[0] = sv[0][tid];
      r[1] = sv[1][tid];
      r[2] = sv[2][tid];
      v[0] = sv[3][tid];
      v[1] = sv[4][tid];
      v[2] = sv[5][tid];
      aom = sv[6][tid];
      bc = sv[7][tid];
      tag = stag[tid];
      __syncthreads();  // the stage is free: the next tile's copies go out now
      if (tid == 0 && t + (int)gridDim.x < nFull) issue(t + (int)gridDim.x);
    } else if (inRange) {
      tag = s.tag[j];
      r[0] = s.x[j];
      r[1] = s.y[j];
      r[2] = s.z[j];
      v[0] = s.vx[j];
      v[1] = s.vy[j];
      v[2] = s.vz[j];
      aom = s.aom[j];
      bc = s.bc[j];
    }
    if (!tagDummy(tag)) yoshidaSteps<SPLIT, MASK>(r, v, aom, bc, tag, nSteps, ephBase, pc, atmS, status);
    if (inRange) {  // deleted objects too: both buffers hold them
      to.x[j] = r[0];
      to.y[j] = r[1];
      to.z[j] = r[2];
      to.vx[j] = v[0];
      to.vy[j] = v[1];
      to.vz[j] = v[2];
    }
    // every lane of the warp reaches this point
    if (SCAN) writeScanInput(scan, g, j, inRange, r, v, tag);
  }
}

// slots of the live objects whose cell layer iz (the z index of the cell key)
// lies in [lo, hi), appended in any order
__global__ void k_select_layers(const double *__restrict__ z, const uint32_t *__restrict__ tag, int n, GridDesc g,
                                int32_t lo, int32_t hi, uint32_t *__restrict__ out, unsigned *__restrict__ count,
                                unsigned cap) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n || tagDummy(tag[j])) return;
  const int32_t iz = (int32_t)cellCoord(z[j], g.boxMin[2], g.invCell, g.n[2]);
  if (iz < lo || iz >= hi) return;
  const unsigned q = atomicAdd(count, 1u);
  if (q < cap) out[q] = tagSlot(tag[j]);
}

// live objects per cell layer
__global__ void k_layer_histogram(const double *__restrict__ z, const uint32_t *__restrict__ tag, int n, GridDesc g,
                                  unsigned long long *__restrict__ counts) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n || tagDummy(tag[j])) return;
  atomicAdd(&counts[cellCoord(z[j], g.boxMin[2], g.invCell, g.n[2])], 1ull);
}

// Ephemeris of the stage times of `nSteps` steps starting at iteration `iter`
// (one thread per stage), written to a global staging table that the host then
// copies into c_eph.
__global__ void k_ephemeris(EphEntry *__restrict__ out, int nSteps, int64_t iter, double t0, double dt, double hc1,
                            double hc2, double jdEpoch, double theta0, uint32_t mask) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * nSteps) return;
  const int st = i / 3, stage = i % 3;
  const double tn = t0 + (double)(iter + st) * dt;
  double tau = tn + hc1;
  if (stage >= 1) tau += hc2;
  if (stage >= 2) tau += hc2;
  ephemerisEntry(jdEpoch, theta0, tau, mask, out[i]);
}

// scan input of the current state
__global__ void k_scan_input(DevState s, int n, GridDesc g, ScanInput scan) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const bool inRange = j < n;
  double r[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0};
  uint32_t tag = 0;
  if (inRange) {
    r[0] = s.x[j], r[1] = s.y[j], r[2] = s.z[j];
    v[0] = s.vx[j], v[1] = s.vy[j], v[2] = s.vz[j];
    tag = s.tag[j];
  }
  writeScanInput(scan, g, j, inRange, r, v, tag);
}

}  // namespace ladds
