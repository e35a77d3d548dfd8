// state.cuh -- device layout of the particle population.
//
// Structure of arrays, one array per attribute of the reference Particle
// (Particle.h:139-195) that the hot path reads, indexed by slot (the upload
// index).  Positions and velocities are binary64 (48 B/object) in a ring of three
// buffers: the propagation that ends at a scan reads one and writes the next, so
// that it can run beside the sort and the scan of the iterations before it; a
// fourth copy is what a call of several launches is undone from.  The per-object
// constants aom / bcInv / radius (binary64), id / parentId (u64) and a u32 tag (the
// slot, the activity state and the dummy "deleted" flag) exist once.  Cell order
// exists only in what the pair scan reads: the row sort gathers 32-byte scan
// records into it.
#pragma once
#include <cstdint>

namespace ladds {

constexpr uint32_t kTagSlotBits = 28;
constexpr uint32_t kTagSlotMask = (1u << kTagSlotBits) - 1u;
constexpr uint32_t kTagActShift = 28;
constexpr uint32_t kTagDummy = 1u << 31;
constexpr size_t kMaxObjects = (size_t)kTagSlotMask;  // 268 M

__host__ __device__ __forceinline__ uint32_t makeTag(uint32_t slot, int act, bool dummy) {
  return (slot & kTagSlotMask) | ((uint32_t)(act & 3) << kTagActShift) | (dummy ? kTagDummy : 0u);
}
__host__ __device__ __forceinline__ uint32_t tagSlot(uint32_t t) { return t & kTagSlotMask; }
__host__ __device__ __forceinline__ int tagAct(uint32_t t) { return (int)((t >> kTagActShift) & 3u); }
__host__ __device__ __forceinline__ bool tagDummy(uint32_t t) { return (t & kTagDummy) != 0; }

// One state buffer: x .. vz are its own, the other arrays are shared by a
// context's buffers.
struct DevState {
  double *x, *y, *z, *vx, *vy, *vz;
  double *aom, *bc, *radius;
  uint64_t *id, *parent;
  uint32_t *tag;
};

// What the pair scan reads of an object, written in slot order with its cell
// key and gathered into cell order by the row sort: one 32-byte sector.
// Binary32 position with a bound on its rounding error per coordinate (its
// sign bit marks a deleted object), binary32 velocity, radius rounded up.
struct __align__(32) ScanRec {
  float4 pos, vel;
};

// cell grid: key = (iz * ny + iy) * nx + ix
struct GridDesc {
  double boxMin[3];
  double cellSize, invCell;
  int32_t n[3];
  int32_t reach;
  uint32_t keyBits;
};

struct ScanConsts {
  double cutoffSq;    // cutoff * cutoff                        (CollisionFunctor.cpp:24)
  double dt;          // interpolation window
  double factor;      // collisionDistanceFactor / 1000.        (CollisionFunctor.cpp:26)
  double minDetectionRadius;
  double evasionSq;   // evasionCutoff * evasionCutoff          (CollisionFunctor.cpp:28)
  double conjSq;      // conjunctionThreshold^2
  double nearRel;
  // binary32 forms for the screen of the pair scan (mayRecord), derived from the
  // fields above by screenConsts() before every scan launch
  float dtF, factorF, relF, thrF, cut2F, cutF, nearBandF, errV, err0;
};

}  // namespace ladds
