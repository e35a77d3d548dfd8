// insert.cuh -- checked insertion of new satellites (Simulation::checkedInsert,
// Simulation.cpp:475-507).
//
// A new satellite at p is inserted only if no particle q inside the box
// [p - c, p + c) (the AutoPas region iterator's half-open box, corners from
// ArrayMath::sub / add) has dot(p - q, p - q) <= c^2 (collisionFree =
// dot > c^2, so NaN also blocks); c = io/constellationCutoff.  The kernel tests
// every new satellite against the device population (deleted objects are
// absent in the reference and skipped here); satellites of the same batch are
// tested against the ones accepted before them on the host, in batch order.
#pragma once
#include "conjunction.cuh"
#include "propagate.cuh"

namespace ladds {

// the reference's test of one particle q against a satellite at p
__host__ __device__ __forceinline__ bool insertBlocks(const double p[3], const double q[3], double c, double c2) {
#ifdef __CUDA_ARCH__
#define LADDS_ADD(a, b) __dadd_rn(a, b)
#define LADDS_SUB(a, b) __dsub_rn(a, b)
#define LADDS_MUL(a, b) __dmul_rn(a, b)
#else
#define LADDS_ADD(a, b) ((a) + (b))
#define LADDS_SUB(a, b) ((a) - (b))
#define LADDS_MUL(a, b) ((a) * (b))
#endif
  for (int k = 0; k < 3; ++k) {
    const double lo = LADDS_SUB(p[k], c), hi = LADDS_ADD(p[k], c);
    if (!(q[k] >= lo && q[k] < hi)) return false;  // outside the region iterator's box
  }
  const double d0 = LADDS_SUB(p[0], q[0]), d1 = LADDS_SUB(p[1], q[1]), d2 = LADDS_SUB(p[2], q[2]);
  double s = LADDS_ADD(0.0, LADDS_MUL(d0, d0));
  s = LADDS_ADD(s, LADDS_MUL(d1, d1));
  s = LADDS_ADD(s, LADDS_MUL(d2, d2));
#undef LADDS_ADD
#undef LADDS_SUB
#undef LADDS_MUL
  return !(s > c2);
}

// one warp per new satellite: blocked[i] = some live particle of the state blocks it
__global__ void k_insert_blocked(DevState s, int n, const double *__restrict__ nx, const double *__restrict__ ny,
                                 const double *__restrict__ nz, int nNew, double c, double c2,
                                 uint8_t *__restrict__ blocked) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= nNew) return;  // whole warps exit together
  const double p[3] = {nx[w], ny[w], nz[w]};
  bool hit = false;
  for (int jb = 0; jb < n; jb += 32) {  // warp-uniform trip count
    const int j = jb + lane;
    if (j < n && !tagDummy(s.tag[j])) {
      const double q[3] = {s.x[j], s.y[j], s.z[j]};
      hit = hit || insertBlocks(p, q, c, c2);
    }
    if (__any_sync(0xffffffffu, hit)) break;
  }
  hit = __any_sync(0xffffffffu, hit);
  if (lane == 0) blocked[w] = hit ? 1 : 0;
}

// records of the objects slots[0..m)
__global__ void k_gather_records(DevState s, const uint32_t *__restrict__ slots, int m,
                                 ladds_state_record *__restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  const uint32_t j = slots[q];
  ladds_state_record r;
  r.r[0] = s.x[j];
  r.r[1] = s.y[j];
  r.r[2] = s.z[j];
  r.v[0] = s.vx[j];
  r.v[1] = s.vy[j];
  r.v[2] = s.vz[j];
  r.radius = s.radius[j];
  r.aom = s.aom[j];
  r.bcInv = s.bc[j];
  r.id = s.id[j];
  r.parentId = s.parent[j];
  r.activity = tagAct(s.tag[j]);
  r.deleted = tagDummy(s.tag[j]) ? 1u : 0u;
  out[q] = r;
}

// Layer selection of the device-resident exchange (ladds_gpu_pack_layers):
// keep[slot] = 0 for the live objects whose cell layer lies in [lo, hi), 1 for
// the others (the removal's flags); then sel[i] = !keep of the i-th object of the
// population's order -- perm for the first m, then slot order.  Through perm go four
// bytes an object, not its position and tag (1e6 objects after a scan, call 79 -> 64 us
// with its counts fetched by one wait).
__global__ void k_layer_flags(const double *__restrict__ z, const uint32_t *__restrict__ tag, int n, GridDesc g,
                              int32_t lo, int32_t hi, uint32_t *__restrict__ keep) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int32_t iz = (int32_t)cellCoord(z[j], g.boxMin[2], g.invCell, g.n[2]);
  keep[j] = (!tagDummy(tag[j]) && iz >= lo && iz < hi) ? 0u : 1u;
}
__global__ void k_order_select(const uint32_t *__restrict__ keep, const uint32_t *__restrict__ perm, int m, int n,
                               uint32_t *__restrict__ sel) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) sel[i] = 1u - keep[i < m ? perm[i] : (uint32_t)i];
}

// slots of the selected objects in that order, *count = their number
__global__ void k_selected_slots(const uint32_t *__restrict__ sel, const uint32_t *__restrict__ pos,
                                 const uint32_t *__restrict__ perm, int m, int n, uint32_t *__restrict__ slots,
                                 uint32_t *__restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (i == n - 1) *count = pos[i] + sel[i];
  if (sel[i]) slots[pos[i]] = i < m ? perm[i] : (uint32_t)i;
}

// compaction of an order: flag[i] = keep[perm[i]]; then moved[at[i]] = the new slot of a kept one, *count = their number
__global__ void k_order_flags(const uint32_t *__restrict__ perm, const uint32_t *__restrict__ keep, int m,
                              uint32_t *__restrict__ flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) flag[i] = keep[perm[i]];
}
__global__ void k_order_compact(const uint32_t *__restrict__ perm, const uint32_t *__restrict__ flag,
                                const uint32_t *__restrict__ at, const uint32_t *__restrict__ pos, int m,
                                uint32_t *__restrict__ moved, uint32_t *__restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  if (i == m - 1) *count = at[i] + flag[i];
  if (flag[i]) moved[at[i]] = pos[perm[i]];
}
// a truncation's flags and slots
__global__ void k_below_flags(int n, uint32_t n0, uint32_t *__restrict__ keep, uint32_t *__restrict__ pos) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) {
    keep[j] = (uint32_t)j < n0 ? 1u : 0u;
    pos[j] = (uint32_t)j;
  }
}

// State records (device memory) appended at slots offset..offset+m; bad[0] counts
// records with a non-finite value or an activity state out of range, bad[1]
// is set when a record has a parent id.
__global__ void k_append_records(const ladds_state_record *__restrict__ in, int m, DevState s, uint32_t offset,
                                 unsigned *__restrict__ bad) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  const ladds_state_record r = in[q];
  const uint32_t at = offset + (uint32_t)q;
  const bool ok = isfinite(r.r[0]) && isfinite(r.r[1]) && isfinite(r.r[2]) && isfinite(r.v[0]) &&
                  isfinite(r.v[1]) && isfinite(r.v[2]) && isfinite(r.radius) && isfinite(r.aom) &&
                  isfinite(r.bcInv) && r.activity >= 0 && r.activity <= 2;
  if (!ok) atomicAdd(bad, 1u);
  if (r.parentId != UINT64_MAX) atomicOr(bad + 1, 1u);
  s.x[at] = r.r[0];
  s.y[at] = r.r[1];
  s.z[at] = r.r[2];
  s.vx[at] = r.v[0];
  s.vy[at] = r.v[1];
  s.vz[at] = r.v[2];
  s.aom[at] = r.aom;
  s.bc[at] = r.bcInv;
  s.radius[at] = r.radius;
  s.id[at] = r.id;
  s.parent[at] = r.parentId;
  s.tag[at] = makeTag(at, ok ? r.activity : 0, r.deleted != 0u);
}

}  // namespace ladds
