// ladds_gpu.cu -- C ABI of the B200 hot path (see include/ladds_gpu.h).
//
// One context = one device, three streams (propagation, sort, pair scan), the
// device-resident population: one array per attribute in slot order, positions
// and velocities in a ring of three buffers (the propagation that ends at a scan
// reads the current one and writes the next, while the scans before it still read
// theirs) and a fourth copy that a ladds_gpu_step call of several propagation
// launches is undone from.
//
// A scan iteration is: ephemeris of the stage times -> constant memory (once for
// up to 128 iterations), Yoshida steps with the cell key, row count and scan record
// of the end state (one kernel), row-start scan, placement into the cell rows, sort
// inside the rows with the gather of the scan records, pair scan.  The population
// itself is never moved.
// Calls of fewer than 125,000 objects, which launches bound, are captured into CUDA
// graphs once they come again: one per (iterations, iteration % k, buffers and sort
// set they begin with, objects, record capacity).
#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include "../../include/ladds_gpu.h"
#include "conjunction.cuh"
#include "cell_sort.cuh"
#include "pair_scan.cuh"
#include "propagate.cuh"
#include "adjoint.cuh"
#include "device_buffers.h"
#include "insert.cuh"
#include "population.h"

using namespace ladds;

namespace {

// c_eph is per device: calls on one device are serialised.
std::mutex g_deviceMutex[64];

// Ephemeris entries of the stage times of the next nSteps iterations
// (<= kMaxEphSteps, one block): also stores the first of them in *iterBase (the
// scans' step index) and advances the iteration counter past them.
template <typename Entry>
__global__ void __launch_bounds__(3 * kMaxEphSteps) k_ephemeris_dev(Entry *__restrict__ out, int nSteps,
                                                                    int64_t *__restrict__ iterPtr,
                                                                    int64_t *__restrict__ iterBase, double t0,
                                                                    double dt, double hc1, double hc2, double jdEpoch,
                                                                    double theta0, uint32_t mask) {
  const int i = threadIdx.x;
  const int64_t iter = *iterPtr;
  __syncthreads();
  if (i == 0) {
    *iterBase = iter;
    *iterPtr = iter + nSteps;
  }
  if (i >= 3 * nSteps) return;
  const int st = i / 3, stage = i % 3;
  const double tn = t0 + (double)(iter + st) * dt;
  double tau = tn + hc1;
  if (stage >= 1) tau += hc2;
  if (stage >= 2) tau += hc2;
  ephemerisEntry(jdEpoch, theta0, tau, mask, out[i]);
}

inline int blocksFor(size_t n, int b) { return (int)((n + (size_t)b - 1) / (size_t)b); }

constexpr uint32_t kMaskFull = LADDS_PROP_ALL;
constexpr uint32_t kMaskDefault =
    LADDS_PROP_KEP | LADDS_PROP_J2 | LADDS_PROP_C22 | LADDS_PROP_S22 | LADDS_PROP_SRP | LADDS_PROP_DRAG;

enum Phase { kPhProp, kPhBucket, kPhRowsort, kPhCandidates, kPhEvaluate };

// ladds_gpu_step_host moves the state in at most this many chunks, each at
// least kHostChunkMin objects (smaller copies cost more than they overlap)
constexpr int kHostChunks = 4;
constexpr size_t kHostChunkMin = (size_t)1 << 17;

// dealing passes that a scan's walk can leave to k_pair_tiles (1024 pair tests each)
constexpr uint32_t kLaterCap = 1u << 17;

// results of a call in pinned host memory: enqueued behind the call's work, so
// that one wait brings them (the words as they lie at dCount, a removal's count,
// and the first records)
constexpr size_t kMailRecords = 256;
struct CallMail {
  unsigned long long words[4];
  ladds_pair recs[kMailRecords];
};

// Everything sized by the population: one allocation, cut up by layoutObjects.
struct ObjectBuffers {
  DevState cur{}, alt{}, alt2{}, snap{};  // the current state, the next two buffers of its ring, the roll-back copy
  uint32_t *keys = nullptr, *arrival = nullptr;  // cell keys and row arrivals of the state to be scanned, slot order
  ScanRec *scanRecs = nullptr;                   // its scan records, slot order
  unsigned long long *sortRec = nullptr;         // (ix << 32 | slot) sort records of the bucket sort
  uint32_t *sortedKeys = nullptr, *perm = nullptr;  // result of the last sort: cell keys, slots
  float4 *posf = nullptr;                 // binary32 positions + rounding bound, cell order
  float4 *velf = nullptr;                 // binary32 velocities + radius of the cell order
  uint32_t *grp = nullptr;                // breakup group of the cell order (parent id, or kNoGroup)
  uint32_t *scratchA = nullptr, *scratchB = nullptr, *scratchC = nullptr;
  uint32_t *denseCells = nullptr, *denseChunk = nullptr;  // dense bin of the pair scan: cells, chunk of each entry
  uint32_t denseCap = 0;
  // second set of the sort's input and results: the propagation and the sort of
  // a step write one set while the sort and the pair scan of the step before
  // still read the other (with the second row tables of the context)
  uint32_t *keysB = nullptr, *arrivalB = nullptr, *sortedKeysB = nullptr, *permB = nullptr, *grpB = nullptr,
           *denseCellsB = nullptr, *denseChunkB = nullptr;
  ScanRec *scanRecsB = nullptr;
  float4 *posfB = nullptr, *velfB = nullptr;
  double *homeX[2] = {};  // x arrays of the buffers that were current and next at allocation
};

// cuts the buffers of `cap` objects out of base (null: only counts); returns the bytes
size_t layoutObjects(ObjectBuffers &o, size_t cap, char *base) {
  size_t at = 0;
  auto take = [&](auto *&p, size_t count) {
    p = base ? reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at) : nullptr;
    at += (count * sizeof(*p) + 255) & ~(size_t)255;
  };
  // x .. vz of a state follow one another at one distance: a copy of all six is
  // one two-dimensional copy
  DevState shared{};
  take(shared.aom, cap);
  take(shared.bc, cap);
  take(shared.radius, cap);
  take(shared.id, cap);
  take(shared.parent, cap);
  take(shared.tag, cap);
  for (DevState *d : {&o.cur, &o.alt, &o.alt2, &o.snap}) {
    *d = shared;
    for (double **q : {&d->x, &d->y, &d->z, &d->vx, &d->vy, &d->vz}) take(*q, cap);
  }
  for (uint32_t **q : {&o.keys, &o.keysB, &o.arrival, &o.arrivalB, &o.scratchA, &o.scratchB, &o.scratchC, &o.perm,
                       &o.permB, &o.sortedKeys, &o.sortedKeysB, &o.grp, &o.grpB})
    take(*q, cap + 1);
  for (float4 **q : {&o.posf, &o.posfB, &o.velf, &o.velfB}) take(*q, cap);
  take(o.scanRecs, cap);
  take(o.scanRecsB, cap);
  take(o.sortRec, cap);
  // every listed cell holds >= kDenseCell objects and adds one entry per kTileChunk of them and part of
  // its staged side (up to 2^kTilePartsLogMax parts, for cells of >= 64 * 4^kTilePartsLogMax objects)
  o.denseCap = (uint32_t)(cap / kDenseCell + cap / kTileChunk * (1u << kTilePartsLogMax) + 1);
  for (uint32_t **q : {&o.denseCells, &o.denseCellsB, &o.denseChunk, &o.denseChunkB}) take(*q, o.denseCap);
  o.homeX[0] = o.cur.x;
  o.homeX[1] = o.alt.x;
  return at;
}

// The cell grid and the row tables that go with it.
struct GridTables {
  GridDesc grid{};
  uint32_t nRows = 0;
  char *tables = nullptr;                 // the allocation behind the row tables
  uint32_t *rowCounts = nullptr;          // objects per row; all zero but between a propagation and its sort
  uint32_t *longRows = nullptr;           // rows with more than 256 objects
  uint32_t *rowStart = nullptr;
  uint16_t *cellOff = nullptr;            // per row: offset of every cell inside the row (cellOffPitch entries)
  uint32_t *rowStartB = nullptr, *rowCountsB = nullptr;  // those of the second set
  uint16_t *cellOffB = nullptr, *cellOffBase = nullptr;
};

}  // namespace

struct ladds_gpu_ctx : ObjectBuffers, GridTables {
  ladds_gpu_config cfg{};
  PropConsts pc{};
  ScanConsts sc{};
  double theta0 = 0;
  int dev = 0;
  cudaStream_t st = nullptr;   // main stream
  cudaStream_t st2 = nullptr;  // pair scans, overlapped with the next propagation
  cudaStream_t st3 = nullptr;  // sorts between a propagation and its scan; device-to-host copies of ladds_gpu_step_host
  cudaEvent_t evProp = nullptr, evSort[2] = {}, evScan[3] = {};  // hand-offs between the streams (evSort, evScan: the last ones)
  cudaEvent_t evPipe[3 * kHostChunks + 1] = {};  // chunk hand-offs of ladds_gpu_step_host
  double *pinStage = nullptr;  // pinned staging of ladds_gpu_step_host for pageable arrays (12 x pinCap)
  size_t pinCap = 0;
  std::vector<ladds_pair> pending;  // records of a ladds_gpu_step_host call whose buffer was too small
  int64_t *dIterBase = nullptr;  // first iteration of the chunk being run (device)
  size_t n = 0, cap = 0;
  char *objects = nullptr;  // the allocation behind the object buffers
  char *words = nullptr;    // the allocation behind the counters and small tables
  CallMail *mail = nullptr;
  uint32_t *longCount = nullptr;          // entries of longRows
  uint32_t *scanWs = nullptr;             // block sums of the exclusive scans
  size_t scanWsWords = 0;
  bool anyParent = false;                 // some object has a parent id: the scan writes and reads grp
  ladds_pair *dPairs = nullptr;
  size_t pairCap = 0;
  unsigned long long *dCount = nullptr;
  uint2 *dCand = nullptr;  // candidate pairs (sorted indices) of the pair scan
  uint2 *dLater = nullptr;  // dealing passes left by the walk (kLaterCap)
  size_t candCap = 0;  // entries of each of the two candidate lists
  unsigned long long *dCandCount = nullptr;  // lengths of the candidate lists of the current scan, dense-bin cursor
  unsigned long long *dCandNeed = nullptr;   // largest candidate count of the call
  unsigned *dStatus = nullptr;
  EphEntry *dEph = nullptr;
  int64_t *dIter = nullptr;
  int64_t hostIter = 0;
  bool orderValid = false;
  // objects that perm has in the order of the last scan (later ones follow in
  // slot order); 0 from before a sort is enqueued until it is known to have run
  size_t orderN = 0;
  bool profiling = false;
  std::vector<std::tuple<int, cudaEvent_t, cudaEvent_t, int>> events;  // phase, start, end, kernels
  std::vector<cudaEvent_t> eventPool;
  ladds_phase_times times{};
  cudaEvent_t callStart = nullptr, callEnd = nullptr;
  using GraphKey = std::tuple<int, int, int, size_t, size_t>;
  std::map<GraphKey, cudaGraphExec_t> graphs;
  std::set<GraphKey> seenChunks;  // chunks that have run once, without a graph
  bool captureAll = false;        // capture chunks at their first sight (an autotuner trial)
  std::string err;
  ladds_object *dObj = nullptr;  // staging of ladds_gpu_functor_pairs (2 x objCap)
  size_t objCap = 0;
  int evalBlocks = 592;     // grid of the candidate-evaluation kernel (4 per SM)
  float cutF = 0.f;         // binary32 pre-filter radius: cutoff * (1 + nearRel), rounded up
  int chunkSteps = kMaxEphSteps;  // iterations per ephemeris chunk / captured graph (autotuned)
  uint32_t *denseCount = nullptr;  // entries of the dense bin
  uint32_t haloStart = 0xffffffffu;  // objects with slot >= haloStart: pair-scan targets only
  // the counters of the second set
  uint32_t *denseCountB = nullptr;
  unsigned long long *dCandCountB = nullptr;
  int sortParity = 0;
  struct Adjoint {          // buffers of the adjoint pair batch (ladds_gpu_adjoint_*)
    size_t nPairs = 0;
    int steps = 0, ck = 0;
    bool forwardDone = false;
    bool whole = false;    // rec holds every step of the forward sweep
    bool ckptDone = false;  // ckpt holds its checkpoints
    double *st = nullptr, *bc = nullptr, *aom = nullptr, *miss = nullptr, *seed = nullptr, *grad = nullptr;
    double *ckpt = nullptr, *rec = nullptr, *off = nullptr;
    int *arg = nullptr;
    EphEntry *eph = nullptr;
    size_t objCap = 0, ckptCap = 0, recCap = 0, ephCap = 0;
  } adj;
};

namespace {

int fail(ladds_gpu_ctx *c, int code, const std::string &msg) {
  if (c) c->err = msg;
  return code;
}

#define CK(call)                                                                                    \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess)                                                                          \
      return fail(c, LADDS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));           \
  } while (0)

// positions and velocities only; a state's six arrays lie at one distance, and one
// copy takes them (10,000 objects, call of two iterations with its roll-back copies:
// 122 us with a copy each, 101 so)
cudaError_t copyDynamic(const DevState &src, const DevState &dst, size_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const size_t from = (size_t)(src.y - src.x) * sizeof(double), to = (size_t)(dst.y - dst.x) * sizeof(double);
  if (copyPitchFits(from) && copyPitchFits(to))
    return cudaMemcpy2DAsync(dst.x, to, src.x, from, n * sizeof(double), 6, cudaMemcpyDeviceToDevice, st);
  const double *sd[] = {src.x, src.y, src.z, src.vx, src.vy, src.vz};
  double *dd[] = {dst.x, dst.y, dst.z, dst.vx, dst.vy, dst.vz};
  for (int k = 0; k < 6; ++k) {
    const cudaError_t e = cudaMemcpyAsync(dd[k], sd[k], n * sizeof(double), cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// the arrays that a context's buffers share
cudaError_t copyShared(const DevState &src, const DevState &dst, size_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const void *sd[] = {src.aom, src.bc, src.radius, src.id, src.parent, src.tag};
  void *dd[] = {dst.aom, dst.bc, dst.radius, dst.id, dst.parent, dst.tag};
  for (int k = 0; k < 6; ++k) {
    cudaError_t e = cudaMemcpyAsync(dd[k], sd[k], n * (k < 5 ? sizeof(double) : sizeof(uint32_t)),
                                    cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t copyState(const DevState &src, const DevState &dst, size_t n, cudaStream_t st) {
  const cudaError_t e = copyDynamic(src, dst, n, st);
  return e != cudaSuccess ? e : copyShared(src, dst, n, st);
}

void dropGraphs(ladds_gpu_ctx *c) {
  for (auto &kv : c->graphs) cudaGraphExecDestroy(kv.second);
  c->graphs.clear();
  c->seenChunks.clear();
}

int ensureCandCapacity(ladds_gpu_ctx *c, size_t need);

// device memory, or null where there is none
void *deviceTake(size_t bytes) {
  void *p = nullptr;
  if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
  cudaGetLastError();
  return nullptr;
}

// device memory for the context.  Where there is none, the records that an
// adjoint's forward sweep has kept for its reverse sweep give way: that sweep then
// takes checkpoints (ladds_gpu_adjoint_backward).
void *contextTake(ladds_gpu_ctx *c, size_t bytes) {
  void *p = deviceTake(bytes);
  if (p || !c->adj.rec) return p;
  cudaFree(c->adj.rec);
  c->adj.rec = nullptr;
  c->adj.recCap = 0;
  c->adj.whole = false;
  return deviceTake(bytes);
}

// block sums of the three-level exclusive scans (objects or rows, whichever is longer)
bool ensureScanWorkspace(ladds_gpu_ctx *c, size_t objects) {
  const size_t scanLen = std::max(objects + 1, (size_t)c->nRows + 1);
  const size_t need = 4 * (scanLen / kScanBlock + 2) + 4 * kScanBlock;
  return growBuffer(c->scanWs, c->scanWsWords, need,
                    [c](size_t bytes) { return contextTake(c, bytes); }, cudaFree);
}

// What a growth carries over: the population of n objects, and the cell order
// and keys of the last scan.
struct Carried {
  void *at;
  size_t bytes;
};
constexpr int kCarried = 14;
void carriedArrays(const ObjectBuffers &o, size_t n, size_t orderN, Carried (&a)[kCarried]) {
  const DevState &s = o.cur;
  void *const p[kCarried] = {s.x,  s.y,      s.z,  s.vx,     s.vy,  s.vz,   s.aom,
                             s.bc, s.radius, s.id, s.parent, s.tag, o.perm, o.sortedKeys};
  for (int k = 0; k < kCarried; ++k) a[k] = {p[k], k < 11 ? n * 8 : k == 11 ? n * 4 : orderN * 4};
}

// Room for `need` objects.  The new block is taken beside the old one, so that a
// growth that fails leaves all as it was.  Where both do not fit the device, the
// population waits in host memory while the old block makes room for the new one
// (the growth by half needs 644 bytes per object of the old capacity on the device instead of
// 1073), or comes back where it was if even that is too little.
int ensureCapacity(ladds_gpu_ctx *c, size_t need) {
  if (need <= c->cap) return LADDS_OK;
  if (need > kMaxObjects) return fail(c, LADDS_ERR_INVALID_ARG, "population exceeds 2^28 - 1 objects");
  size_t newCap = std::max<size_t>({need, c->cap + c->cap / 2, 4096});
  newCap = std::min(newCap, kMaxObjects);
  const std::string noMemory = "device allocation failed: no memory for " + std::to_string(newCap) + " objects";
  if (!ensureScanWorkspace(c, newCap)) return fail(c, LADDS_ERR_ALLOC, noMemory);
  const size_t orderN = std::min(c->orderN, c->n);
  Carried from[kCarried], to[kCarried];
  carriedArrays(*c, c->n, orderN, from);
  ObjectBuffers fresh;
  size_t cap = newCap;
  char *base = static_cast<char *>(contextTake(c, layoutObjects(fresh, cap, nullptr)));
  std::unique_ptr<char[]> aside;
  if (!base && c->objects) {
    size_t total = 0;
    for (const Carried &a : from) total += a.bytes;
    aside.reset(new (std::nothrow) char[total]);
    if (!aside) return fail(c, LADDS_ERR_ALLOC, noMemory);
    char *at = aside.get();
    for (Carried &a : from) {
      if (a.bytes) CK(cudaMemcpyAsync(at, a.at, a.bytes, cudaMemcpyDeviceToHost, c->st));
      a.at = at;
      at += a.bytes;
    }
    CK(cudaStreamSynchronize(c->st));
    dropGraphs(c);
    cudaFree(c->objects);
    c->objects = nullptr;
    base = static_cast<char *>(deviceTake(layoutObjects(fresh, cap, nullptr)));
    if (!base) {
      cap = c->cap;
      base = static_cast<char *>(deviceTake(layoutObjects(fresh, cap, nullptr)));
    }
    if (!base) {  // the memory just given back has gone elsewhere
      static_cast<ObjectBuffers &>(*c) = ObjectBuffers{};
      c->n = c->cap = c->orderN = 0;
      c->orderValid = false;
      return fail(c, LADDS_ERR_ALLOC, noMemory + "; the population could not be put back");
    }
  }
  if (!base) return fail(c, LADDS_ERR_ALLOC, noMemory);
  layoutObjects(fresh, cap, base);
  carriedArrays(fresh, c->n, orderN, to);
  cudaError_t m = cudaSuccess;
  for (int k = 0; k < kCarried && m == cudaSuccess; ++k)
    if (from[k].bytes) m = cudaMemcpyAsync(to[k].at, from[k].at, from[k].bytes, cudaMemcpyDefault, c->st);
  if (m == cudaSuccess) m = cudaStreamSynchronize(c->st);
  if (m != cudaSuccess && !aside) {
    cudaFree(base);
    return fail(c, LADDS_ERR_CUDA, cudaGetErrorString(m));
  }
  if (c->objects) cudaFree(c->objects);
  c->objects = base;
  static_cast<ObjectBuffers &>(*c) = fresh;
  c->orderN = orderN;
  c->cap = cap;
  if (m != cudaSuccess) return fail(c, LADDS_ERR_CUDA, cudaGetErrorString(m));
  if (cap < need) return fail(c, LADDS_ERR_ALLOC, noMemory);
  c->orderValid = false;
  dropGraphs(c);
  // candidates that pass the closest-approach screen: a few per thousand objects at LEO
  // densities; the buffer grows on overflow
  return ensureCandCapacity(c, std::max<size_t>(newCap / 8, (size_t)1 << 16));
}

int ensurePairCapacity(ladds_gpu_ctx *c, size_t need) {
  if (need <= c->pairCap) return LADDS_OK;
  size_t newCap = std::max<size_t>(need + need / 2, 1);
  auto *p = static_cast<ladds_pair *>(contextTake(c, newCap * sizeof(ladds_pair)));
  if (!p) return fail(c, LADDS_ERR_ALLOC, "device allocation failed (pair buffer)");
  if (c->dPairs) cudaFree(c->dPairs);
  c->dPairs = p;
  c->pairCap = newCap;
  dropGraphs(c);
  return LADDS_OK;
}

int ensureCandCapacity(ladds_gpu_ctx *c, size_t need) {
  if (need <= c->candCap) return LADDS_OK;
  size_t newCap = std::max<size_t>(need + need / 2, 1);
  // the screened and the spilled list, newCap entries each
  auto *p = static_cast<uint2 *>(contextTake(c, 2 * newCap * sizeof(uint2)));
  if (!p) return fail(c, LADDS_ERR_ALLOC, "device allocation failed (candidate buffer)");
  if (c->dCand) cudaFree(c->dCand);
  c->dCand = p;
  c->candCap = newCap;
  dropGraphs(c);
  return LADDS_OK;
}

cudaEvent_t takeEvent(ladds_gpu_ctx *c) {
  if (!c->eventPool.empty()) {
    cudaEvent_t e = c->eventPool.back();
    c->eventPool.pop_back();
    return e;
  }
  cudaEvent_t e;
  cudaEventCreate(&e);
  return e;
}

// CUDA events around one phase on the stream that runs it (profiling only)
struct PhaseScope {
  ladds_gpu_ctx *c;
  int phase;
  cudaStream_t s;
  int kernels;
  cudaEvent_t a = nullptr;
  PhaseScope(ladds_gpu_ctx *c_, int ph, cudaStream_t s_, int kernels_ = 1)
      : c(c_), phase(ph), s(s_), kernels(kernels_) {
    if (c->profiling) {
      a = takeEvent(c);
      cudaEventRecord(a, s);
    }
  }
  ~PhaseScope() {
    if (c->profiling) {
      cudaEvent_t b = takeEvent(c);
      cudaEventRecord(b, s);
      c->events.emplace_back(phase, a, b, kernels);
    }
  }
};

void collectTimes(ladds_gpu_ctx *c) {
  for (auto &t : c->events) {
    float ms = 0;
    cudaEventElapsedTime(&ms, std::get<1>(t), std::get<2>(t));
    ladds_phase_times &T = c->times;
    const int k = std::get<3>(t);
    switch (std::get<0>(t)) {
      case kPhProp:
        T.propagateMs += ms;
        T.propagateLaunches += k;
        break;
      case kPhBucket:
        T.bucketMs += ms;
        T.bucketLaunches += k;
        break;
      case kPhRowsort:
        T.rowsortMs += ms;
        T.rowsortLaunches += k;
        break;
      case kPhCandidates:
        T.candidatesMs += ms;
        T.candidatesLaunches += k;
        break;
      default:
        T.evaluateMs += ms;
        T.evaluateLaunches += k;
        break;
    }
    c->eventPool.push_back(std::get<1>(t));
    c->eventPool.push_back(std::get<2>(t));
  }
  c->events.clear();
}

// ----- pipeline pieces (enqueue on the stream they are given, else on c->st; no synchronisation) -----

cudaError_t enqueueEphemeris(ladds_gpu_ctx *c, int nSteps) {
  const int threads = 3 * nSteps, b = (threads + 31) / 32 * 32;
  const bool split = c->cfg.precision == LADDS_PRECISION_SPLIT;
  if (split)
    k_ephemeris_dev<<<1, b, 0, c->st>>>(reinterpret_cast<EphEntryF *>(c->dEph), nSteps, c->dIter, c->dIterBase,
                                          c->cfg.startTime, c->cfg.deltaT, c->pc.hc1, c->pc.hc2, c->cfg.epochJD,
                                          c->theta0, c->pc.mask);
  else
    k_ephemeris_dev<<<1, b, 0, c->st>>>(c->dEph, nSteps, c->dIter, c->dIterBase, c->cfg.startTime, c->cfg.deltaT,
                                          c->pc.hc1, c->pc.hc2, c->cfg.epochJD, c->theta0, c->pc.mask);
  return cudaMemcpyToSymbolAsync(c_eph, c->dEph, (size_t)threads * (split ? sizeof(EphEntryF) : sizeof(EphEntry)), 0,
                                 cudaMemcpyDeviceToDevice, c->st);
}

// the propagation kernel of a component mask: the full and the default set have
// kernels of their own, whose terms are not cut off from one another by branches
// on the mask (a force evaluation is a long chain: 1e6 objects, full set, 30.0 ->
// 27.4 us per step in FP64 and 30.2 -> 26.9 in the split form)
template <typename Pick>
auto forMask(uint32_t mask, Pick pick) {
  if (mask == kMaskFull) return pick(std::integral_constant<uint32_t, kMaskFull>{});
  if (mask == kMaskDefault) return pick(std::integral_constant<uint32_t, kMaskDefault>{});
  return pick(std::integral_constant<uint32_t, 0u>{});
}

ScanInput scanInput(const ladds_gpu_ctx *c) {
  return ScanInput{c->keys, c->rowCounts, c->arrival, c->scanRecs, c->cur.radius};
}

// nSteps steps of the objects [lo, lo + n), from s to `to`, with the scan
// input of the end state if a scan follows.  lo is a multiple of 256, so that
// every array the kernel's bulk copies read starts on a 16-byte boundary.
void launchPropagate(ladds_gpu_ctx *c, DevState s, DevState to, size_t lo, int n, int nSteps, int ephBase,
                     bool scan) {
  ScanInput in = scanInput(c);
  for (DevState *d : {&s, &to}) {
    d->x += lo; d->y += lo; d->z += lo; d->vx += lo; d->vy += lo; d->vz += lo;
    d->aom += lo; d->bc += lo; d->tag += lo;
  }
  in.keys += lo;
  in.arrival += lo;
  in.rec += lo;
  in.radius += lo;
  // three CTAs per SM: the sort and the scan of the iterations before run
  // beside the kernel on streams of their own, and four fit.  Graph step (or its like,
  // launched one by one) in us with two / three / four, full set:
  //   FP64, scan every step: 100,000 objects 33.3 / 32.9 / 32.9, 250,000 54.8 / 53.7 / 55.0,
  //     500,000 97.9 / 99.7 / 100.2, 1e6 175 / 168 / 173
  //   FP64, every fourth: 250,000 19.8 / 18.6 / 18.7, 500,000 32.6 / 31.3 / 35.6, 1e6 62.3 / 57.7 / 57.6
  //   split, scan every step: 500,000 81.1 / 78.3 / 81.5, 1e6 148.9 / 148.4 / 144.2,
  //     2e6 364 / 353 / 355, 8e6 (40 km) 3003 / 2986 / 2978
  //   split, every fourth: 500,000 31.5 / 29.7 / 29.3, 1e6 59.6 / 62.2 / 62.7, 2e6 125 / 123 / 126
  const int sg = std::max(1, std::min(blocksFor((size_t)n, kStageObjects), c->evalBlocks * 3 / 4));
  const bool split = c->cfg.precision == LADDS_PRECISION_SPLIT;
  auto pick = [&](auto mask) {
    constexpr uint32_t M = decltype(mask)::value;
    return split ? (scan ? k_propagate_staged<true, true, M> : k_propagate_staged<true, false, M>)
                 : (scan ? k_propagate_staged<false, true, M> : k_propagate_staged<false, false, M>);
  };
  auto kernel = forMask(c->pc.mask, pick);
  kernel<<<sg, kStageObjects, 0, c->st>>>(s, to, n, nSteps, ephBase, c->pc, c->grid, in, c->dStatus);
}

// nSteps steps, in place (stage ephemerides c_eph[ephBase ...])
void enqueuePropagate(ladds_gpu_ctx *c, int nSteps, int ephBase) {
  if (!c->n) return;
  PhaseScope ps(c, kPhProp, c->st);
  const int b = c->cfg.propagateBlock > 0 ? c->cfg.propagateBlock : 256, g = blocksFor(c->n, b);
  const bool split = c->cfg.precision == LADDS_PRECISION_SPLIT;
  auto kernel = forMask(c->pc.mask, [&](auto mask) {
    constexpr uint32_t M = decltype(mask)::value;
    return split ? k_propagate<true, M> : k_propagate<false, M>;
  });
  kernel<<<g, b, 0, c->st>>>(c->cur, (int)c->n, nSteps, ephBase, c->pc, c->dStatus);
}

// the next buffer of the ring becomes the current state
void rotateStates(ladds_gpu_ctx *c) {
  const DevState old = c->cur;
  c->cur = c->alt;
  c->alt = c->alt2;
  c->alt2 = old;
}
// position in the ring and sort set, as captured graphs have them baked in
int bufferRoles(const ladds_gpu_ctx *c) {
  return (c->cur.x == c->homeX[0] ? 0 : c->cur.x == c->homeX[1] ? 1 : 2) | 4 * c->sortParity;
}

// nSteps steps into the next state buffer, which becomes the current one, with
// the input of the scan that follows them
void enqueuePropagateStaged(ladds_gpu_ctx *c, int nSteps, int ephBase, bool scan) {
  PhaseScope ps(c, kPhProp, c->st);
  launchPropagate(c, c->cur, c->alt, 0, (int)c->n, nSteps, ephBase, scan);
  rotateStates(c);
}

// kernels launched by enqueueExclusiveScan for `count` values
int exclusiveScanKernels(size_t count) {
  const int nb1 = blocksFor(count, kScanBlock);
  if (nb1 == 1) return 1;
  if (nb1 <= kScanBlock) return 2;
  return blocksFor((size_t)nb1, kScanBlock) > 1 ? 5 : 3;
}

// exclusive scan of `count` u32 values (1024-wide block scans; up to 2^20
// values: block scans, then each block adds the sum of the blocks before it;
// beyond: three levels, count <= 2^30); block sums live in c->scanWs
void enqueueExclusiveScan(ladds_gpu_ctx *c, const uint32_t *in, size_t count, uint32_t *out, cudaStream_t s) {
  const int nb1 = blocksFor(count, kScanBlock);
  uint32_t *s1 = c->scanWs, *s1x = s1 + nb1 + 1;
  k_scan_blocks<<<nb1, kScanBlock, 0, s>>>(in, (int)count, out, s1);
  if (nb1 == 1) return;
  if (nb1 <= kScanBlock) {
    k_scan_add_prefix<<<nb1, kScanBlock, 0, s>>>(out, (int)count, s1);
    return;
  }
  const int nb2 = blocksFor((size_t)nb1, kScanBlock);
  uint32_t *s2 = s1x + nb1 + 1;
  k_scan_blocks<<<nb2, kScanBlock, 0, s>>>(s1, nb1, s1x, s2);
  if (nb2 > 1) {
    uint32_t *s2x = s2 + nb2 + 1, *s3 = s2x + nb2 + 1;
    k_scan_blocks<<<1, kScanBlock, 0, s>>>(s2, nb2, s2x, s3);
    k_scan_add<<<nb2, kScanBlock, 0, s>>>(s1x, nb1, s2x);
  }
  k_scan_add<<<nb1, kScanBlock, 0, s>>>(out, (int)count, s1x);
}

// the dense bin of the pair scan: on with the counting row sort and the cell tables
DenseBin denseBin(const ladds_gpu_ctx *c) {
  const bool on = c->cellOff && c->denseCells && (uint32_t)c->grid.n[0] <= (uint32_t)kRowCountMaxNx &&
                  c->grid.reach <= 3;  // k_pair_tiles: one lane per half-shell row (<= 25 rows)
  return DenseBin{on ? c->denseCells : nullptr, c->denseCount, c->denseCap, kDenseCell, c->denseChunk};
}

// called before a scan's input is written: the set that neither the sort nor
// the pair scan before it uses
void swapSortSets(ladds_gpu_ctx *c) {
  std::swap(c->keys, c->keysB);
  std::swap(c->arrival, c->arrivalB);
  std::swap(c->rowCounts, c->rowCountsB);
  std::swap(c->scanRecs, c->scanRecsB);
  std::swap(c->rowStart, c->rowStartB);
  std::swap(c->sortedKeys, c->sortedKeysB);
  std::swap(c->perm, c->permB);
  std::swap(c->posf, c->posfB);
  std::swap(c->velf, c->velfB);
  std::swap(c->grp, c->grpB);
  std::swap(c->cellOff, c->cellOffB);
  std::swap(c->denseCells, c->denseCellsB);
  std::swap(c->denseChunk, c->denseChunkB);
  std::swap(c->denseCount, c->denseCountB);
  std::swap(c->dCandCount, c->dCandCountB);
  c->sortParity ^= 1;
}

// row-start table from the row counts; kernels launched
int enqueueRowScan(ladds_gpu_ctx *c, cudaStream_t s) {
  const size_t count = (size_t)c->nRows + 1;
  const int nb = blocksFor(count, kScanBlock);
  if (nb <= kRowScanBlocks) {
    k_row_scan<<<nb, kScanBlock, 0, s>>>(c->rowCounts, (int)count, c->rowStart);
    return 1;
  }
  enqueueExclusiveScan(c, c->rowCounts, count, c->rowStart, s);
  return exclusiveScanKernels(count);
}

// keys, arrival, rowCounts and scanRecs hold the scan input of the current
// state (writeScanInput) -> row-start table, sortedKeys and perm (order = sort
// by (cell key, slot)) and the scan records in that order.  The placement
// clears what the next sort and scan on this set count in.
void enqueueSort(ladds_gpu_ctx *c, cudaStream_t s) {
  const int n = (int)c->n;
  const uint32_t nx = (uint32_t)c->grid.n[0], nRows = c->nRows;
  {
    PhaseScope ps(c, kPhBucket, s, 2);
    const int k = enqueueRowScan(c, s);
    ps.kernels = 1 + k;
    // blocks for the objects or, on a fine grid with few of them, for the counts that the
    // kernel clears: 10 objects in 2.56e6 rows, iteration 339 us by their one block, 152 so
    const int placeBlocks = std::max(blocksFor(c->n, kBucketThreads),
                                     std::min(blocksFor((size_t)nRows + 1, 4 * kBucketThreads), c->evalBlocks));
    k_bucket_place<<<placeBlocks, kBucketThreads, 0, s>>>(
        c->keys, c->arrival, n, nx, c->rowStart, c->sortRec, c->rowCounts, nRows + 1, c->longCount, c->denseCount,
        c->dCandCount, c->dStatus);
  }
  PhaseScope ps(c, kPhRowsort, s, 2);
  const DenseBin dense = denseBin(c);
  const CellOrderOut out{c->sortedKeys, c->perm, c->scanRecs, c->posf, c->velf,
                         c->anyParent ? c->cur.parent : nullptr, c->grp};
  // Few objects per row: most rows are empty or hold one or two, and a warp per
  // row waits out a chain of shared-memory steps for each.  Graph step by
  // batches / by rows at 62,500 rows: 10,000 objects 16.1 / 22.6 us, 31,000 20.9 /
  // 27.0, 62,000 26.8 / 30.9, 78,000 30.7 / 32.8, 94,000 34.2 / 33.6, 180,000 56 / 49.
  if (nx <= (uint32_t)kRowCountMaxNx && 4 * c->n <= 5 * (size_t)nRows) {
    const int batchBlocks = std::min(blocksFor(((size_t)nRows + kBatchRows - 1) / kBatchRows * 32, kRowSortThreads),
                                     5 * c->evalBlocks / 2);
    k_bucket_sort_batches<<<batchBlocks, kRowSortThreads, 0, s>>>(c->rowStart, nRows, nx, c->sortRec, out,
                                                                  c->longRows, c->longCount, c->cellOff, dense);
  } else if (nx <= (uint32_t)kRowCountMaxNx) {  // counting sort inside the rows
    // one resident wave (10 CTAs of 4 warps per SM); each warp pipelines its rows
    const int rowBlocks = std::min(blocksFor((size_t)nRows * 32, kRowSortThreads), 5 * c->evalBlocks / 2);
    k_bucket_sort_rows<<<rowBlocks, kRowSortThreads, rowSortSmem(nx), s>>>(
        c->rowStart, nRows, nx, c->sortRec, out, c->longRows, c->longCount, c->cellOff, dense);
  } else {
    const int smallBlocks = std::min(blocksFor((size_t)nRows * 32, kBucketThreads), 16 * c->evalBlocks);
    k_bucket_sort_small<<<smallBlocks, kBucketThreads, 0, s>>>(c->rowStart, nRows, nx, c->sortRec, out, c->longRows,
                                                               c->longCount, c->cellOff);
  }
  k_bucket_sort_large<<<c->evalBlocks / 2, kBucketThreads, kLargeRow * 8, s>>>(
      c->rowStart, nx, c->sortRec, out, c->longRows, c->longCount, c->cellOff, dense);
}

// what the scan of the current state reads
inline ScanPack scanPack(const ladds_gpu_ctx *c) { return ScanPack{c->posf, c->velf, c->cur, c->perm}; }

// binary32 pre-filter radius of a cutoff: cutoff * (1 + nearRel), rounded up
// and widened for the test on squares (prefilterPass)
inline float prefilterRadius(double cutoff, double nearRel) {
  return (float)(cutoff * (1.0 + nearRel) * (1.0 + 2e-6));
}

// candidates + evaluation on stream s; records carry *iterPtr + iterOffset
void enqueueScanWith(ladds_gpu_ctx *c, cudaStream_t s, const ScanConsts &scIn, float cutF, const int64_t *iterPtr,
                     int64_t iterOffset) {
  const ScanConsts sc = screenConsts(scIn);
  const DenseBin dense = denseBin(c);
  {
    PhaseScope ps(c, kPhCandidates, s, dense.cells ? 2 : 1);
    const bool buffer = c->cfg.scanScreen == LADDS_SCREEN_BUFFER;
    // the largest separation a record or a near-band flag can have, with room for rounding
    const double reach = std::sqrt(sc.cutoffSq) * (1.0 + sc.nearRel) * (1.0 + 1e-6);
    WalkIn in{c->perm,   c->posf, (int)c->n,     c->sortedKeys, c->rowStart, c->cellOff,
              c->grid,   cutF,    reach * reach, dense.cells ? dense.minCount : 0xffffffffu,
              c->denseCount, {},  0};
    buildHalfShellRows(in.rows, c->grid.reach, c->grid.cellSize, reach * reach);
    // reach 1 and 2 with every row at its full half-width: rows known at compile time
    const int full = c->grid.reach == 1 ? 5 : c->grid.reach == 2 ? 13 : -1;
    bool whole = in.rows.n == full;
    for (int q = 0; q < in.rows.n && whole; ++q) whole = (in.rows.e[q] >> 16) == (uint32_t)c->grid.reach;
    const int r = whole ? c->grid.reach : 0;
    in.groupRows = walkGroup(r);
    // passes are left for later only where k_pair_tiles follows and the rows are in the table
    const bool later = dense.cells && in.rows.n > 0 && in.rows.n <= kLaterGroups * in.groupRows;
    const CandSink out{sc,           c->posf, c->velf, c->dCand, c->dCandCount, (unsigned long long)c->candCap,
                       c->haloStart, c->anyParent ? c->grp : nullptr, later ? c->dLater : nullptr, kLaterCap};
    auto walk = buffer ? (r == 1   ? k_pair_walk<LADDS_SCREEN_BUFFER, 1>
                          : r == 2 ? k_pair_walk<LADDS_SCREEN_BUFFER, 2>
                                   : k_pair_walk<LADDS_SCREEN_BUFFER, 0>)
                       : (r == 1   ? k_pair_walk<LADDS_SCREEN_LISTS, 1>
                          : r == 2 ? k_pair_walk<LADDS_SCREEN_LISTS, 2>
                                   : k_pair_walk<LADDS_SCREEN_LISTS, 0>);
    walk<<<blocksFor(c->n, kScanCta), kScanCta, 0, s>>>(in, out);
    if (dense.cells)  // the dense bin and the passes left by the walk, drawn entry by entry: one resident wave
      (buffer ? k_pair_tiles<LADDS_SCREEN_BUFFER>
              : k_pair_tiles<LADDS_SCREEN_LISTS>)<<<kTileCtasPerSm * c->evalBlocks / 4, kScanCta, 0,
                                                  s>>>(dense.cells, dense.chunk, dense.cap, in, out);
  }
  PhaseScope ps(c, kPhEvaluate, s);
  const int b = c->cfg.scanBlock > 0 ? c->cfg.scanBlock : 256;
  // grid-stride over both candidate lists (their lengths are only known on the device): one resident wave
  const int evalGrid = std::max(1, std::min(blocksFor(2 * c->candCap, b), c->evalBlocks * 256 / b));
  k_pair_eval<<<evalGrid, b, 0, s>>>(scanPack(c), c->dCand, c->dCandCount, (unsigned long long)c->candCap,
                                     c->dCandNeed, sc, iterPtr, iterOffset, c->dPairs, c->dCount,
                                     (unsigned long long)c->pairCap);
}

// Iterations of a chunk that one propagation launch covers: from iteration i
// to the next one that is followed by a scan (or to the chunk's end).
struct StepGroup {
  int len;
  bool scan;
};
StepGroup nextGroup(int64_t itStart, int i, int len, int k) {
  int j = i;
  while (j < len && (itStart + j) % k != 0) ++j;
  return j < len ? StepGroup{j - i + 1, true} : StepGroup{len - i, false};
}

// `len` iterations starting at iteration itStart (len <= kMaxEphSteps): one
// ephemeris kernel + one constant-memory copy for the whole chunk, and one
// propagation launch per scan (the state stays in registers over the steps
// since the scan before).  Three streams hand the scanned iterations on:
// propagation (st), sort (st3), pair scan (st2), so that the scan of an
// iteration runs beside the sort of the next and the propagation of the one
// after it.  The state goes round a ring of three buffers and the sort's input
// and results alternate between two sets, hence, for the i-th scanned iteration:
//   the propagation waits for sort i - 2 (its input set) and scan i - 3 (its
//     state buffer),
//   the sort for its propagation and scan i - 2 (its result set),
//   the scan for its sort.
// Records carry the chunk's first iteration (stored by the ephemeris kernel) + i.
void enqueueChunk(ladds_gpu_ctx *c, int64_t itStart, int len, int k) {
  enqueueEphemeris(c, len);
  if (!c->n) return;
  const bool overlap = !c->profiling;
  const cudaStream_t sSort = overlap ? c->st3 : c->st, sScan = overlap ? c->st2 : c->st;
  int scans = 0;
  for (int i = 0; i < len;) {
    const StepGroup g = nextGroup(itStart, i, len, k);
    if (overlap && scans >= 2) cudaStreamWaitEvent(c->st, c->evSort[scans % 2], 0);
    if (overlap && scans >= 3) cudaStreamWaitEvent(c->st, c->evScan[scans % 3], 0);
    if (g.scan) swapSortSets(c);
    enqueuePropagateStaged(c, g.len, 3 * i, g.scan);
    i += g.len;
    if (!g.scan) break;
    if (overlap) {
      cudaEventRecord(c->evProp, c->st);
      cudaStreamWaitEvent(sSort, c->evProp, 0);
      if (scans >= 2) cudaStreamWaitEvent(sSort, c->evScan[(scans - 2) % 3], 0);
    }
    enqueueSort(c, sSort);
    if (overlap) {
      cudaEventRecord(c->evSort[scans % 2], sSort);
      cudaStreamWaitEvent(sScan, c->evSort[scans % 2], 0);
    }
    ScanConsts sc = c->sc;
    sc.dt = c->cfg.deltaT * (double)k;
    enqueueScanWith(c, sScan, sc, c->cutF, c->dIterBase, i - 1);
    if (overlap) cudaEventRecord(c->evScan[scans % 3], sScan);
    ++scans;
  }
  if (overlap && scans) cudaStreamWaitEvent(c->st, c->evScan[(scans - 1) % 3], 0);
}

// A chunk is captured into a graph where the launches bound its iterations
// (eight kernels of an iteration take about 30 us to launch, and 20 us in a graph
// at 31,000 objects; 1e6 objects take 152.2 us in a graph and 153.3 us launched one
// by one), and only once it is known to come again: capturing 128 iterations
// takes some 10 ms.
constexpr size_t kGraphObjects = 125000;

// host-side effect of replaying a captured chunk: the buffer swaps of its
// propagations and sorts
void replaySwaps(ladds_gpu_ctx *c, int64_t itStart, int len, int k) {
  if (!c->n) return;
  int launches = 0, scans = 0;
  for (int i = 0; i < len;) {
    const StepGroup g = nextGroup(itStart, i, len, k);
    i += g.len;
    ++launches;
    scans += g.scan;
  }
  for (int r = launches % 3; r > 0; --r) rotateStates(c);
  if (scans % 2 == 1) swapSortSets(c);
}

// The buffers of a call's start state are baked into its graphs, and a call leaves
// them one or two places on: three captures of the same chunk (six with the sort
// sets).  Before a call of some length the state goes back to the first buffer
// and the first sort set instead, so that the second call of a loop finds or makes its last
// graph: 31,000 objects, 128 iterations a call: the copy is 10 us of 2.8 ms, a
// capture 13 - 35 ms, which the fourth to the sixth call had each.  Short calls keep
// their roles: their captures are short too.
constexpr int kHomeIterations = 32;

int homeBuffers(ladds_gpu_ctx *c, bool scans) {
  if (c->cur.x != c->homeX[0]) {
    const DevState from = c->cur;
    do rotateStates(c);
    while (c->cur.x != c->homeX[0]);
    CK(copyDynamic(from, c->cur, c->n, c->st));
  }
  // without a scan the call leaves the last scan's cell order, in the set that is current
  if (scans && c->sortParity) swapSortSets(c);
  return LADDS_OK;
}

// whether every chunk of a call has a graph, has run before, or comes twice in
// the call; notes those that come for the first time
bool chunksWorthCapturing(ladds_gpu_ctx *c, int64_t it0, int iterations, int k) {
  const DevState ring0[3] = {c->cur, c->alt, c->alt2};
  const int par0 = c->sortParity;
  bool worth = true;
  std::map<ladds_gpu_ctx::GraphKey, int> times;
  for (int done = 0; done < iterations;) {
    const int len = std::min(iterations - done, c->chunkSteps);
    ++times[std::make_tuple(len, (int)((it0 + done) % k), bufferRoles(c), c->n, c->pairCap)];
    replaySwaps(c, it0 + done, len, k);
    done += len;
  }
  c->cur = ring0[0];
  c->alt = ring0[1];
  c->alt2 = ring0[2];
  if (c->sortParity != par0) swapSortSets(c);
  for (const auto &t : times)
    if (t.second < 2 && !c->graphs.count(t.first) && c->seenChunks.insert(t.first).second) worth = false;
  return worth;
}

// what a status word means
int statusError(ladds_gpu_ctx *c, unsigned status) {
  if (status) CK(cudaMemsetAsync(c->dStatus, 0, sizeof(unsigned), c->st));
  if (status & 4u) return fail(c, LADDS_ERR_DEVICE_CHECK, "a device-side index check failed (sort / gather)");
  if (status & 8u) return fail(c, LADDS_ERR_DEVICE_CHECK, "a bounded device wait ran out (staged propagation)");
  if (status & 1u) return fail(c, LADDS_ERR_NONFINITE, "a position or velocity became NaN/Inf during propagation");
  return LADDS_OK;
}

int syncAndStatus(ladds_gpu_ctx *c) {
  c->mail->words[2] = 0;
  CK(cudaMemcpyAsync(&c->mail->words[2], c->dStatus, sizeof(unsigned), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return statusError(c, (unsigned)(c->mail->words[2] & 0xffffffffull));
}

// The end of a call with scans: the counts, the status and the first records
// come with the call's work, so that one wait brings them; grows the buffers
// that overflowed (*overflow: the scans have to run again).
int syncStatusAndGrow(ladds_gpu_ctx *c, unsigned long long *records, bool *overflow) {
  CK(cudaMemcpyAsync(c->mail->words, c->dCount, 3 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->st));
  CK(cudaMemcpyAsync(c->mail->recs, c->dPairs, std::min(c->pairCap, kMailRecords) * sizeof(ladds_pair),
                     cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  const unsigned long long *w = c->mail->words;  // record count, largest candidate count, status
  const int rc = statusError(c, (unsigned)(w[2] & 0xffffffffull));
  if (rc) return rc;
  *records = w[0];
  *overflow = w[0] > c->pairCap || w[1] > c->candCap;
  if (w[0] > c->pairCap) {
    const int rp = ensurePairCapacity(c, (size_t)w[0]);
    if (rp) return rp;
  }
  if (w[1] > c->candCap) {
    const int rp = ensureCandCapacity(c, (size_t)w[1]);
    if (rp) return rp;
  }
  return LADDS_OK;
}

// the cnt records of the scans that syncStatusAndGrow waited for
cudaError_t fetchRecords(ladds_gpu_ctx *c, size_t cnt, std::vector<ladds_pair> &recs) {
  recs.resize(cnt);
  if (!cnt) return cudaSuccess;
  if (cnt > kMailRecords)
    return cudaMemcpy(recs.data(), c->dPairs, cnt * sizeof(ladds_pair), cudaMemcpyDeviceToHost);
  std::memcpy(recs.data(), c->mail->recs, cnt * sizeof(ladds_pair));
  return cudaSuccess;
}

// up to eight bytes of device memory, after the work enqueued on the stream
int fetchWord(ladds_gpu_ctx *c, const void *device, size_t bytes, unsigned long long *word) {
  c->mail->words[3] = 0;
  CK(cudaMemcpyAsync(&c->mail->words[3], device, bytes, cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  *word = c->mail->words[3];
  return LADDS_OK;
}
int fetchCount(ladds_gpu_ctx *c, const unsigned *device, unsigned *count) {
  unsigned long long w = 0;
  const int rc = fetchWord(c, device, sizeof(unsigned), &w);
  *count = (unsigned)w;
  return rc;
}

bool pairLess(const ladds_pair &a, const ladds_pair &b) {
  if (a.step != b.step) return a.step < b.step;
  if (a.idA != b.idA) return a.idA < b.idA;
  if (a.idB != b.idB) return a.idB < b.idB;
  if (a.slotA != b.slotA) return a.slotA < b.slotA;
  return a.slotB < b.slotB;
}

int validateArrays(ladds_gpu_ctx *c, size_t n, const double *const *arrs, int nArr, const int8_t *activity) {
  for (int a = 0; a < nArr; ++a)
    if (n && !arrs[a]) return fail(c, LADDS_ERR_INVALID_ARG, "null array pointer");
  for (int a = 0; a < 6; ++a)
    for (size_t i = 0; i < n; ++i)
      if (!std::isfinite(arrs[a][i])) return fail(c, LADDS_ERR_INVALID_ARG, "non-finite position or velocity");
  if (activity)
    for (size_t i = 0; i < n; ++i)
      if (activity[i] < 0 || activity[i] > 2) return fail(c, LADDS_ERR_INVALID_ARG, "activity state out of range");
  return LADDS_OK;
}

int writeArrays(ladds_gpu_ctx *c, size_t offset, size_t n, const double *x, const double *y, const double *z,
                const double *vx, const double *vy, const double *vz, const double *radius, const double *aom,
                const double *bcInv, const uint64_t *id, const uint64_t *parentId, const int8_t *activity) {
  if (!n) return LADDS_OK;
  const double *src[] = {x, y, z, vx, vy, vz, aom, bcInv, radius};
  double *dst[] = {c->cur.x, c->cur.y, c->cur.z, c->cur.vx, c->cur.vy, c->cur.vz, c->cur.aom, c->cur.bc,
                   c->cur.radius};
  for (int k = 0; k < 9; ++k)
    CK(cudaMemcpyAsync(dst[k] + offset, src[k], n * sizeof(double), cudaMemcpyHostToDevice, c->st));
  CK(cudaMemcpyAsync(c->cur.id + offset, id, n * sizeof(uint64_t), cudaMemcpyHostToDevice, c->st));
  std::vector<uint64_t> par;
  if (!parentId) par.assign(n, UINT64_MAX);
  for (size_t i = 0; i < n && parentId && !c->anyParent; ++i) c->anyParent = parentId[i] != UINT64_MAX;
  CK(cudaMemcpyAsync(c->cur.parent + offset, parentId ? parentId : par.data(), n * sizeof(uint64_t),
                     cudaMemcpyHostToDevice, c->st));
  std::vector<uint32_t> tags(n);
  for (size_t i = 0; i < n; ++i) tags[i] = makeTag((uint32_t)(offset + i), activity ? activity[i] : 0, false);
  CK(cudaMemcpyAsync(c->cur.tag + offset, tags.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, c->st));
  CK(cudaStreamSynchronize(c->st));
  return LADDS_OK;
}

int buildGrid(ladds_gpu_ctx *c) {
  const ladds_gpu_config &f = c->cfg;
  // default edge: just above the cutoff, so that the neighbour reach is one cell
  double cell = f.cellSize > 0 ? f.cellSize : f.cutoff * (1.0 + 1e-6);
  const double minCell = std::max(f.cutoff * 1e-3, 1e-9);
  if (!(cell > minCell)) cell = minCell;
  for (int d = 0; d < 3; ++d)
    if (!(f.boxMax[d] > f.boxMin[d]) || !std::isfinite(f.boxMax[d] - f.boxMin[d]))
      return fail(c, LADDS_ERR_INVALID_ARG, "boxMax must exceed boxMin");
  GridDesc g{};
  uint64_t total = 0;
  // coarsen until the keys fit 32 bits and no axis exceeds 65535 cells
  for (;;) {
    g.cellSize = cell;
    g.invCell = 1.0 / cell;
    total = 1;
    bool ok = true;
    for (int d = 0; d < 3; ++d) {
      g.boxMin[d] = f.boxMin[d];
      double cells = std::ceil((f.boxMax[d] - f.boxMin[d]) * g.invCell);
      if (!(cells >= 1.0)) cells = 1.0;
      if (cells > 65535.0) ok = false;
      g.n[d] = (int32_t)std::min(cells, 65535.0);
      total *= (uint64_t)g.n[d];
    }
    if (ok && total <= (1ull << 32)) break;
    cell *= 1.25;
  }
  int32_t r = (int32_t)std::ceil(f.cutoff * (1.0 + 1e-9) * g.invCell);
  if (r < 1) r = 1;
  while ((double)r * cell < f.cutoff * (1.0 + 1e-9)) ++r;
  g.reach = r;
  uint32_t bits = 0;
  while (bits < 32 && ((total - 1) >> bits) != 0) ++bits;
  g.keyBits = bits;
  c->grid = g;
  c->nRows = (uint32_t)((uint64_t)g.n[1] * (uint64_t)g.n[2]);
  return LADDS_OK;
}

void freeGridBuffers(ladds_gpu_ctx *c) {
  if (c->tables) cudaFree(c->tables);
  if (c->cellOffBase) cudaFree(c->cellOffBase);
  c->tables = nullptr;
  c->cellOffBase = nullptr;
  c->rowStart = c->rowStartB = c->rowCounts = c->rowCountsB = c->longRows = nullptr;
  c->cellOff = c->cellOffB = nullptr;
}

// the row counts of both sets start at zero (every sort leaves them so)
cudaError_t clearRowCounts(ladds_gpu_ctx *c) {
  const size_t bytes = ((size_t)c->nRows + 1) * sizeof(uint32_t);
  const cudaError_t e = cudaMemsetAsync(c->rowCounts, 0, bytes, c->st);
  return e == cudaSuccess ? cudaMemsetAsync(c->rowCountsB, 0, bytes, c->st) : e;
}

// row tables of c->grid; the two cell-offset tables when each fits 512 MiB (250^3 cells: 31 MB)
int allocGridBuffers(ladds_gpu_ctx *c) {
  const size_t row = (((size_t)c->nRows + 1) * sizeof(uint32_t) + 255) & ~(size_t)255;
  if (cudaMalloc(&c->tables, 5 * row) != cudaSuccess) {
    cudaGetLastError();
    c->tables = nullptr;
    return fail(c, LADDS_ERR_ALLOC, "device allocation of the cell-row tables failed");
  }
  uint32_t **t[] = {&c->rowStart, &c->rowStartB, &c->rowCounts, &c->rowCountsB, &c->longRows};
  for (int k = 0; k < 5; ++k) *t[k] = reinterpret_cast<uint32_t *>(c->tables + k * row);
  if (clearRowCounts(c) != cudaSuccess) {
    cudaGetLastError();
    freeGridBuffers(c);
    return fail(c, LADDS_ERR_CUDA, "the cell-row tables could not be cleared");
  }
  const size_t cells = (size_t)c->nRows * cellOffPitch((uint32_t)c->grid.n[0]);
  if (cells * sizeof(uint16_t) <= ((size_t)1 << 29)) {
    if (cudaMalloc(&c->cellOffBase, 2 * cells * sizeof(uint16_t)) == cudaSuccess) {
      c->cellOff = c->cellOffBase;
      c->cellOffB = c->cellOffBase + cells;
    } else {
      cudaGetLastError();
      c->cellOffBase = nullptr;  // the scan then searches the sorted keys
    }
  }
  return LADDS_OK;
}

// the counters and small tables of a context: one allocation, zeroed
cudaError_t allocWords(ladds_gpu_ctx *c) {
  constexpr size_t line = 256;
  const size_t later = kLaterCap * sizeof(uint2), eph = 3 * kMaxEphSteps * sizeof(EphEntry);
  cudaError_t e = cudaMalloc(&c->words, 8 * line + later + eph + kAtmFine * sizeof(double2));
  if (e != cudaSuccess) {
    c->words = nullptr;
    return e;
  }
  auto at = [&](size_t k) { return reinterpret_cast<unsigned long long *>(c->words + k * line); };
  // record count, largest candidate count and status side by side: one read after a call
  c->dCount = at(0);
  c->dCandNeed = c->dCount + 1;
  c->dStatus = reinterpret_cast<unsigned *>(c->dCount + 2);
  c->dCandCount = at(1);
  c->dCandCountB = at(2);
  c->dIter = reinterpret_cast<int64_t *>(at(3));
  c->dIterBase = c->dIter + 1;
  c->longCount = reinterpret_cast<uint32_t *>(at(4));
  c->denseCount = reinterpret_cast<uint32_t *>(at(5));
  c->denseCountB = reinterpret_cast<uint32_t *>(at(6));
  c->dLater = reinterpret_cast<uint2 *>(at(8));
  c->dEph = reinterpret_cast<EphEntry *>(c->words + 8 * line + later);
  auto *fineT = reinterpret_cast<double2 *>(c->words + 8 * line + later + eph);
  k_atm_table<<<blocksFor(kAtmFine, 256), 256, 0, c->st>>>(fineT);
  c->pc.atm = fineT;
  e = cudaGetLastError();
  return e != cudaSuccess ? e : cudaMemsetAsync(c->words, 0, 8 * line, c->st);
}

constexpr size_t kHostCopyBlock = (size_t)1 << 17;  // doubles per task of the staging copies

bool isPinned(const void *p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// dst[a][lo, lo + len) = src[a][lo, lo + len) for the arrays with use[a], on all host threads
void hostCopy(double *const dst[6], const double *const src[6], const bool use[6], size_t lo, size_t len) {
  const long per = (long)((len + kHostCopyBlock - 1) / kHostCopyBlock);
  // few objects: waking all threads costs more than the copies (a host-owned
  // iteration of 10,000 objects: 128 us with three threads, 147 with one or all)
  const int threads = len <= kHostCopyBlock / 4 ? std::min(3, omp_get_max_threads()) : omp_get_max_threads();
#pragma omp parallel for schedule(static) num_threads(threads)
  for (long t = 0; t < 6 * per; ++t) {
    const int a = (int)(t / per);
    if (!use[a]) continue;
    const size_t b = lo + (size_t)(t % per) * kHostCopyBlock, e = std::min(b + kHostCopyBlock, lo + len);
    std::memcpy(dst[a] + b, src[a] + b, (e - b) * sizeof(double));
  }
}

// six arrays, elements [lo, lo + len): one two-dimensional copy where both
// sides hold them at one distance that such a copy can take, else a copy each
cudaError_t copySix(double *const dst[6], const double *const src[6], size_t lo, size_t len, bool together,
                    size_t srcStride, size_t dstStride, cudaMemcpyKind kind, cudaStream_t st) {
  if (together && copyPitchFits(srcStride * sizeof(double)) && copyPitchFits(dstStride * sizeof(double)))
    return cudaMemcpy2DAsync(dst[0] + lo, dstStride * sizeof(double), src[0] + lo, srcStride * sizeof(double),
                             len * sizeof(double), 6, kind, st);
  for (int a = 0; a < 6; ++a) {
    const cudaError_t e = cudaMemcpyAsync(dst[a] + lo, src[a] + lo, len * sizeof(double), kind, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// dst[0, n) = src[0, n) on all host threads
void hostCopyOne(double *dst, const double *src, size_t n) {
  const double *const s6[6] = {src, nullptr, nullptr, nullptr, nullptr, nullptr};
  double *const d6[6] = {dst, nullptr, nullptr, nullptr, nullptr, nullptr};
  const bool use[6] = {true, false, false, false, false, false};
  hostCopy(d6, s6, use, 0, n);
}

// the context's pinned staging buffer for pageable host arrays: 12 arrays of
// at least n doubles (six in, six out); false if no pinned memory is to be had
// (the CUDA driver then stages the copies itself)
bool ensurePinStage(ladds_gpu_ctx *c, size_t n) {
  if (c->pinStage && c->pinCap >= n) return true;
  if (c->pinStage) cudaFreeHost(c->pinStage);
  c->pinStage = nullptr;
  c->pinCap = 0;
  if (cudaHostAlloc(&c->pinStage, 12 * n * sizeof(double), cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError();
    c->pinStage = nullptr;
    return false;
  }
  c->pinCap = n;
  return true;
}
}  // namespace

extern "C" {

int ladds_gpu_abi_version(void) { return LADDS_GPU_ABI_VERSION; }

void ladds_gpu_config_default(ladds_gpu_config *f) {
  if (!f) return;
  std::memset(f, 0, sizeof(*f));
  f->deltaT = 10.0;
  f->componentMask = kMaskDefault;
  f->epochJD = 2459580.5;  // 2022-01-01 00:00 UTC (cfg/default_cfg.yaml:9)
  f->startTime = 0.0;
  f->cutoff = 80.0;
  f->collisionDistanceFactor = 1.0;
  f->minDetectionRadius = 0.05;
  f->evasionCutoff = 0.1;
  f->conjunctionThreshold = 0.1;
  f->nearThresholdRel = 1e-9;
  f->precision = LADDS_PRECISION_FP64;
  f->timestepsPerCollisionDetection = 1;
  f->cellSize = 0.0;
  for (int d = 0; d < 3; ++d) {
    f->boxMin[d] = -10000.0;
    f->boxMax[d] = 10000.0;
  }
  f->device = 0;
  f->propagateBlock = 256;
  f->scanBlock = 256;
  f->useGraphs = 1;
  f->pairCapacity = 0;
  f->scanScreen = LADDS_SCREEN_LISTS;
  f->walkForm = LADDS_WALK_AUTO;
}

const char *ladds_gpu_last_error(const ladds_gpu_ctx *c) { return c ? c->err.c_str() : "null context"; }

int ladds_gpu_create(const ladds_gpu_config *f, ladds_gpu_ctx **out) {
  if (!f || !out) return LADDS_ERR_INVALID_ARG;
  *out = nullptr;
  if (!(f->deltaT != 0.0 && std::isfinite(f->deltaT)) || !(f->cutoff > 0) || f->timestepsPerCollisionDetection < 1 ||
      (f->precision != LADDS_PRECISION_FP64 && f->precision != LADDS_PRECISION_SPLIT) ||
      (f->componentMask & ~LADDS_PROP_ALL) || !(f->nearThresholdRel >= 0))
    return LADDS_ERR_INVALID_ARG;
  if (f->propagateBlock < 0 || f->propagateBlock > 256 || (f->propagateBlock % 32) || f->scanBlock < 0 ||
      f->scanBlock > 256 || (f->scanBlock % 32) ||
      (f->scanScreen != LADDS_SCREEN_LISTS && f->scanScreen != LADDS_SCREEN_BUFFER) ||
      (f->walkForm != LADDS_WALK_AUTO && f->walkForm != LADDS_WALK_GROUPED && f->walkForm != LADDS_WALK_ROWS))
    return LADDS_ERR_INVALID_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
    cudaGetLastError();
    return LADDS_ERR_NO_DEVICE;
  }
  if (f->device < 0 || f->device >= ndev) return LADDS_ERR_NO_DEVICE;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, f->device) != cudaSuccess || prop.major < 10) return LADDS_ERR_NO_DEVICE;
  ladds_gpu_ctx *c = new ladds_gpu_ctx();
  c->cfg = *f;
  c->dev = f->device;
  int rc = buildGrid(c);
  if (rc) {
    delete c;
    return rc;
  }
  const double dt = f->deltaT;
  c->pc.hc1 = kYoshidaC1 * dt;
  c->pc.hc2 = kYoshidaC2 * dt;
  c->pc.hd1 = kYoshidaD1 * dt;
  c->pc.hd2 = kYoshidaD2 * dt;
  c->pc.mask = f->componentMask;
  c->sc.cutoffSq = f->cutoff * f->cutoff;
  c->sc.dt = dt;
  c->sc.factor = f->collisionDistanceFactor / 1000.;
  c->sc.minDetectionRadius = f->minDetectionRadius;
  c->sc.evasionSq = f->evasionCutoff * f->evasionCutoff;
  c->sc.conjSq = f->conjunctionThreshold * f->conjunctionThreshold;
  c->sc.nearRel = f->nearThresholdRel;
  c->cutF = prefilterRadius(f->cutoff, f->nearThresholdRel);
  c->theta0 = gmstIAU1982(f->epochJD);
  if (cudaSetDevice(c->dev) != cudaSuccess || cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess ||
      allocGridBuffers(c) != LADDS_OK || allocWords(c) != cudaSuccess ||
      cudaHostAlloc(&c->mail, sizeof(CallMail), cudaHostAllocDefault) != cudaSuccess ||
      cudaStreamCreateWithFlags(&c->st2, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&c->st3, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    ladds_gpu_destroy(c);
    return LADDS_ERR_ALLOC;
  }
  cudaEventCreate(&c->callStart);
  cudaEventCreate(&c->callEnd);
  cudaEventCreateWithFlags(&c->evProp, cudaEventDisableTiming);
  for (auto &e : c->evSort) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  for (auto &e : c->evScan) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  for (auto &e : c->evPipe) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  c->evalBlocks = 4 * std::max(prop.multiProcessorCount, 1);
  rc = ensurePairCapacity(c, f->pairCapacity ? (size_t)f->pairCapacity : (size_t)1 << 16);
  if (!rc) rc = ensureCandCapacity(c, (size_t)1 << 16);
  if (rc) {
    ladds_gpu_destroy(c);
    return rc;
  }
  if (cudaDeviceSynchronize() != cudaSuccess) {
    cudaGetLastError();
    ladds_gpu_destroy(c);
    return LADDS_ERR_CUDA;
  }
  *out = c;
  return LADDS_OK;
}

int ladds_gpu_destroy(ladds_gpu_ctx *c) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  cudaSetDevice(c->dev);
  if (c->st) cudaStreamSynchronize(c->st);
  dropGraphs(c);
  freeGridBuffers(c);
  void *ptrs[] = {c->objects,  c->words,    c->scanWs,  c->dPairs,   c->dCand,   c->dObj,
                  c->adj.st,   c->adj.bc,   c->adj.aom, c->adj.miss, c->adj.seed, c->adj.grad, c->adj.ckpt,
                  c->adj.rec,  c->adj.off,  c->adj.arg, c->adj.eph};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  for (auto &t : c->events) {
    cudaEventDestroy(std::get<1>(t));
    cudaEventDestroy(std::get<2>(t));
  }
  for (auto e : c->eventPool) cudaEventDestroy(e);
  if (c->callStart) cudaEventDestroy(c->callStart);
  if (c->callEnd) cudaEventDestroy(c->callEnd);
  if (c->evProp) cudaEventDestroy(c->evProp);
  for (auto e : c->evSort)
    if (e) cudaEventDestroy(e);
  for (auto e : c->evScan)
    if (e) cudaEventDestroy(e);
  for (auto e : c->evPipe)
    if (e) cudaEventDestroy(e);
  if (c->pinStage) cudaFreeHost(c->pinStage);
  if (c->mail) cudaFreeHost(c->mail);
  if (c->st3) cudaStreamDestroy(c->st3);
  if (c->st2) cudaStreamDestroy(c->st2);
  if (c->st) cudaStreamDestroy(c->st);
  delete c;
  return LADDS_OK;
}

int ladds_gpu_upload(ladds_gpu_ctx *c, size_t n, const double *x, const double *y, const double *z,
                     const double *vx, const double *vy, const double *vz, const double *radius, const double *aom,
                     const double *bcInv, const uint64_t *id, const uint64_t *parentId, const int8_t *activity) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  const double *arrs[] = {x, y, z, vx, vy, vz, radius, aom, bcInv};
  int rc = validateArrays(c, n, arrs, 9, activity);
  if (rc) return rc;
  if (n && !id) return fail(c, LADDS_ERR_INVALID_ARG, "null id array");
  CK(cudaSetDevice(c->dev));
  rc = ensureCapacity(c, n);
  if (rc) return rc;
  c->n = 0;
  c->orderN = 0;
  c->anyParent = false;
  rc = writeArrays(c, 0, n, x, y, z, vx, vy, vz, radius, aom, bcInv, id, parentId, activity);
  if (rc) return rc;
  c->n = n;
  c->orderValid = false;
  dropGraphs(c);
  return LADDS_OK;
}

int ladds_gpu_append(ladds_gpu_ctx *c, size_t n, const double *x, const double *y, const double *z,
                     const double *vx, const double *vy, const double *vz, const double *radius, const double *aom,
                     const double *bcInv, const uint64_t *id, const uint64_t *parentId, const int8_t *activity) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  const double *arrs[] = {x, y, z, vx, vy, vz, radius, aom, bcInv};
  int rc = validateArrays(c, n, arrs, 9, activity);
  if (rc) return rc;
  if (n && !id) return fail(c, LADDS_ERR_INVALID_ARG, "null id array");
  if (!n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  rc = ensureCapacity(c, c->n + n);
  if (rc) return rc;
  rc = writeArrays(c, c->n, n, x, y, z, vx, vy, vz, radius, aom, bcInv, id, parentId, activity);
  if (rc) return rc;
  c->n += n;
  c->orderValid = false;
  dropGraphs(c);
  return LADDS_OK;
}

int ladds_gpu_reserve(ladds_gpu_ctx *c, size_t capacity) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (capacity <= c->cap) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  return ensureCapacity(c, capacity);
}

int ladds_gpu_checked_insert(ladds_gpu_ctx *c, size_t n, const double *x, const double *y, const double *z,
                             const double *vx, const double *vy, const double *vz, const double *radius,
                             const double *aom, const double *bcInv, const uint64_t *id, const uint64_t *parentId,
                             const int8_t *activity, double constellationCutoff, uint8_t *delayed,
                             size_t *nInserted) {
  if (!c || (n && (!x || !y || !z || !id || !delayed)) || !(constellationCutoff >= 0.0))
    return fail(c, LADDS_ERR_INVALID_ARG, "checked_insert: bad argument");
  if (nInserted) *nInserted = 0;
  if (!n) return LADDS_OK;
  const double cc = constellationCutoff, c2 = cc * cc;
  std::vector<uint8_t> blocked(n, 0);
  {
    std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
    CK(cudaSetDevice(c->dev));
    if (c->n) {
      double *dp = nullptr;
      uint8_t *db = nullptr;
      if (cudaMalloc(&dp, 3 * n * sizeof(double)) != cudaSuccess || cudaMalloc(&db, n) != cudaSuccess) {
        cudaGetLastError();
        if (dp) cudaFree(dp);
        return fail(c, LADDS_ERR_ALLOC, "checked_insert: staging allocation failed");
      }
      cudaError_t e = cudaMemcpyAsync(dp, x, n * sizeof(double), cudaMemcpyHostToDevice, c->st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dp + n, y, n * sizeof(double), cudaMemcpyHostToDevice, c->st);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dp + 2 * n, z, n * sizeof(double), cudaMemcpyHostToDevice, c->st);
      if (e == cudaSuccess) {
        k_insert_blocked<<<blocksFor(n * 32, 128), 128, 0, c->st>>>(c->cur, (int)c->n, dp, dp + n, dp + 2 * n,
                                                                     (int)n, cc, c2, db);
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = cudaMemcpyAsync(blocked.data(), db, n, cudaMemcpyDeviceToHost, c->st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
      cudaFree(dp);
      cudaFree(db);
      if (e != cudaSuccess) return fail(c, LADDS_ERR_CUDA, std::string("checked_insert: ") + cudaGetErrorString(e));
    }
  }
  // satellites of the batch, in order, against the ones accepted before them
  std::vector<size_t> acc;
  for (size_t i = 0; i < n; ++i) {
    bool hit = blocked[i] != 0;
    const double p[3] = {x[i], y[i], z[i]};
    for (size_t q = 0; q < acc.size() && !hit; ++q) {
      const double o[3] = {x[acc[q]], y[acc[q]], z[acc[q]]};
      hit = insertBlocks(p, o, cc, c2);
    }
    delayed[i] = hit ? 1 : 0;
    if (!hit) acc.push_back(i);
  }
  if (acc.empty()) return LADDS_OK;
  const size_t m = acc.size();
  std::vector<double> d[9];
  const double *src[9] = {x, y, z, vx, vy, vz, radius, aom, bcInv};
  for (int k = 0; k < 9; ++k) {
    d[k].resize(m);
    for (size_t q = 0; q < m; ++q) d[k][q] = src[k] ? src[k][acc[q]] : 0.0;
  }
  std::vector<uint64_t> ids(m), parents(m);
  std::vector<int8_t> acts(m);
  for (size_t q = 0; q < m; ++q) {
    ids[q] = id[acc[q]];
    parents[q] = parentId ? parentId[acc[q]] : UINT64_MAX;
    acts[q] = activity ? activity[acc[q]] : (int8_t)LADDS_PASSIVE;
  }
  const int rc = ladds_gpu_append(c, m, d[0].data(), d[1].data(), d[2].data(), d[3].data(), d[4].data(),
                                  d[5].data(), d[6].data(), d[7].data(), d[8].data(), ids.data(), parents.data(),
                                  acts.data());
  if (!rc && nInserted) *nInserted = m;
  return rc;
}

int ladds_gpu_get_objects(ladds_gpu_ctx *c, const uint32_t *slots, size_t m, ladds_state_record *out) {
  if (!c || (m && (!slots || !out))) return fail(c, LADDS_ERR_INVALID_ARG, "get_objects: bad argument");
  if (!m) return LADDS_OK;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  for (size_t q = 0; q < m; ++q)
    if (slots[q] >= c->n) return fail(c, LADDS_ERR_INVALID_ARG, "get_objects: no object with slot " + std::to_string(slots[q]));
  CK(cudaSetDevice(c->dev));
  uint32_t *dWant = nullptr;
  ladds_state_record *dRec = nullptr;
  if (cudaMalloc(&dWant, m * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&dRec, m * sizeof(ladds_state_record)) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(dWant);
    return fail(c, LADDS_ERR_ALLOC, "get_objects: staging allocation failed");
  }
  cudaError_t e = cudaMemcpyAsync(dWant, slots, m * sizeof(uint32_t), cudaMemcpyHostToDevice, c->st);
  if (e == cudaSuccess) k_gather_records<<<blocksFor(m, 128), 128, 0, c->st>>>(c->cur, dWant, (int)m, dRec);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out, dRec, m * sizeof(ladds_state_record), cudaMemcpyDeviceToHost, c->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
  cudaFree(dWant);
  cudaFree(dRec);
  if (e != cudaSuccess) return fail(c, LADDS_ERR_CUDA, std::string("get_objects: ") + cudaGetErrorString(e));
  return LADDS_OK;
}

int ladds_gpu_download(ladds_gpu_ctx *c, size_t cap, size_t *nOut, double *x, double *y, double *z, double *vx,
                       double *vy, double *vz, double *radius, double *aom, double *bcInv, uint64_t *id,
                       uint64_t *parentId, int8_t *activity) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (nOut) *nOut = c->n;
  if (cap < c->n) return fail(c, LADDS_ERR_CAPACITY, "download buffer smaller than the population");
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  const double *src[] = {c->cur.x,  c->cur.y,   c->cur.z,  c->cur.vx,    c->cur.vy,
                         c->cur.vz, c->cur.aom, c->cur.bc, c->cur.radius};
  double *dst[] = {x, y, z, vx, vy, vz, aom, bcInv, radius};
  for (int k = 0; k < 9; ++k)
    if (dst[k]) CK(cudaMemcpyAsync(dst[k], src[k], c->n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
  if (id) CK(cudaMemcpyAsync(id, c->cur.id, c->n * sizeof(uint64_t), cudaMemcpyDeviceToHost, c->st));
  if (parentId)
    CK(cudaMemcpyAsync(parentId, c->cur.parent, c->n * sizeof(uint64_t), cudaMemcpyDeviceToHost, c->st));
  if (activity) {
    int8_t *act = reinterpret_cast<int8_t *>(c->scratchA);
    k_activity<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur.tag, (int)c->n, act);
    CK(cudaMemcpyAsync(activity, act, c->n, cudaMemcpyDeviceToHost, c->st));
  }
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

int ladds_gpu_set_state(ladds_gpu_ctx *c, size_t n, const double *x, const double *y, const double *z,
                        const double *vx, const double *vy, const double *vz) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (n != c->n) return fail(c, LADDS_ERR_INVALID_ARG, "set_state: n differs from the population size");
  const double *src[] = {x, y, z, vx, vy, vz};
  for (int k = 0; k < 6; ++k)
    if (n && !src[k]) return fail(c, LADDS_ERR_INVALID_ARG, "null array pointer");
  if (!n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  double *dst[] = {c->cur.x, c->cur.y, c->cur.z, c->cur.vx, c->cur.vy, c->cur.vz};
  // pageable arrays go through the context's pinned staging, copied on all host
  // threads while the previous array crosses PCIe
  bool pinned[6], staged = false;
  for (int k = 0; k < 6; ++k) {
    pinned[k] = isPinned(src[k]);
    staged |= !pinned[k];
  }
  if (staged && !ensurePinStage(c, n))
    for (bool &p : pinned) p = true;  // no pinned memory to spare: the driver stages them
  for (int k = 0; k < 6; ++k) {
    const double *from = src[k];
    if (!pinned[k]) {
      double *pin = c->pinStage + (size_t)k * c->pinCap;
      hostCopyOne(pin, src[k], n);
      from = pin;
    }
    CK(cudaMemcpyAsync(dst[k], from, n * sizeof(double), cudaMemcpyHostToDevice, c->st));
  }
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

int ladds_gpu_get_state(ladds_gpu_ctx *c, size_t n, double *x, double *y, double *z, double *vx, double *vy,
                        double *vz) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (n < c->n) return fail(c, LADDS_ERR_CAPACITY, "get_state: buffer smaller than the population");
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  const double *src[] = {c->cur.x, c->cur.y, c->cur.z, c->cur.vx, c->cur.vy, c->cur.vz};
  double *dst[] = {x, y, z, vx, vy, vz};
  // pageable arrays come back through the context's pinned staging: each
  // array leaves the pinned buffer on all host threads while the next crosses PCIe
  bool pinned[6], staged = false;
  for (int k = 0; k < 6; ++k) {
    pinned[k] = !dst[k] || isPinned(dst[k]);
    staged |= !pinned[k];
  }
  if (staged && !ensurePinStage(c, c->n))
    for (bool &p : pinned) p = true;  // no pinned memory to spare: the driver stages them
  for (int k = 0; k < 6; ++k) {
    if (!dst[k]) continue;
    double *to = pinned[k] ? dst[k] : c->pinStage + (size_t)(6 + k) * c->pinCap;
    CK(cudaMemcpyAsync(to, src[k], c->n * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    CK(cudaEventRecord(c->evPipe[k], c->st));
  }
  for (int k = 0; k < 6; ++k) {
    if (!dst[k] || pinned[k]) continue;
    CK(cudaEventSynchronize(c->evPipe[k]));
    hostCopyOne(dst[k], c->pinStage + (size_t)(6 + k) * c->pinCap, c->n);
  }
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

int ladds_gpu_size(const ladds_gpu_ctx *c, size_t *n) {
  if (!c || !n) return LADDS_ERR_INVALID_ARG;
  *n = c->n;
  return LADDS_OK;
}

int ladds_gpu_iteration(const ladds_gpu_ctx *c, int64_t *it) {
  if (!c || !it) return LADDS_ERR_INVALID_ARG;
  *it = c->hostIter;
  return LADDS_OK;
}

int ladds_gpu_set_iteration(ladds_gpu_ctx *c, int64_t it) {
  if (!c || it < 0) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  CK(cudaMemcpyAsync(c->dIter, &it, sizeof(int64_t), cudaMemcpyHostToDevice, c->st));
  CK(cudaStreamSynchronize(c->st));
  c->hostIter = it;
  return LADDS_OK;
}

int ladds_gpu_set_profiling(ladds_gpu_ctx *c, int enable) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  c->profiling = enable != 0;
  std::memset(&c->times, 0, sizeof(c->times));
  return LADDS_OK;
}

int ladds_gpu_phase_times(ladds_gpu_ctx *c, ladds_phase_times *t) {
  if (!c || !t) return LADDS_ERR_INVALID_ARG;
  *t = c->times;
  t->totalMs = t->propagateMs + t->bucketMs + t->rowsortMs + t->permuteMs + t->candidatesMs + t->evaluateMs;
  return LADDS_OK;
}

int ladds_gpu_integrate(ladds_gpu_ctx *c, int steps) {
  if (!c || steps < 0) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  int left = steps;
  while (left > 0) {
    const int chunk = std::min(left, c->chunkSteps);
    CK(enqueueEphemeris(c, chunk));
    enqueuePropagate(c, chunk, 0);
    left -= chunk;
  }
  const int rc = syncAndStatus(c);
  collectTimes(c);
  c->hostIter += steps;
  c->orderValid = false;
  return rc;
}

}  // extern "C"

namespace {
// The order of the last scan without the objects that a removal takes out
// (keep[slot] = 0 among n slots; pos = their new slots), enqueued; its length goes
// to *count.  False: there is no order.
bool enqueueCompactOrder(ladds_gpu_ctx *c, const uint32_t *keep, const uint32_t *pos, size_t n, uint32_t *count) {
  const int m = (int)std::min(c->orderN, n);
  c->orderN = 0;  // until it is known to have run
  if (!m) return false;
  uint32_t *flag = c->keys, *at = c->scratchC, *moved = c->permB;  // free between calls
  k_order_flags<<<blocksFor(m, 256), 256, 0, c->st>>>(c->perm, keep, m, flag);
  enqueueExclusiveScan(c, flag, (size_t)m, at, c->st);
  k_order_compact<<<blocksFor(m, 256), 256, 0, c->st>>>(c->perm, flag, at, pos, m, moved, count);
  cudaMemcpyAsync(c->perm, moved, (size_t)m * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->st);
  return true;
}

// Compaction of the objects flagged keep[j] = 1 in scratchA: survivors keep
// their relative slot order and are renumbered 0..n'-1.  The arrays that the
// state buffers share are compacted through the roll-back buffer's, which
// hold nothing between calls.  One wait brings both counts: 500 of 10,500 objects
// removed after a scan in 55 us, 118 with a wait for each count and copy.
int compactKept(ladds_gpu_ctx *c) {
  const int n = (int)c->n, blocks = blocksFor(n, 256);
  uint32_t *keep = c->scratchA, *pos = c->scratchB;
  auto *counts = reinterpret_cast<uint32_t *>(c->dCandNeed);  // scratch words (reset by every scan)
  enqueueExclusiveScan(c, keep, (size_t)n, pos, c->st);
  DevState tmp{};
  tmp.aom = c->snap.x;
  tmp.bc = c->snap.y;
  tmp.radius = c->snap.z;
  tmp.id = reinterpret_cast<uint64_t *>(c->snap.vx);
  tmp.parent = reinterpret_cast<uint64_t *>(c->snap.vy);
  tmp.tag = reinterpret_cast<uint32_t *>(c->snap.vz);
  k_compact<<<blocks, 256, 0, c->st>>>(c->cur, c->alt, keep, pos, n, tmp, counts);
  k_compact_shared<<<blocks, 256, 0, c->st>>>(tmp, c->cur, counts);
  const bool order = enqueueCompactOrder(c, keep, pos, (size_t)n, counts + 1);
  unsigned long long both = 0;
  const int rc = fetchWord(c, counts, sizeof(both), &both);
  if (rc) return rc;
  std::swap(c->cur, c->alt);
  c->n = (size_t)(both & 0xffffffffull);
  if (order) c->orderN = (size_t)(both >> 32);
  c->orderValid = false;
  dropGraphs(c);
  return LADDS_OK;
}

// Conjunction scan of the current state (cell keys, sort, gather, pair scan),
// re-run with larger buffers after an overflow; sorted records in recs.
int scanState(ladds_gpu_ctx *c, const ScanConsts &sc, float cutF, std::vector<ladds_pair> &recs) {
  recs.clear();
  if (!c->n) return LADDS_OK;
  for (int attempt = 0; attempt < 5; ++attempt) {
    CK(cudaMemsetAsync(c->dCount, 0, 2 * sizeof(unsigned long long), c->st));
    c->orderN = 0;
    swapSortSets(c);
    k_scan_input<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur, (int)c->n, c->grid, scanInput(c));
    enqueueSort(c, c->st);
    enqueueScanWith(c, c->st, sc, cutF, c->dIter, -1);  // records carry the index of the last integrated iteration
    unsigned long long cnt = 0;
    bool overflow = false;
    const int rc = syncStatusAndGrow(c, &cnt, &overflow);
    collectTimes(c);
    if (rc) return rc;
    c->orderN = c->n;
    if (!overflow) {
      CK(fetchRecords(c, (size_t)cnt, recs));
      c->orderValid = true;
      std::sort(recs.begin(), recs.end(), pairLess);
      return LADDS_OK;
    }
  }
  return fail(c, LADDS_ERR_CAPACITY, "scan buffers kept overflowing");
}
}  // namespace

extern "C" {

int ladds_gpu_scan(ladds_gpu_ctx *c, const ladds_scan_params *p, ladds_pair *out, size_t cap, size_t *nOut) {
  if (!c || !p || !nOut || !std::isfinite(p->dt) || !(p->cutoff > 0) || !(p->nearThresholdRel >= 0))
    return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (p->cutoff > c->cfg.cutoff)
    return fail(c, LADDS_ERR_INVALID_ARG, "scan cutoff larger than the cutoff the cell grid was built for");
  CK(cudaSetDevice(c->dev));
  ScanConsts sc;
  sc.cutoffSq = p->cutoff * p->cutoff;
  sc.dt = p->dt;
  sc.factor = p->collisionDistanceFactor / 1000.;
  sc.minDetectionRadius = p->minDetectionRadius;
  sc.evasionSq = p->evasionCutoff * p->evasionCutoff;
  sc.conjSq = p->conjunctionThreshold * p->conjunctionThreshold;
  sc.nearRel = p->nearThresholdRel;
  std::vector<ladds_pair> recs;
  const int rc = scanState(c, sc, prefilterRadius(p->cutoff, p->nearThresholdRel), recs);
  if (rc) return rc;
  *nOut = recs.size();
  if (recs.size() > cap || (!out && !recs.empty()))
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small for the conjunction records");
  if (!recs.empty()) std::memcpy(out, recs.data(), recs.size() * sizeof(ladds_pair));
  return LADDS_OK;
}

int ladds_gpu_conjunctions(ladds_gpu_ctx *c, double dtScan, ladds_pair *out, size_t cap, size_t *nOut,
                           size_t *nCollisions, size_t *nEvasions, size_t *nConjunctions) {
  if (!c || !nOut || !std::isfinite(dtScan)) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  std::vector<ladds_pair> recs;
  ScanConsts sc = c->sc;
  sc.dt = dtScan;
  const int rc = scanState(c, sc, c->cutF, recs);
  if (rc) return rc;
  size_t nc = 0, ne = 0, nj = 0;
  for (const auto &p : recs) {
    nc += (p.flags & LADDS_PAIR_COLLISION) != 0;
    ne += (p.flags & LADDS_PAIR_EVASION) != 0;
    nj += (p.flags & LADDS_PAIR_CONJUNCTION) != 0;
  }
  if (nCollisions) *nCollisions = nc;
  if (nEvasions) *nEvasions = ne;
  if (nConjunctions) *nConjunctions = nj;
  *nOut = recs.size();
  if (recs.size() > cap || (!out && !recs.empty()))
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small for the conjunction records");
  if (!recs.empty()) std::memcpy(out, recs.data(), recs.size() * sizeof(ladds_pair));
  return LADDS_OK;
}

int ladds_gpu_step(ladds_gpu_ctx *c, int iterations, ladds_pair *out, size_t cap, size_t *nOut,
                   ladds_step_stats *stats) {
  if (!c || iterations < 0 || !nOut) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  if (stats) std::memset(stats, 0, sizeof(*stats));
  const int k = c->cfg.timestepsPerCollisionDetection;
  int scans = 0;
  for (int i = 0; i < iterations; ++i) scans += ((c->hostIter + i) % k) == 0;
  // the call's start state and the order of the last scan: the call is re-run
  // after a device pair-buffer overflow and undone when the caller's buffer is
  // too small.  A call of one propagation launch leaves the state in its buffer and
  // the order in the other sort set; for longer ones both are copied, and come
  // back into the buffer and the set that were current.
  const bool home = c->cfg.useGraphs && !c->profiling && c->n < kGraphObjects && iterations >= kHomeIterations;
  const bool oneLaunch = iterations > 0 && iterations <= c->chunkSteps &&
                         nextGroup(c->hostIter, 0, iterations, k).len == iterations;
  const size_t orderStart = c->orderN;
  const bool copyOrder = scans && orderStart && (home || !oneLaunch);
  if (copyOrder)
    CK(cudaMemcpyAsync(c->scratchC, c->perm, orderStart * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->st));
  if (home) {
    const int rc = homeBuffers(c, scans > 0);
    if (rc) return rc;
  }
  const DevState ringStart[3] = {c->cur, c->alt, c->alt2};
  const int setStart = c->sortParity;
  if (!oneLaunch) CK(copyDynamic(c->cur, c->snap, c->n, c->st));
  const int64_t startIter = c->hostIter;
  auto rollBack = [&]() -> int {
    c->cur = ringStart[0];
    c->alt = ringStart[1];
    c->alt2 = ringStart[2];
    if (!oneLaunch) CK(copyDynamic(c->snap, c->cur, c->n, c->st));
    if (c->sortParity != setStart) swapSortSets(c);
    if (copyOrder)
      CK(cudaMemcpyAsync(c->perm, c->scratchC, orderStart * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->st));
    CK(cudaMemcpyAsync(c->dIter, &startIter, sizeof(int64_t), cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
    c->hostIter = startIter;
    c->orderN = orderStart;
    c->orderValid = false;
    return LADDS_OK;
  };
  unsigned long long cnt = 0;
  int retries = 0;
  for (;;) {
    if (scans) c->orderN = 0;
    CK(cudaMemsetAsync(c->dCount, 0, 2 * sizeof(unsigned long long), c->st));
    const int64_t it0 = c->hostIter;
    const bool graph = c->cfg.useGraphs && !c->profiling && iterations >= 1 && c->n < kGraphObjects &&
                       (c->captureAll || chunksWorthCapturing(c, it0, iterations, k));
    if (graph) {
      // pass 1: capture the graphs this call needs (capture performs the host-side
      // buffer swaps; they are undone afterwards), so that no capture happens
      // between the timing events
      const DevState ring0[3] = {c->cur, c->alt, c->alt2};
      const int par0 = c->sortParity;
      for (int done = 0; done < iterations;) {
        const int len = std::min(iterations - done, c->chunkSteps);
        const int bufs = bufferRoles(c);
        const auto key = std::make_tuple(len, (int)((it0 + done) % k), bufs, c->n, c->pairCap);
        if (c->graphs.find(key) == c->graphs.end()) {
          CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
          enqueueChunk(c, it0 + done, len, k);
          cudaGraph_t gr = nullptr;
          CK(cudaStreamEndCapture(c->st, &gr));
          cudaGraphExec_t ex = nullptr;
          const cudaError_t ie = cudaGraphInstantiate(&ex, gr, 0);
          cudaGraphDestroy(gr);
          CK(ie);
          c->graphs.emplace(key, ex);
          CK(cudaGraphUpload(ex, c->st));  // else its first launch does, inside the timing events
        } else {
          replaySwaps(c, it0 + done, len, k);
        }
        done += len;
      }
      c->cur = ring0[0];
      c->alt = ring0[1];
      c->alt2 = ring0[2];
      if (c->sortParity != par0) swapSortSets(c);
      // pass 2: replay
      CK(cudaEventRecord(c->callStart, c->st));
      for (int done = 0; done < iterations;) {
        const int len = std::min(iterations - done, c->chunkSteps);
        const int bufs = bufferRoles(c);
        const auto key = std::make_tuple(len, (int)((it0 + done) % k), bufs, c->n, c->pairCap);
        auto git = c->graphs.find(key);
        if (git == c->graphs.end()) return fail(c, LADDS_ERR_STATE, "graph cache inconsistent");
        replaySwaps(c, it0 + done, len, k);
        CK(cudaGraphLaunch(git->second, c->st));
        done += len;
      }
    } else {
      CK(cudaEventRecord(c->callStart, c->st));
      for (int done = 0; done < iterations;) {
        const int len = std::min(iterations - done, c->chunkSteps);
        enqueueChunk(c, it0 + done, len, k);
        done += len;
      }
    }
    CK(cudaEventRecord(c->callEnd, c->st));
    bool overflow = false;
    int rc = syncStatusAndGrow(c, &cnt, &overflow);
    collectTimes(c);
    if (rc) {
      const int rb = rollBack();
      return rb ? rb : rc;
    }
    if (!overflow) break;
    // a device record or candidate buffer overflowed: it has grown; roll back, run the batch again
    if (++retries > 4) {
      rollBack();
      return fail(c, LADDS_ERR_CAPACITY, "device scan buffers kept overflowing");
    }
    rc = rollBack();
    if (rc) return rc;
  }
  float ms = 0;
  cudaEventElapsedTime(&ms, c->callStart, c->callEnd);
  std::vector<ladds_pair> recs;
  CK(fetchRecords(c, (size_t)cnt, recs));
  std::sort(recs.begin(), recs.end(), pairLess);
  *nOut = recs.size();
  if (recs.size() > cap || (!out && !recs.empty())) {
    const int rb = rollBack();
    if (rb) return rb;
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small for the conjunction records");
  }
  if (!recs.empty()) std::memcpy(out, recs.data(), recs.size() * sizeof(ladds_pair));
  c->hostIter += iterations;
  if (scans) {
    c->orderValid = true;
    c->orderN = c->n;
  }
  if (stats) {
    stats->iterations = (uint64_t)iterations;
    stats->scans = (uint64_t)scans;
    stats->records = cnt;
    stats->retries = (uint64_t)retries;
    stats->deviceMs = ms;
    for (const auto &p : recs) {
      stats->collisions += (p.flags & LADDS_PAIR_COLLISION) != 0;
      stats->evasions += (p.flags & LADDS_PAIR_EVASION) != 0;
      stats->conjunctions += (p.flags & LADDS_PAIR_CONJUNCTION) != 0;
    }
  }
  return LADDS_OK;
}

}  // extern "C"


extern "C" {

int ladds_gpu_step_host(ladds_gpu_ctx *c, size_t n, const double *const in[6], double *const outState[6],
                        ladds_pair *out, size_t cap, size_t *nOut, ladds_step_stats *stats) {
  if (!c || !in || !outState || !nOut) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  *nOut = 0;
  if (n != c->n) return fail(c, LADDS_ERR_INVALID_ARG, "step_host: n differs from the population size");
  for (int a = 0; a < 6; ++a)
    if (n && (!in[a] || !outState[a])) return fail(c, LADDS_ERR_INVALID_ARG, "null array pointer");
  CK(cudaSetDevice(c->dev));
  if (stats) std::memset(stats, 0, sizeof(*stats));
  c->pending.clear();
  const int k = c->cfg.timestepsPerCollisionDetection;
  const bool scan = (c->hostIter % k) == 0 && n;
  const int64_t startIter = c->hostIter;
  // the host's positions and velocities go to the other buffer, are propagated
  // there, and make it the current one
  const DevState S = c->alt;
  // any failure once work is enqueued: nothing of this call may still run when
  // it returns -- its copies into the caller's arrays and its kernels are
  // drained on all three streams -- and the iteration is not counted (the device
  // copy of the state is replaced by the next call's host state)
  auto abortCall = [&](int rc) {
    cudaStreamSynchronize(c->st2);
    cudaStreamSynchronize(c->st3);
    cudaStreamSynchronize(c->st);
    cudaMemcpyAsync(c->dIter, &startIter, sizeof(int64_t), cudaMemcpyHostToDevice, c->st);
    clearRowCounts(c);
    cudaStreamSynchronize(c->st);
    c->orderValid = false;
    return rc;
  };
#define CKS(call)                                                                                   \
  do {                                                                                              \
    cudaError_t e_ = (call);                                                                        \
    if (e_ != cudaSuccess)                                                                          \
      return abortCall(fail(c, LADDS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_))); \
  } while (0)
  CKS(cudaMemsetAsync(c->dCount, 0, 2 * sizeof(unsigned long long), c->st));
  CKS(cudaEventRecord(c->callStart, c->st));
  CKS(enqueueEphemeris(c, 1));
  if (scan) {
    c->orderN = 0;
    swapSortSets(c);
  }
  // pageable arrays go through pinned staging, copied on all host threads
  // chunk by chunk (the CUDA driver's own staging of pageable copies is slower)
  bool stageIn[6] = {}, stageOut[6] = {}, anyIn = false, anyOut = false;
  for (int a = 0; a < 6 && n; ++a) {
    stageIn[a] = !isPinned(in[a]);
    stageOut[a] = !isPinned(outState[a]);
    anyIn |= stageIn[a];
    anyOut |= stageOut[a];
  }
  if ((anyIn || anyOut) && !ensurePinStage(c, n)) {  // no pinned memory to spare: the driver stages the copies
    for (int a = 0; a < 6; ++a) stageIn[a] = stageOut[a] = false;
    anyIn = anyOut = false;
  }
  double *pinIn[6], *pinOut[6];
  const double *src[6];
  double *dstHost[6];
  for (int a = 0; a < 6; ++a) {
    pinIn[a] = c->pinStage ? c->pinStage + (size_t)a * c->pinCap : nullptr;
    pinOut[a] = c->pinStage ? c->pinStage + (size_t)(6 + a) * c->pinCap : nullptr;
    src[a] = stageIn[a] ? pinIn[a] : in[a];
    dstHost[a] = stageOut[a] ? pinOut[a] : outState[a];
  }
  // all six arrays through the staging buffer: one two-dimensional copy a chunk
  const bool allIn = anyIn && std::all_of(stageIn, stageIn + 6, [](bool b) { return b; });
  const bool allOut = anyOut && std::all_of(stageOut, stageOut + 6, [](bool b) { return b; });
  // chunks: host->device on st2, propagation on st, device->host on st3
  const int chunks = (int)std::max<size_t>(1, std::min<size_t>((size_t)kHostChunks, n / kHostChunkMin));
  // chunk starts on multiples of 256 objects keep every chunk's arrays 16-byte aligned (staged propagation)
  const size_t per = ((n + (size_t)chunks - 1) / (size_t)chunks + 255) / 256 * 256;
  double *const sArr[6] = {S.x, S.y, S.z, S.vx, S.vy, S.vz};
  const size_t devStride = (size_t)(S.y - S.x);
  int used = 0;
  for (int ch = 0; ch < chunks && n; ++ch) {
    const size_t lo = (size_t)ch * per;
    if (lo >= n) break;
    const size_t len = std::min(per, n - lo);
    if (anyIn) hostCopy(pinIn, in, stageIn, lo, len);
    CKS(copySix(sArr, src, lo, len, allIn, c->pinCap, devStride, cudaMemcpyHostToDevice, c->st2));
    CKS(cudaEventRecord(c->evPipe[ch], c->st2));
    CKS(cudaStreamWaitEvent(c->st, c->evPipe[ch], 0));
    launchPropagate(c, S, S, lo, (int)len, 1, 0, scan);
    CKS(cudaEventRecord(c->evPipe[kHostChunks + ch], c->st));
    CKS(cudaStreamWaitEvent(c->st3, c->evPipe[kHostChunks + ch], 0));
    CKS(copySix(dstHost, sArr, lo, len, allOut, devStride, c->pinCap, cudaMemcpyDeviceToHost, c->st3));
    CKS(cudaEventRecord(c->evPipe[2 * kHostChunks + ch], c->st3));
    used = ch + 1;
  }
  ScanConsts sc = c->sc;
  sc.dt = c->cfg.deltaT * (double)k;
  if (n) rotateStates(c);
  if (scan) {
    enqueueSort(c, c->st);
    enqueueScanWith(c, c->st, sc, c->cutF, c->dIterBase, 0);
  }
  if (used) {
    CKS(cudaEventRecord(c->evPipe[3 * kHostChunks], c->st3));
    CKS(cudaStreamWaitEvent(c->st, c->evPipe[3 * kHostChunks], 0));
  }
  CKS(cudaEventRecord(c->callEnd, c->st));
  // staged outputs: each chunk leaves the pinned buffer as soon as it is there
  for (int ch = 0; ch < used && anyOut; ++ch) {
    CKS(cudaEventSynchronize(c->evPipe[2 * kHostChunks + ch]));
    const size_t lo = (size_t)ch * per;
    hostCopy(outState, pinOut, stageOut, lo, std::min(per, n - lo));
  }
  unsigned long long cnt = 0;
  bool overflow = false;
  int rc = syncStatusAndGrow(c, &cnt, &overflow);
  collectTimes(c);
  if (rc) return abortCall(rc);
  int retries = 0;
  while (overflow) {  // the device buffers have grown: the scan alone runs again on the same state
    if (++retries > 4) return abortCall(fail(c, LADDS_ERR_STATE, "device scan buffers kept overflowing"));
    CKS(cudaMemsetAsync(c->dCount, 0, 2 * sizeof(unsigned long long), c->st));
    CKS(cudaMemsetAsync(c->dCandCount, 0, kScanCounters * sizeof(unsigned long long), c->st));  // the sort cleared them for one scan
    enqueueScanWith(c, c->st, sc, c->cutF, c->dIterBase, 0);
    rc = syncStatusAndGrow(c, &cnt, &overflow);
    collectTimes(c);
    if (rc) return abortCall(rc);
  }
  CKS(cudaStreamSynchronize(c->st3));
  float ms = 0;
  cudaEventElapsedTime(&ms, c->callStart, c->callEnd);
  std::vector<ladds_pair> recs;
  CKS(fetchRecords(c, (size_t)cnt, recs));
  std::sort(recs.begin(), recs.end(), pairLess);
  c->hostIter += 1;
  if (scan) {
    c->orderValid = true;
    c->orderN = n;
  }
  if (stats) {
    stats->iterations = 1;
    stats->scans = scan ? 1 : 0;
    stats->records = cnt;
    stats->retries = (uint64_t)retries;
    stats->deviceMs = ms;
    for (const auto &p : recs) {
      stats->collisions += (p.flags & LADDS_PAIR_COLLISION) != 0;
      stats->evasions += (p.flags & LADDS_PAIR_EVASION) != 0;
      stats->conjunctions += (p.flags & LADDS_PAIR_CONJUNCTION) != 0;
    }
  }
  *nOut = recs.size();
  if (recs.size() > cap || (!out && !recs.empty())) {
    c->pending = std::move(recs);
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small: the records wait in ladds_gpu_pending_records");
  }
  if (!recs.empty()) std::memcpy(out, recs.data(), recs.size() * sizeof(ladds_pair));
  return LADDS_OK;
#undef CKS
}

int ladds_gpu_pending_records(ladds_gpu_ctx *c, ladds_pair *out, size_t cap, size_t *nOut) {
  if (!c || !nOut) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  *nOut = c->pending.size();
  if (c->pending.size() > cap || (!out && !c->pending.empty()))
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small for the pending records");
  if (!c->pending.empty()) std::memcpy(out, c->pending.data(), c->pending.size() * sizeof(ladds_pair));
  c->pending.clear();
  return LADDS_OK;
}

int ladds_gpu_cell_order(ladds_gpu_ctx *c, size_t cap, size_t *n, uint32_t *keys, uint32_t *slots) {
  if (!c || !n) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (!c->orderValid) return fail(c, LADDS_ERR_STATE, "no conjunction scan since the last change of the state");
  *n = c->n;
  if (cap < c->n) return fail(c, LADDS_ERR_CAPACITY, "buffer smaller than the population");
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  if (keys) CK(cudaMemcpy(keys, c->sortedKeys, c->n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
  if (slots) CK(cudaMemcpy(slots, c->perm, c->n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
  return LADDS_OK;
}

int ladds_gpu_grid(const ladds_gpu_ctx *c, int32_t dims[3], int32_t *reach, double *cellSize) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  if (dims)
    for (int d = 0; d < 3; ++d) dims[d] = c->grid.n[d];
  if (reach) *reach = c->grid.reach;
  if (cellSize) *cellSize = c->grid.cellSize;
  return LADDS_OK;
}

int ladds_gpu_clear_parents(ladds_gpu_ctx *c) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  k_clear_parents<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur.parent, (int)c->n);
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

int ladds_gpu_mark_deleted(ladds_gpu_ctx *c, const uint32_t *slots, size_t m) {
  if (!c || (m && !slots)) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (!m || !c->n) return LADDS_OK;
  for (size_t i = 0; i < m; ++i)
    if (slots[i] >= c->n) return fail(c, LADDS_ERR_INVALID_ARG, "slot out of range");
  CK(cudaSetDevice(c->dev));
  std::vector<uint8_t> mark(c->n, 0);
  for (size_t i = 0; i < m; ++i) mark[slots[i]] = 1;
  uint8_t *dMark = reinterpret_cast<uint8_t *>(c->scratchA);
  CK(cudaMemcpyAsync(dMark, mark.data(), c->n, cudaMemcpyHostToDevice, c->st));
  k_mark_deleted<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur.tag, dMark, (int)c->n);
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

}  // extern "C"

namespace {
// ids of the objects flagged keep[j] == 0 in scratchA, in slot order (at most
// cap of them), gathered on the device: only the removed ones cross to the host
int removedIdsInSlotOrder(ladds_gpu_ctx *c, uint64_t *removedIds, size_t cap) {
  const int n = (int)c->n;
  unsigned *dCnt = reinterpret_cast<unsigned *>(c->dCandNeed) + 1;  // word 0 holds the removal count
  CK(cudaMemsetAsync(dCnt, 0, sizeof(unsigned), c->st));
  // keys / scratchB / scratchC are free between calls (scratchB is compactKept's output, written later)
  k_removed_ids<<<blocksFor(n, 256), 256, 0, c->st>>>(c->scratchA, c->cur.id, n, c->keys, c->scratchC, c->scratchB,
                                                       dCnt);
  CK(cudaGetLastError());
  unsigned m = 0;
  CK(cudaMemcpyAsync(&m, dCnt, sizeof(unsigned), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  std::vector<uint32_t> sl(m), lo(m), hi(m);
  if (m) {
    CK(cudaMemcpyAsync(sl.data(), c->keys, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(lo.data(), c->scratchC, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(hi.data(), c->scratchB, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
  }
  std::vector<uint32_t> order(m);
  for (uint32_t i = 0; i < m; ++i) order[i] = i;
  std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return sl[a] < sl[b]; });
  for (size_t w = 0; w < m && w < cap; ++w) removedIds[w] = ((uint64_t)hi[order[w]] << 32) | lo[order[w]];
  return LADDS_OK;
}

}  // namespace

extern "C" {

int ladds_gpu_remove_below(ladds_gpu_ctx *c, double minAltitude, size_t *nRemoved, uint64_t *removedIds,
                           size_t cap) {
  if (!c || !std::isfinite(minAltitude)) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (nRemoved) *nRemoved = 0;
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  const int n = (int)c->n;
  const double crit = kREarth + minAltitude;  // Simulation.cpp:573
  const double critSq = crit * crit;           // Simulation.cpp:581
  unsigned *dBurnt = reinterpret_cast<unsigned *>(c->dCandNeed);  // scratch word (reset by every scan)
  CK(cudaMemsetAsync(dBurnt, 0, sizeof(unsigned), c->st));
  k_burnup_flags<<<blocksFor(n, 256), 256, 0, c->st>>>(c->cur.x, c->cur.y, c->cur.z, n, critSq, c->scratchA,
                                                        dBurnt);
  unsigned burnt = 0;
  int rc = fetchCount(c, dBurnt, &burnt);
  if (rc) return rc;
  if (!burnt) return LADDS_OK;  // nothing burns up: the state, its order and the captured graphs stay
  if (removedIds) {  // ids of the removed objects, in slot order, before the compaction renumbers them
    const int rid = removedIdsInSlotOrder(c, removedIds, cap);
    if (rid) return rid;
  }
  rc = compactKept(c);
  if (rc) return rc;
  if (nRemoved) *nRemoved = (size_t)n - c->n;
  return LADDS_OK;
}

int ladds_gpu_remove_escaping(ladds_gpu_ctx *c, size_t *nRemoved, uint64_t *removedIds, size_t cap) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (nRemoved) *nRemoved = 0;
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  const int n = (int)c->n;
  const double3 lo = make_double3(c->cfg.boxMin[0], c->cfg.boxMin[1], c->cfg.boxMin[2]);
  const double3 hi = make_double3(c->cfg.boxMax[0], c->cfg.boxMax[1], c->cfg.boxMax[2]);
  unsigned *dOut = reinterpret_cast<unsigned *>(c->dCandNeed);  // scratch word (reset by every scan)
  CK(cudaMemsetAsync(dOut, 0, sizeof(unsigned), c->st));
  k_escape_flags<<<blocksFor(n, 256), 256, 0, c->st>>>(c->cur, n, lo, hi, c->scratchA, dOut);
  unsigned escaped = 0;
  int rc = fetchCount(c, dOut, &escaped);
  if (rc) return rc;
  if (!escaped) return LADDS_OK;  // nobody leaves: the state, its order and the captured graphs stay
  if (removedIds) {  // ids of the removed objects, in slot order, before the compaction renumbers them
    const int rid = removedIdsInSlotOrder(c, removedIds, cap);
    if (rid) return rid;
  }
  rc = compactKept(c);
  if (rc) return rc;
  if (nRemoved) *nRemoved = (size_t)n - c->n;
  return LADDS_OK;
}

int ladds_gpu_pack_layers(ladds_gpu_ctx *c, int32_t izLo, int32_t izHi, int remove, ladds_state_record *out,
                          size_t cap, size_t *nOut) {
  if (!c || !nOut || (cap && !out) || (!out && !remove))
    return fail(c, LADDS_ERR_INVALID_ARG, "pack_layers: bad argument");
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  *nOut = 0;
  if (!c->n || izHi <= izLo) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  if (cap) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, out) != cudaSuccess ||
        !((at.type == cudaMemoryTypeDevice && at.device == c->dev) || at.type == cudaMemoryTypeManaged)) {
      cudaGetLastError();
      return fail(c, LADDS_ERR_INVALID_ARG, "pack_layers: out must be device memory of the context's device");
    }
  }
  const int n = (int)c->n;
  // the sort's keys and arrivals are free between calls; scratchA takes the
  // removal flags of compactKept
  uint32_t *sel = c->keys, *pos = c->scratchC, *idx = c->scratchB;
  const int m = (int)std::min(c->orderN, c->n);  // records leave in the order of the last scan
  k_layer_flags<<<blocksFor(n, 256), 256, 0, c->st>>>(c->cur.z, c->cur.tag, n, c->grid, izLo, izHi, c->scratchA);
  k_order_select<<<blocksFor(n, 256), 256, 0, c->st>>>(c->scratchA, c->perm, m, n, sel);
  enqueueExclusiveScan(c, sel, (size_t)n, pos, c->st);
  auto *dSelected = reinterpret_cast<uint32_t *>(c->dCandNeed);  // scratch word (reset by every scan)
  k_selected_slots<<<blocksFor(n, 256), 256, 0, c->st>>>(sel, pos, c->perm, m, n, idx, dSelected);
  CK(cudaGetLastError());
  unsigned count = 0;
  const int rl = fetchCount(c, dSelected, &count);
  if (rl) return rl;
  *nOut = count;
  if (!count) return LADDS_OK;
  if (remove && !out) return compactKept(c);  // removed without being packed
  if (count > cap) return fail(c, LADDS_ERR_CAPACITY, "pack_layers: more particles than the output holds");
  k_gather_records<<<blocksFor(count, 128), 128, 0, c->st>>>(c->cur, idx, (int)count, out);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->st));
  return remove ? compactKept(c) : LADDS_OK;
}

int ladds_gpu_append_records(ladds_gpu_ctx *c, const ladds_state_record *records, size_t m) {
  if (!c || (m && !records)) return fail(c, LADDS_ERR_INVALID_ARG, "append_records: bad argument");
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (!m) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, records) != cudaSuccess ||
      !((at.type == cudaMemoryTypeDevice && at.device == c->dev) || at.type == cudaMemoryTypeManaged)) {
    cudaGetLastError();
    return fail(c, LADDS_ERR_INVALID_ARG, "append_records: records must be device memory of the context's device");
  }
  if (c->n + m > (size_t)kTagSlotMask) return fail(c, LADDS_ERR_TOO_LARGE, "append_records: too many particles");
  int rc = ensureCapacity(c, c->n + m);
  if (rc) return rc;
  // scratch words (reset by every scan): [0] bad records, [1] records with a parent
  unsigned *dBad = reinterpret_cast<unsigned *>(c->dCandNeed);
  CK(cudaMemsetAsync(dBad, 0, 2 * sizeof(unsigned), c->st));
  k_append_records<<<blocksFor(m, 128), 128, 0, c->st>>>(records, (int)m, c->cur, (uint32_t)c->n, dBad);
  CK(cudaGetLastError());
  unsigned flags[2] = {0, 0};
  CK(cudaMemcpyAsync(flags, dBad, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  if (flags[0]) return fail(c, LADDS_ERR_INVALID_ARG, "append_records: a record holds NaN/Inf or a bad activity state");
  if (flags[1]) c->anyParent = true;
  c->n += m;
  c->orderValid = false;
  dropGraphs(c);
  return LADDS_OK;
}

int ladds_gpu_truncate(ladds_gpu_ctx *c, size_t n0) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (n0 >= c->n) return LADDS_OK;
  if (c->orderN) {
    CK(cudaSetDevice(c->dev));
    k_below_flags<<<blocksFor(c->n, 256), 256, 0, c->st>>>((int)c->n, (uint32_t)n0, c->scratchA, c->scratchB);
    auto *count = reinterpret_cast<uint32_t *>(c->dCandNeed);  // scratch word (reset by every scan)
    unsigned left = 0;
    enqueueCompactOrder(c, c->scratchA, c->scratchB, c->n, count);
    const int rc = fetchCount(c, count, &left);
    if (rc) return rc;
    c->orderN = left;
  }
  c->n = n0;  // the objects with the last slots
  c->orderValid = false;
  dropGraphs(c);
  return LADDS_OK;
}

int ladds_gpu_remove_slots(ladds_gpu_ctx *c, const uint32_t *slots, size_t m) {
  if (!c || (m && !slots)) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  if (!m || !c->n) return LADDS_OK;
  for (size_t i = 0; i < m; ++i)
    if (slots[i] >= c->n) return fail(c, LADDS_ERR_INVALID_ARG, "slot out of range");
  CK(cudaSetDevice(c->dev));
  std::vector<uint8_t> mark(c->n, 0);
  for (size_t i = 0; i < m; ++i) mark[slots[i]] = 1;
  uint8_t *dMark = reinterpret_cast<uint8_t *>(c->scratchB);  // read before compactKept writes scratchB
  CK(cudaMemcpyAsync(dMark, mark.data(), c->n, cudaMemcpyHostToDevice, c->st));
  k_slot_mark_flags<<<blocksFor(c->n, 256), 256, 0, c->st>>>((int)c->n, dMark, c->scratchA);
  return compactKept(c);
}

int ladds_gpu_select_layers(ladds_gpu_ctx *c, int32_t izLo, int32_t izHi, uint32_t *slots, size_t cap, size_t *n) {
  if (!c || !n || (cap && !slots)) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  *n = 0;
  if (!c->n || izHi <= izLo) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  unsigned *dCount = reinterpret_cast<unsigned *>(c->dCandNeed);  // scratch word (reset by every scan)
  CK(cudaMemsetAsync(dCount, 0, sizeof(unsigned), c->st));
  k_select_layers<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur.z, c->cur.tag, (int)c->n, c->grid, izLo, izHi,
                                                            c->scratchA, dCount, (unsigned)c->n);
  unsigned cnt = 0;
  CK(cudaMemcpyAsync(&cnt, dCount, sizeof(unsigned), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  *n = cnt;
  if (cnt > cap) return fail(c, LADDS_ERR_CAPACITY, "select_layers: buffer too small");
  std::vector<uint32_t> h(cnt);
  if (cnt) CK(cudaMemcpy(h.data(), c->scratchA, cnt * sizeof(uint32_t), cudaMemcpyDeviceToHost));
  std::sort(h.begin(), h.end());
  std::copy(h.begin(), h.end(), slots);
  return LADDS_OK;
}

int ladds_gpu_layer_histogram(ladds_gpu_ctx *c, uint64_t *counts, size_t nLayers) {
  if (!c || !counts) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  const size_t nz = (size_t)c->grid.n[2];
  if (nLayers < nz) return fail(c, LADDS_ERR_CAPACITY, "layer_histogram: fewer entries than cell layers");
  std::fill(counts, counts + nLayers, 0ull);
  if (!c->n) return LADDS_OK;
  CK(cudaSetDevice(c->dev));
  if (nz > c->cap) return fail(c, LADDS_ERR_CAPACITY, "layer_histogram: more cell layers than capacity");
  auto *dCounts = reinterpret_cast<unsigned long long *>(c->sortRec);  // cap entries of 8 B
  CK(cudaMemsetAsync(dCounts, 0, nz * sizeof(unsigned long long), c->st));
  k_layer_histogram<<<blocksFor(c->n, 256), 256, 0, c->st>>>(c->cur.z, c->cur.tag, (int)c->n, c->grid, dCounts);
  CK(cudaMemcpyAsync(counts, dCounts, nz * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  CK(cudaGetLastError());
  return LADDS_OK;
}

int ladds_gpu_set_halo(ladds_gpu_ctx *c, size_t haloStart) {
  if (!c) return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  const uint32_t h = haloStart >= (size_t)0xffffffffu ? 0xffffffffu : (uint32_t)haloStart;
  if (h != c->haloStart) dropGraphs(c);  // captured scans carry the old value
  c->haloStart = h;
  return LADDS_OK;
}

int ladds_gpu_functor_pairs(ladds_gpu_ctx *c, const ladds_scan_params *p, size_t nPairs, const ladds_object *first,
                            const ladds_object *second, ladds_pair *out, size_t cap, size_t *nOut) {
  if (!c || !p || !nOut || (nPairs && (!first || !second)) || nPairs > (size_t)INT32_MAX)
    return LADDS_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  *nOut = 0;
  if (!nPairs) return LADDS_OK;
  for (size_t k = 0; k < nPairs; ++k)
    for (const ladds_object *o : {&first[k], &second[k]})
      if (o->activity < 0 || o->activity > 2 || o->slot > kTagSlotMask)
        return fail(c, LADDS_ERR_INVALID_ARG, "object activity or slot out of range");
  CK(cudaSetDevice(c->dev));
  if (nPairs > c->objCap) {
    if (c->dObj) cudaFree(c->dObj);
    c->dObj = nullptr;
    c->objCap = 0;
    if (cudaMalloc(&c->dObj, 2 * nPairs * sizeof(ladds_object)) != cudaSuccess) {
      cudaGetLastError();
      return fail(c, LADDS_ERR_ALLOC, "device allocation failed (pair objects)");
    }
    c->objCap = nPairs;
  }
  CK(cudaMemcpyAsync(c->dObj, first, nPairs * sizeof(ladds_object), cudaMemcpyHostToDevice, c->st));
  CK(cudaMemcpyAsync(c->dObj + nPairs, second, nPairs * sizeof(ladds_object), cudaMemcpyHostToDevice, c->st));
  ScanConsts sc;
  sc.cutoffSq = p->cutoff * p->cutoff;
  sc.dt = p->dt;
  sc.factor = p->collisionDistanceFactor / 1000.;
  sc.minDetectionRadius = p->minDetectionRadius;
  sc.evasionSq = p->evasionCutoff * p->evasionCutoff;
  sc.conjSq = p->conjunctionThreshold * p->conjunctionThreshold;
  sc.nearRel = p->nearThresholdRel;
  std::vector<ladds_pair> recs;
  for (int attempt = 0; attempt < 3; ++attempt) {
    CK(cudaMemsetAsync(c->dCount, 0, sizeof(unsigned long long), c->st));
    k_functor_pairs<<<blocksFor(nPairs, 256), 256, 0, c->st>>>(c->dObj, c->dObj + nPairs, (int)nPairs, sc,
                                                                c->dPairs, c->dCount,
                                                                (unsigned long long)c->pairCap);
    CK(cudaStreamSynchronize(c->st));
    CK(cudaGetLastError());
    unsigned long long cnt = 0;
    CK(cudaMemcpy(&cnt, c->dCount, sizeof(cnt), cudaMemcpyDeviceToHost));
    if (cnt <= c->pairCap) {
      recs.resize(cnt);
      if (cnt) CK(cudaMemcpy(recs.data(), c->dPairs, cnt * sizeof(ladds_pair), cudaMemcpyDeviceToHost));
      break;
    }
    const int rc = ensurePairCapacity(c, (size_t)cnt);
    if (rc) return rc;
  }
  std::sort(recs.begin(), recs.end(), pairLess);
  *nOut = recs.size();
  if (recs.size() > cap || (!out && !recs.empty()))
    return fail(c, LADDS_ERR_CAPACITY, "output buffer too small for the pair records");
  if (!recs.empty()) std::memcpy(out, recs.data(), recs.size() * sizeof(ladds_pair));
  return LADDS_OK;
}

}  // extern "C"

// ----------------------------------------------------------------------------
// Autotuner: cell size, block shapes and the captured chunk length.
namespace {

// one timed trial of `cfg` (+ chunk length) on a copy of c's population
int tuneTrial(ladds_gpu_ctx *c, const ladds_gpu_config &cfg, int chunk, int steps, ladds_tune_trial &t) {
  ladds_gpu_ctx *tc = nullptr;
  int rc = ladds_gpu_create(&cfg, &tc);
  if (rc) return fail(c, rc, "autotune: a trial context could not be created");
  tc->chunkSteps = chunk;
  // a trial's calls come once; where the context's come again and run in graphs, the trial's do too
  tc->captureAll = true;
  rc = ensureCapacity(tc, c->n);
  if (!rc && c->n) {
    const cudaError_t e = copyState(c->cur, tc->cur, c->n, c->st);
    if (e != cudaSuccess) rc = fail(c, LADDS_ERR_CUDA, cudaGetErrorString(e));
  }
  if (!rc && cudaStreamSynchronize(c->st) != cudaSuccess) rc = fail(c, LADDS_ERR_CUDA, "autotune: state copy");
  if (!rc) {
    tc->n = c->n;
    tc->anyParent = c->anyParent;  // the trial's scans skip and walk what the context's do
    tc->haloStart = c->haloStart;
    rc = ladds_gpu_set_iteration(tc, c->hostIter);
  }
  std::vector<ladds_pair> recs((size_t)1 << 16);
  ladds_step_stats st{};
  for (int pass = 0; pass < 2 && !rc; ++pass) {  // warm-up, then the timed run (captures come before its timing events)
    const int n = pass == 0 ? std::min(steps, 2 * chunk) : steps;
    size_t got = 0;
    rc = ladds_gpu_step(tc, n, recs.data(), recs.size(), &got, &st);
    if (rc == LADDS_ERR_CAPACITY) {
      recs.resize(got);
      rc = ladds_gpu_step(tc, n, recs.data(), recs.size(), &got, &st);
    }
    if (rc) rc = fail(c, rc, std::string("autotune trial: ") + ladds_gpu_last_error(tc));
  }
  if (!rc) {
    t.cellSize = tc->grid.cellSize;
    t.reach = tc->grid.reach;
    t.propagateBlock = cfg.propagateBlock;
    t.scanBlock = cfg.scanBlock;
    t.chunkSteps = chunk;
    t.scanScreen = cfg.scanScreen;
    t.walkForm = cfg.walkForm;
    t.msPerStep = st.deviceMs / std::max(steps, 1);
  }
  ladds_gpu_destroy(tc);
  return rc;
}

}  // namespace

extern "C" {

int ladds_gpu_autotune(ladds_gpu_ctx *c, int stepsPerTrial, ladds_tune_trial *trials, size_t cap, size_t *nTrials,
                       ladds_tune_trial *best) {
  if (!c || stepsPerTrial < 1 || !best || (cap && !trials)) return fail(c, LADDS_ERR_INVALID_ARG, "autotune: bad argument");
  std::vector<ladds_tune_trial> all;
  ladds_gpu_config cfg = c->cfg;
  cfg.pairCapacity = c->pairCap;
  cfg.useGraphs = 1;
  ladds_tune_trial bestT{};
  bestT.msPerStep = INFINITY;
  int bestChunk = c->chunkSteps;
  auto run = [&](const ladds_gpu_config &k, int chunk) -> int {
    ladds_tune_trial t{};
    const int rc = tuneTrial(c, k, chunk, stepsPerTrial, t);
    if (rc) return rc;
    all.push_back(t);
    if (t.msPerStep < bestT.msPerStep) {
      bestT = t;
      cfg = k;
      bestChunk = chunk;
    }
    return LADDS_OK;
  };
  // 0. the current cell edge, with full candidate buffers listed and screened
  //    in place (the population's density decides)
  const int screens[] = {LADDS_SCREEN_LISTS, LADDS_SCREEN_BUFFER};
  {
    const ladds_gpu_config base = cfg;
    for (int screen : screens) {
      ladds_gpu_config k = base;
      k.scanScreen = screen;
      const int rc = run(k, bestChunk);
      if (rc) return rc;
    }
  }
  // 1. cell edge in [20, 160] km: cutoff / R (neighbour reach R = 1..4) and
  //    coarser cells 1.5 and 2 cutoffs wide (reach 1), each with both screens,
  //    whose order differs between edges (8e6 small debris: 80 km 5.6 ms listed, 5.7
  //    in place; 40 km 4.3 and 3.0); the current edge is measured already
  {
    const ladds_gpu_config base = cfg;
    std::vector<double> cells = {base.cellSize};
    for (int R = 1; R <= 4; ++R) cells.push_back(base.cutoff * (1.0 + 1e-6) / R);
    cells.push_back(1.5 * base.cutoff);
    cells.push_back(2.0 * base.cutoff);
    for (size_t i = 1; i < cells.size(); ++i) {
      const double cs = cells[i];
      if (cs < 20.0 || cs > 160.0) continue;
      if (i == 1 && base.cellSize <= 0) continue;  // the default edge: measured as the current one
      if (i > 1 && cs == base.cellSize) continue;
      for (int screen : screens) {
        ladds_gpu_config k = base;
        k.cellSize = cs;
        k.scanScreen = screen;
        const int rc = run(k, bestChunk);
        if (rc) return rc;
      }
    }
  }
  // 2. block shapes of the propagation and of the pair evaluation
  {
    const ladds_gpu_config base = cfg;
    for (int pb : {128, 256})
      for (int sb : {128, 256}) {
        ladds_gpu_config k = base;
        k.propagateBlock = pb;
        k.scanBlock = sb;
        if ((pb == base.propagateBlock || (pb == 256 && base.propagateBlock == 0)) &&
            (sb == base.scanBlock || (sb == 256 && base.scanBlock == 0)))
          continue;  // measured already
        const int rc = run(k, bestChunk);
        if (rc) return rc;
      }
  }
  // 3. iterations per captured chunk
  {
    const ladds_gpu_config base = cfg;
    for (int chunk : {32, 64, 128}) {
      if (chunk == bestChunk) continue;
      const int rc = run(base, chunk);
      if (rc) return rc;
    }
  }
  // apply the best configuration to the context (its state is untouched)
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  CK(cudaStreamSynchronize(c->st));
  if (cfg.cellSize != c->cfg.cellSize) {  // new tables beside the old ones: without memory for them, all stays as it was
    const double edge = c->cfg.cellSize;
    const GridTables old = *c;
    static_cast<GridTables &>(*c) = GridTables{};
    c->cfg.cellSize = cfg.cellSize;
    int rc = buildGrid(c);
    if (!rc) rc = allocGridBuffers(c);
    if (!rc && c->cap && !ensureScanWorkspace(c, c->cap)) rc = fail(c, LADDS_ERR_ALLOC, "autotune: scan workspace");
    GridTables spare = old;
    if (rc) {
      spare = *c;
      static_cast<GridTables &>(*c) = old;
      c->cfg.cellSize = edge;
    }
    CK(cudaStreamSynchronize(c->st));  // the new tables are cleared
    if (spare.tables) cudaFree(spare.tables);
    if (spare.cellOffBase) cudaFree(spare.cellOffBase);
    if (rc) return rc;
    c->orderValid = false;
  }
  c->cfg.propagateBlock = cfg.propagateBlock;
  c->cfg.scanBlock = cfg.scanBlock;
  c->cfg.scanScreen = cfg.scanScreen;
  c->cfg.walkForm = cfg.walkForm;
  c->chunkSteps = bestChunk;
  dropGraphs(c);
  *best = bestT;
  if (nTrials) *nTrials = all.size();
  for (size_t i = 0; i < all.size() && i < cap; ++i) trials[i] = all[i];
  return LADDS_OK;
}

}  // extern "C"

// ----------------------------------------------------------------------------
// Adjoint of the propagation for conjunction pairs (kernels in adjoint.cuh).
namespace {

template <typename T>
int ensureDev(ladds_gpu_ctx *c, T *&p, size_t &cap, size_t need) {
  if (need <= cap && p) return LADDS_OK;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  p = static_cast<T *>(contextTake(c, need * sizeof(T)));
  if (!p && need) return fail(c, LADDS_ERR_ALLOC, "device allocation for the adjoint pair batch failed");
  cap = need;
  return LADDS_OK;
}

// buffers of nPairs pairs and the ephemeris of `steps` steps
int adjPrepare(ladds_gpu_ctx *c, size_t nPairs, int steps) {
  auto &A = c->adj;
  const size_t nObj = 2 * nPairs;
  size_t objCap = A.objCap;
  int rc;
  if (nObj > A.objCap) {
    size_t cap0 = 0, cap1 = 0, cap2 = 0, cap3 = 0, cap4 = 0, cap5 = 0, cap6 = 0, cap7 = 0;
    if ((rc = ensureDev(c, A.st, cap0, 6 * nObj)) || (rc = ensureDev(c, A.bc, cap1, nObj)) ||
        (rc = ensureDev(c, A.aom, cap2, nObj)) || (rc = ensureDev(c, A.miss, cap3, nPairs)) ||
        (rc = ensureDev(c, A.grad, cap4, 7 * nObj)) || (rc = ensureDev(c, A.arg, cap5, nPairs)) ||
        (rc = ensureDev(c, A.off, cap6, 6 * nPairs)) || (rc = ensureDev(c, A.seed, cap7, 6 * nObj))) {
      A.objCap = 0;
      return rc;
    }
    objCap = nObj;
  }
  A.objCap = objCap;
  return ensureDev(c, A.eph, A.ephCap, (size_t)3 * steps);
}

// The forward sweep leaves the reverse sweep's records (12 doubles per object
// and step) where all of them fit in this many bytes -- 4096 pairs of 1080 steps
// are 0.85 GB of the device's 180 -- and checkpoints elsewhere, from which the
// reverse sweep makes the records segment by segment: a second forward sweep,
// which is the longer part.  4096 pairs, reverse sweep: 0.79 us per step from kept
// records, 2.40 by segments of 64 steps.
constexpr size_t kAdjRecordBytes = (size_t)1 << 30;
constexpr size_t kAdjRecord = 12;

int adjCheckpoints(ladds_gpu_ctx *c, size_t nObj, int steps, int ck) {
  const size_t nSeg = ((size_t)steps + ck - 1) / ck;
  return ensureDev(c, c->adj.ckpt, c->adj.ckptCap, nSeg * 6 * nObj);
}

// whole or by segments, with the buffers of either
int adjStorage(ladds_gpu_ctx *c, size_t nObj, int steps, int ck) {
  auto &A = c->adj;
  const size_t all = (size_t)steps * kAdjRecord * nObj;
  A.whole = all * sizeof(double) <= kAdjRecordBytes && ensureDev(c, A.rec, A.recCap, all) == LADDS_OK;
  return A.whole ? LADDS_OK : adjCheckpoints(c, nObj, steps, ck);
}

int adjEphemeris(ladds_gpu_ctx *c, int steps) {
  k_ephemeris<<<blocksFor((size_t)3 * steps, 128), 128, 0, c->st>>>(c->adj.eph, steps, 0, c->cfg.startTime,
                                                                     c->cfg.deltaT, c->pc.hc1, c->pc.hc2,
                                                                     c->cfg.epochJD, c->theta0, c->pc.mask);
  CK(cudaGetLastError());
  return LADDS_OK;
}

// steps s0 + 1 .. s1 from the states st; records from step s0 + 1 on (or null)
void adjForward(ladds_gpu_ctx *c, const double *st, int nObj, int s0, int s1, bool sweep, double *rec) {
  auto &A = c->adj;
  auto kernel = forMask(c->pc.mask, [](auto mask) { return k_adj_forward<decltype(mask)::value>; });
  kernel<<<blocksFor(nObj, kAdjObjs), kAdjFwdThreads, 0, c->st>>>(
      st, A.bc, A.aom, nObj, s0, s1, A.eph, c->pc, c->cfg.deltaT, A.ck, sweep && !A.whole ? A.ckpt : nullptr, rec,
      sweep ? A.miss : nullptr, A.arg, A.seed);
}

// the reverse of steps s1 .. s0 + 1 from their records
int adjBackward(ladds_gpu_ctx *c, int nObj, int s0, int s1) {
  auto &A = c->adj;
  auto kernel = forMask(c->pc.mask, [](auto mask) { return k_adj_backward<decltype(mask)::value>; });
  CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AdjBackShared)));
  kernel<<<blocksFor(nObj, kAdjObjs), kAdjBwdThreads, sizeof(AdjBackShared), c->st>>>(
      A.bc, A.aom, nObj, s0, s1, A.eph, c->pc, A.rec, A.arg, A.seed, s1 == A.steps, A.grad);
  CK(cudaGetLastError());
  return LADDS_OK;
}

}  // namespace

extern "C" {

int ladds_gpu_adjoint_forward(ladds_gpu_ctx *c, const ladds_adjoint_pair *pairs, size_t nPairs, int steps,
                              int checkpointEvery, double *missSq, int32_t *tcaStep, double *loss,
                              double *deviceMs) {
  if (!c || (nPairs && !pairs) || steps < 1 || checkpointEvery < 1 || nPairs > (size_t)(1 << 29))
    return fail(c, LADDS_ERR_INVALID_ARG, "adjoint_forward: bad argument");
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  auto &A = c->adj;
  A.forwardDone = false;
  const size_t nObj = 2 * nPairs;
  int rc = adjPrepare(c, nPairs, steps);
  if (rc || (rc = adjStorage(c, nObj, steps, checkpointEvery))) return rc;
  A.nPairs = nPairs;
  A.steps = steps;
  A.ck = checkpointEvery;
  // pairs (AoS) -> object SoA
  std::vector<double> st(6 * nObj), bc(nObj), aom(nObj);
  for (size_t p = 0; p < nPairs; ++p) {
    const ladds_adjoint_pair &q = pairs[p];
    for (int k = 0; k < 3; ++k) {
      st[k * nObj + 2 * p] = q.rA[k];
      st[(3 + k) * nObj + 2 * p] = q.vA[k];
      st[k * nObj + 2 * p + 1] = q.rB[k];
      st[(3 + k) * nObj + 2 * p + 1] = q.vB[k];
    }
    bc[2 * p] = q.bcInvA;
    bc[2 * p + 1] = q.bcInvB;
    aom[2 * p] = q.aomA;
    aom[2 * p + 1] = q.aomB;
  }
  if (nObj) {
    CK(cudaMemcpyAsync(A.st, st.data(), st.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(A.bc, bc.data(), bc.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(A.aom, aom.data(), aom.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
  }
  if ((rc = adjEphemeris(c, steps))) return rc;
  CK(cudaEventRecord(c->callStart, c->st));
  if (nObj) adjForward(c, A.st, (int)nObj, 0, steps, true, A.whole ? A.rec : nullptr);
  A.ckptDone = !A.whole;
  CK(cudaEventRecord(c->callEnd, c->st));
  CK(cudaGetLastError());
  std::vector<double> miss(nPairs);
  std::vector<int> arg(nPairs);
  if (nPairs) {
    CK(cudaMemcpyAsync(miss.data(), A.miss, nPairs * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(arg.data(), A.arg, nPairs * sizeof(int), cudaMemcpyDeviceToHost, c->st));
  }
  CK(cudaStreamSynchronize(c->st));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, c->callStart, c->callEnd));
  if (deviceMs) *deviceMs = ms;
  double sum = 0.0;
  for (size_t p = 0; p < nPairs; ++p) {
    if (missSq) missSq[p] = miss[p];
    if (tcaStep) tcaStep[p] = arg[p];
    if (arg[p] > 0) sum += miss[p];
  }
  if (loss) *loss = sum;
  A.forwardDone = true;
  return LADDS_OK;
}

int ladds_gpu_adjoint_backward(ladds_gpu_ctx *c, double *dL_dx0, double *dL_dbc, double *deviceMs) {
  if (!c || !dL_dx0 || !dL_dbc) return fail(c, LADDS_ERR_INVALID_ARG, "adjoint_backward: null output");
  auto &A = c->adj;
  if (!A.forwardDone) return fail(c, LADDS_ERR_STATE, "adjoint_backward needs a preceding adjoint_forward");
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  const size_t nObj = 2 * A.nPairs;
  int rc = LADDS_OK;
  const bool again = !A.whole && !A.ckptDone;  // the records have given way: the forward sweep again, for checkpoints
  if (again && (rc = adjCheckpoints(c, nObj, A.steps, A.ck))) return rc;
  const int segment = A.whole ? A.steps : std::min(A.ck, A.steps);  // the records last: a buffer taken after them could free them
  if ((rc = ensureDev(c, A.rec, A.recCap, (size_t)segment * kAdjRecord * nObj))) return rc;
  CK(cudaEventRecord(c->callStart, c->st));
  if (again && nObj) adjForward(c, A.st, (int)nObj, 0, A.steps, true, nullptr);
  A.ckptDone = !A.whole;
  for (int s1 = A.steps; nObj && s1 > 0;) {
    const int s0 = (s1 - 1) / segment * segment;
    if (!A.whole) adjForward(c, A.ckpt + (size_t)(s0 / segment) * 6 * nObj, (int)nObj, s0, s1, false, A.rec);
    if ((rc = adjBackward(c, (int)nObj, s0, s1))) return rc;
    s1 = s0;
  }
  CK(cudaEventRecord(c->callEnd, c->st));
  CK(cudaGetLastError());
  std::vector<double> g(7 * nObj);
  if (nObj) CK(cudaMemcpyAsync(g.data(), A.grad, g.size() * sizeof(double), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, c->callStart, c->callEnd));
  if (deviceMs) *deviceMs = ms;
  for (size_t p = 0; p < A.nPairs; ++p) {
    for (int k = 0; k < 6; ++k) {
      dL_dx0[12 * p + k] = g[k * nObj + 2 * p];
      dL_dx0[12 * p + 6 + k] = g[k * nObj + 2 * p + 1];
    }
    dL_dbc[2 * p] = g[6 * nObj + 2 * p];
    dL_dbc[2 * p + 1] = g[6 * nObj + 2 * p + 1];
  }
  return LADDS_OK;
}

int ladds_gpu_adjoint_make_pairs(ladds_gpu_ctx *c, uint64_t seed, size_t nPairs, int steps,
                                 ladds_adjoint_pair *out, int32_t *tcaStep) {
  if (!c || (nPairs && !out) || steps < 2 || nPairs > (size_t)(1 << 29))
    return fail(c, LADDS_ERR_INVALID_ARG, "adjoint_make_pairs: bad argument");
  std::lock_guard<std::mutex> lk(g_deviceMutex[c->dev & 63]);
  CK(cudaSetDevice(c->dev));
  auto &A = c->adj;
  A.forwardDone = false;
  int rc = adjPrepare(c, nPairs, steps);
  if (rc) return rc;
  const size_t nObj = 2 * nPairs;
  std::vector<double> st(6 * nObj), bc(nObj), aom(nObj), off(6 * nPairs);
  std::vector<int> tca(nPairs);
  for (size_t p = 0; p < nPairs; ++p) {
    double sa[6], sb[6], dr[3], dv[3];
    adjointPairDraw(seed, p, c->cfg.deltaT, steps, sa, sb, bc[2 * p], aom[2 * p], bc[2 * p + 1], aom[2 * p + 1],
                    dr, dv, tca[p]);
    for (int k = 0; k < 6; ++k) {
      st[k * nObj + 2 * p] = sa[k];
      st[k * nObj + 2 * p + 1] = sb[k];
    }
    for (int k = 0; k < 3; ++k) {
      off[6 * p + k] = dr[k];
      off[6 * p + 3 + k] = dv[k];
    }
  }
  int *dTca = A.arg;  // the forward's argmin buffer serves as scratch here
  if (nObj) {
    CK(cudaMemcpyAsync(A.st, st.data(), st.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(A.bc, bc.data(), bc.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(A.aom, aom.data(), aom.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(A.off, off.data(), off.size() * sizeof(double), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(dTca, tca.data(), tca.size() * sizeof(int), cudaMemcpyHostToDevice, c->st));
  }
  if ((rc = adjEphemeris(c, steps))) return rc;
  PropConsts back = c->pc;
  back.hc1 = -back.hc1;
  back.hc2 = -back.hc2;
  back.hd1 = -back.hd1;
  back.hd2 = -back.hd2;
  if (nPairs)
    k_adj_make_pairs<<<blocksFor(nPairs, 128), 128, 0, c->st>>>(A.st, A.bc, A.aom, (int)nPairs, dTca, A.off, A.eph,
                                                                c->pc, back);
  CK(cudaGetLastError());
  if (nObj) CK(cudaMemcpyAsync(st.data(), A.st, st.size() * sizeof(double), cudaMemcpyDeviceToHost, c->st));
  CK(cudaStreamSynchronize(c->st));
  for (size_t p = 0; p < nPairs; ++p) {
    ladds_adjoint_pair &q = out[p];
    for (int k = 0; k < 3; ++k) {
      q.rA[k] = st[k * nObj + 2 * p];
      q.vA[k] = st[(3 + k) * nObj + 2 * p];
      q.rB[k] = st[k * nObj + 2 * p + 1];
      q.vB[k] = st[(3 + k) * nObj + 2 * p + 1];
    }
    q.bcInvA = bc[2 * p];
    q.bcInvB = bc[2 * p + 1];
    q.aomA = aom[2 * p];
    q.aomB = aom[2 * p + 1];
    if (tcaStep) tcaStep[p] = tca[p];
  }
  return LADDS_OK;
}

}  // extern "C"

// ----------------------------------------------------------------------------
// Cell sort without allocation (ladds_gpu_cell_sort_noalloc).
//
// For callers that cannot allocate device memory: processes in which another
// framework's caching allocator (JAX, PyTorch) has reserved nearly all of HBM,
// so that cudaMalloc fails, and callers on a per-iteration latency path that
// cannot take the implicit device synchronisation of cudaMalloc / cudaFree.
// All scratch of the sort (row counts and cursors, row-start table, sort
// records, long-row list, scan partial sums, status word)
// lives in one file-scope device array of fixed size; the caller supplies the
// keys and the output buffers.  Every call shares the array and it keeps the
// last call's contents, so each call clears what must start at zero, and calls
// that overlap on the GPU (other streams, other host threads) race.
namespace {

constexpr size_t naRound(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t kNaMaxObjects = LADDS_NOALLOC_SORT_MAX_OBJECTS;
constexpr size_t kNaMaxRows = LADDS_NOALLOC_SORT_MAX_ROWS;
constexpr size_t kNaScanBlocks = (kNaMaxRows + 1 + kScanBlock - 1) / kScanBlock;
static_assert(kNaScanBlocks <= (size_t)kScanBlock, "two scan levels must cover the row table");
// byte offsets inside the scratch array
constexpr size_t kNaRec = 0;                                                   // u64 per object
constexpr size_t kNaCounts = kNaRec + naRound(8 * kNaMaxObjects);              // counts | cursors
constexpr size_t kNaRowStart = kNaCounts + naRound(8 * (kNaMaxRows + 1));      // u32 per row + 1
constexpr size_t kNaLong = kNaRowStart + naRound(4 * (kNaMaxRows + 1));        // long-row list
constexpr size_t kNaMisc = kNaLong + naRound(4 * kNaMaxRows);                  // longCount, status
constexpr size_t kNaScan = kNaMisc + 256;                                      // scan partial sums
constexpr size_t kNaBytes = kNaScan + naRound(4 * (2 * (kNaScanBlocks + 1) + 2));

static __device__ __align__(256) unsigned char g_noallocSortScratch[kNaBytes];

struct NaDevice {
  unsigned char *scratch = nullptr;  // device address of g_noallocSortScratch on this device
  int sms = 0;
};
NaDevice g_naDevice[64];
std::mutex g_naMutex;

void naMessage(char *msg, size_t cap, const char *text) {
  if (msg && cap) std::snprintf(msg, cap, "%s", text);
}

// status bits: 1 = a key beyond the grid, 2 = inconsistent row counts
__global__ void __launch_bounds__(kBucketThreads) k_na_count(const uint32_t *__restrict__ keys, int n, uint32_t nx,
                                                             uint32_t nRows, uint32_t *__restrict__ rowCount,
                                                             unsigned *__restrict__ status) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t row = 0xffffffffu;
  if (j < n) {
    row = keys[j] / nx;
    if (row >= nRows) {
      atomicOr(status, 1u);
      row = 0xffffffffu;
    }
  }
  const bool valid = row != 0xffffffffu;
  const uint32_t peers = __match_any_sync(0xffffffffu, row);
  if (valid && (__ffs(peers) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&rowCount[row], (uint32_t)__popc(peers));
}

// sort record ix << 32 | j of every object j (the index in keys)
__global__ void __launch_bounds__(kBucketThreads) k_na_scatter(const uint32_t *__restrict__ keys, int n, uint32_t nx,
                                                               uint32_t nRows, const uint32_t *__restrict__ rowStart,
                                                               uint32_t *__restrict__ rowCursor,
                                                               unsigned long long *__restrict__ rec,
                                                               unsigned *__restrict__ status) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const uint32_t key = j < n ? keys[j] : 0u;
  uint32_t row = j < n ? key / nx : 0xffffffffu;
  if (row >= nRows) row = 0xffffffffu;  // counted as an error by k_na_count
  const bool valid = row != 0xffffffffu;
  const uint32_t peers = __match_any_sync(0xffffffffu, row);
  const int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (valid && lane == leader) base = atomicAdd(&rowCursor[row], (uint32_t)__popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (!valid) return;
  const uint32_t pos = rowStart[row] + base + (uint32_t)__popc(peers & laneMaskLt());
  if (pos >= rowStart[row + 1]) {
    atomicOr(status, 2u);
    return;
  }
  rec[pos] = ((unsigned long long)(key - row * nx) << 32) | (uint32_t)j;
}

struct DeviceGuard {
  int prev = -1;
  cudaError_t status;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    status = cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

}  // namespace

extern "C" {

int ladds_gpu_cell_sort_noalloc(int device, void *stream, const uint32_t *keys, size_t n, const int32_t dims[3],
                                uint32_t *sortedKeys, uint32_t *order, uint32_t *rowStart, char *errMsg,
                                size_t errMsgCap) {
  naMessage(errMsg, errMsgCap, "");
  if (!dims || device < 0 || device >= 64 || (n && (!keys || !sortedKeys || !order))) {
    naMessage(errMsg, errMsgCap, "invalid argument: null pointer or device index");
    return LADDS_ERR_INVALID_ARG;
  }
  if (dims[0] < 1 || dims[1] < 1 || dims[2] < 1 ||
      (uint64_t)dims[0] * (uint64_t)dims[1] * (uint64_t)dims[2] > (1ull << 32)) {
    naMessage(errMsg, errMsgCap, "invalid argument: grid dimensions must be >= 1 with at most 2^32 cells");
    return LADDS_ERR_INVALID_ARG;
  }
  const uint64_t nRows64 = (uint64_t)dims[1] * (uint64_t)dims[2];
  if (n > kNaMaxObjects || nRows64 > kNaMaxRows) {
    char text[160];
    std::snprintf(text, sizeof(text),
                  "too large: %zu objects and %llu cell rows exceed the fixed scratch maximum of %zu objects / "
                  "%zu rows",
                  n, (unsigned long long)nRows64, kNaMaxObjects, kNaMaxRows);
    naMessage(errMsg, errMsgCap, text);
    return LADDS_ERR_TOO_LARGE;
  }
  // an error that earlier work left in this thread's CUDA state is not this
  // call's: report it without clearing it
  if (const cudaError_t pending = cudaPeekAtLastError(); pending != cudaSuccess) {
    char text[200];
    std::snprintf(text, sizeof(text), "a CUDA error of earlier work is pending (not cleared): %s",
                  cudaGetErrorString(pending));
    naMessage(errMsg, errMsgCap, text);
    return LADDS_ERR_CUDA;
  }
  DeviceGuard guard(device);
  if (guard.status != cudaSuccess) {
    cudaGetLastError();
    naMessage(errMsg, errMsgCap, cudaGetErrorString(guard.status));
    return guard.status == cudaErrorInvalidDevice || guard.status == cudaErrorNoDevice ? LADDS_ERR_NO_DEVICE
                                                                                        : LADDS_ERR_CUDA;
  }
  // the call waits for its stream and reads a status word back: it cannot be
  // part of a stream capture
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (const cudaError_t ce = cudaStreamIsCapturing(s, &capturing); ce != cudaSuccess) {
    cudaGetLastError();
    naMessage(errMsg, errMsgCap, cudaGetErrorString(ce));
    return LADDS_ERR_CUDA;
  }
  if (capturing != cudaStreamCaptureStatusNone) {
    naMessage(errMsg, errMsgCap, "invalid argument: the stream is capturing; this call synchronises its stream");
    return LADDS_ERR_INVALID_ARG;
  }
  NaDevice &d = g_naDevice[device];
  {
    std::lock_guard<std::mutex> lk(g_naMutex);
    if (!d.scratch) {  // set-up, once per device, with that device current
      int sms = 0;
      unsigned char *ptr = nullptr;
      const cudaError_t e1 = cudaGetSymbolAddress((void **)&ptr, g_noallocSortScratch);
      const cudaError_t e2 = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
      if (e1 != cudaSuccess || e2 != cudaSuccess || !ptr) {
        cudaGetLastError();
        naMessage(errMsg, errMsgCap, cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
        return LADDS_ERR_CUDA;
      }
      d.sms = std::max(sms, 1);
      d.scratch = ptr;
    }
  }
  const uint32_t nx = (uint32_t)dims[0], nRows = (uint32_t)nRows64;
  auto *rec = reinterpret_cast<unsigned long long *>(d.scratch + kNaRec);
  auto *rowCount = reinterpret_cast<uint32_t *>(d.scratch + kNaCounts);
  uint32_t *rowCursor = rowCount + nRows + 1;
  auto *rowStartS = reinterpret_cast<uint32_t *>(d.scratch + kNaRowStart);
  auto *longRows = reinterpret_cast<uint32_t *>(d.scratch + kNaLong);
  auto *longCount = reinterpret_cast<uint32_t *>(d.scratch + kNaMisc);
  auto *status = reinterpret_cast<unsigned *>(d.scratch + kNaMisc + 4);
  auto *s1 = reinterpret_cast<uint32_t *>(d.scratch + kNaScan);
  uint32_t *s1x = s1 + kNaScanBlocks + 1, *s2 = s1x + kNaScanBlocks + 1;

  const CellOrderOut out{sortedKeys, order, nullptr, nullptr, nullptr, nullptr, nullptr};

  // every enqueue is checked where it is made; on a failure the stream is
  // drained before returning, so that no copy of this call is still running
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t r) {
    if (e == cudaSuccess && r != cudaSuccess) e = r;
    return e == cudaSuccess;
  };
  ok(cudaMemsetAsync(rowCount, 0, 2 * ((size_t)nRows + 1) * sizeof(uint32_t), s));
  ok(cudaMemsetAsync(longCount, 0, 2 * sizeof(uint32_t), s));  // longCount and status
  if (e == cudaSuccess && n) {
    const int gridN = blocksFor(n, kBucketThreads);
    k_na_count<<<gridN, kBucketThreads, 0, s>>>(keys, (int)n, nx, nRows, rowCount, status);
    ok(cudaGetLastError());
  }
  const size_t count = (size_t)nRows + 1;
  const int nb1 = blocksFor(count, kScanBlock);
  if (e == cudaSuccess) {
    k_scan_blocks<<<nb1, kScanBlock, 0, s>>>(rowCount, (int)count, rowStartS, s1);
    ok(cudaGetLastError());
  }
  if (e == cudaSuccess && nb1 > 1) {
    k_scan_blocks<<<1, kScanBlock, 0, s>>>(s1, nb1, s1x, s2);
    if (ok(cudaGetLastError())) {
      k_scan_add<<<nb1, kScanBlock, 0, s>>>(rowStartS, (int)count, s1x);
      ok(cudaGetLastError());
    }
  }
  if (e == cudaSuccess && n) {
    const int gridN = blocksFor(n, kBucketThreads);
    k_na_scatter<<<gridN, kBucketThreads, 0, s>>>(keys, (int)n, nx, nRows, rowStartS, rowCursor, rec, status);
    if (ok(cudaGetLastError())) {
      const int smallBlocks = std::min(blocksFor((size_t)nRows * 32, kBucketThreads), 64 * d.sms);
      k_bucket_sort_small<<<smallBlocks, kBucketThreads, 0, s>>>(rowStartS, nRows, nx, rec, out, longRows, longCount,
                                                                 nullptr);
    }
    if (ok(cudaGetLastError())) {
      k_bucket_sort_large<<<2 * d.sms, kBucketThreads, kLargeRow * 8, s>>>(
          rowStartS, nx, rec, out, longRows, longCount, nullptr, DenseBin{nullptr, nullptr, 0, 0, nullptr});
      ok(cudaGetLastError());
    }
  }
  if (e == cudaSuccess && rowStart)
    ok(cudaMemcpyAsync(rowStart, rowStartS, count * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  unsigned hostStatus = 0;
  if (e == cudaSuccess) ok(cudaMemcpyAsync(&hostStatus, status, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  const cudaError_t es = cudaStreamSynchronize(s);  // also on a failure: nothing of this call left running
  ok(es);
  if (e != cudaSuccess) {
    cudaGetLastError();
    naMessage(errMsg, errMsgCap, cudaGetErrorString(e));
    return LADDS_ERR_CUDA;
  }
  if (hostStatus & 1u) {
    naMessage(errMsg, errMsgCap, "invalid argument: a key lies beyond the grid (key >= dims[0]*dims[1]*dims[2])");
    return LADDS_ERR_INVALID_ARG;
  }
  if (hostStatus) {
    naMessage(errMsg, errMsgCap, "device check: inconsistent row counts");
    return LADDS_ERR_DEVICE_CHECK;
  }
  return LADDS_OK;
}

}  // extern "C"
