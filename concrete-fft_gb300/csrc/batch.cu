// batch.cu -- mixed-size c64 transforms in a few persistent launches.
//
// A batch is a list of transforms of different power-of-two sizes and kinds
// (ordered n <= 1024, unordered n <= 65536) living anywhere in one device
// buffer.  At creation the host groups the items by (kind, size, direction)
// into work units of `tpc` same-size transforms, orders the units longest
// first, and picks each size class's schedule (base algorithm, base size,
// transforms per unit) by timing candidates on the device.  Transforms above
// 2048 points are cut up: their outer levels into units of 4096 points of
// butterflies in global memory, the sub-transforms below into units of 2048
// points like the small transforms.  A run is one persistent kernel per phase
// (forward levels, one launch each; everything that fits shared memory; inverse
// levels): every CTA takes the next unit from a device counter (atomicAdd, no
// waiting on other CTAs) until the queue is empty.  So a batch takes the time of
// its work and not that of its largest transform on one CTA (300 items of 256 to
// 65536 points, forward and inverse: 2578 us with a unit per item).  Runs on a
// user stream are replayed from a CUDA graph captured on the first run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "../../include/cfft.h"
#include "cfft_internal.h"
#include "runtime.h"
#include "stockham.cuh"

using namespace cfft;

namespace cfft {

constexpr int kBatchSmemLog2 = 11;  // 2048 points x 2 buffers x 16 B = 64 KiB per CTA
constexpr int kBatchThreads = 256;

struct SizeClass {
  DevLevels L;
  const double2* w;
  const double2* winv;
  int algo;  // 2 (Dif4) or 4 (Dif8): the base algorithms compiled into the persistent kernel
  int d0;    // first level handled in shared memory
  int log2n;
};

struct Unit {
  uint16_t cls;
  uint8_t count;  // transforms in this unit (<= tpc of the class), or sub-transforms of one
  uint8_t dir;    // 1 forward, 2 inverse, 3 forward then inverse
  int first;      // index into the sorted item-offset array
  int level;      // outer level in global memory, or -1: transforms in shared memory
  int part;       // which part of the level, or the first sub-transform
};
constexpr int kLevelUnitLog2 = 12;  // points of an outer level per unit

// Butterflies [part, part + 1) * 2^kLevelUnitLog2 / r of outer level l of the transform at g.
template <bool FWD>
__device__ void run_level(double2* g, const SizeClass& C, int l, int part, int tid, int nth) {
  const int log2r = C.L.log2r[l], lm = C.L.log2n[l] - log2r;
  const double2* wl = FWD ? C.w + C.L.w_off[l] : C.winv + C.L.winv_off[l];
  const int per = 1 << (min(kLevelUnitLog2, C.log2n) - log2r);
  for (int b = part * per + tid; b < (part + 1) * per; b += nth) {
    double2* zc = g + ((long)(b >> lm) << C.L.log2n[l]);
    const int i = b & ((1 << lm) - 1);
    if (log2r == 1) outer_group<2, FWD, kAddsBatch>(zc, lm, i, wl);
    else if (log2r == 2) outer_group<4, FWD, kAddsBatch>(zc, lm, i, wl);
    else outer_group<8, FWD, kAddsBatch>(zc, lm, i, wl);
  }
}

template <int ALGO>
__device__ void run_unit(double2* __restrict__ data, const SizeClass& C, const uint64_t* __restrict__ offs,
                         const Unit& U, double2* x, double2* y, int tid, int nth) {
  const int log2sub = C.L.log2n[C.d0];
  const bool fwd = U.dir & 1, inv = (U.dir & 2) != 0;
  const int n = 1 << log2sub;
  // whole transforms (d0 = 0), or consecutive sub-transforms of one, back to back
  const long step = C.d0 == 0 ? 0 : 1;
  for (int t = 0; t < U.count; ++t) {
    const double2* g = data + offs[U.first + (step ? 0 : t)] + ((long)(step ? U.part + t : 0) << log2sub);
    for (int i = tid; i < n; i += nth) x[(t << log2sub) + i] = g[i];
  }
  __syncthreads();
  double2* r = x;
  if (fwd) r = unordered_smem<true, kAddsBatch, ALGO>(C.L, C.d0, U.count, x, y, C.w, tid, nth);
  if (inv) r = unordered_smem<false, kAddsBatch, ALGO>(C.L, C.d0, U.count, r, r == x ? y : x, C.winv, tid, nth);
  for (int t = 0; t < U.count; ++t) {
    double2* g = data + offs[U.first + (step ? 0 : t)] + ((long)(step ? U.part + t : 0) << log2sub);
    for (int i = tid; i < n; i += nth) g[i] = r[(t << log2sub) + i];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kBatchThreads, 3) batch_kernel(double2* __restrict__ data,
                                                             const SizeClass* __restrict__ classes,
                                                             const uint64_t* __restrict__ offs,
                                                             const Unit* __restrict__ units, int nunits,
                                                             unsigned int* __restrict__ head) {
  extern __shared__ double2 smem[];
  __shared__ int s_unit;
  double2* x = smem;
  double2* y = smem + (1 << kBatchSmemLog2);
  const int tid = threadIdx.x, nth = blockDim.x;
  for (;;) {
    if (tid == 0) s_unit = (int)atomicAdd(head, 1u);
    __syncthreads();
    const int u = s_unit;
    __syncthreads();
    if (u >= nunits) break;
    const Unit U = units[u];
    const SizeClass C = classes[U.cls];
    if (U.level >= 0) {
      double2* g = data + offs[U.first];
      if (U.dir == 1) run_level<true>(g, C, U.level, U.part, tid, nth);
      else run_level<false>(g, C, U.level, U.part, tid, nth);
    } else if (C.algo == 2) run_unit<2>(data, C, offs, U, x, y, tid, nth);
    else run_unit<4>(data, C, offs, U, x, y, tid, nth);
  }
}

}  // namespace cfft

// ============================================================ host side
namespace {

struct ClassKey {
  int kind, log2n, dir;
  bool operator<(const ClassKey& o) const { return std::tie(kind, log2n, dir) < std::tie(o.kind, o.log2n, o.dir); }
};

struct ClassHost {
  ClassKey key;
  int algo = 2, base_log2 = 10, tpc = 1;
  double2 *w = nullptr, *winv = nullptr;
  std::vector<uint64_t> items;  // offsets (points)
};

void free_tables(ClassHost& c) {
  if (c.w) cudaFree(c.w);
  if (c.winv) cudaFree(c.winv);
  c.w = c.winv = nullptr;
}

cfft_status build_tables(ClassHost& c) {
  free_tables(c);
  const size_t n = size_t(1) << c.key.log2n, base = size_t(1) << c.base_log2;
  std::vector<c64h> w(n + base), wi(n + base);
  unordered_twiddles(n, base, algo_radix(c.algo), w.data(), wi.data());
  cfft_status st = upload((const double2*)w.data(), n + base, &c.w);
  if (st == CFFT_OK) st = upload((const double2*)wi.data(), n + base, &c.winv);
  return st;
}

SizeClass device_class(const ClassHost& c) {
  const size_t n = size_t(1) << c.key.log2n, base = size_t(1) << c.base_log2;
  const LevelDesc lv = make_levels(n, base);
  SizeClass d;
  std::memset(&d, 0, sizeof(d));
  d.L.nlevels = lv.nlevels;
  for (int i = 0; i <= kMaxLevels; ++i) {
    d.L.log2n[i] = lv.log2n[i];
    d.L.w_off[i] = lv.w_off[i];
  }
  for (int i = 0; i < kMaxLevels; ++i) {
    d.L.log2r[i] = lv.log2r[i];
    d.L.winv_off[i] = lv.winv_off[i];
  }
  d.w = c.w;
  d.winv = c.winv;
  d.algo = c.algo;
  d.log2n = c.key.log2n;
  d.d0 = 0;
  while (lv.log2n[d.d0] > kBatchSmemLog2) ++d.d0;
  return d;
}

// The units of one launch of each phase of a run: forward levels 0, 1, ..., the
// transforms in shared memory, inverse levels ..., 1, 0.
struct Phases {
  std::vector<Unit> units;   // of all phases, in order
  std::vector<int> count;    // units per phase
};
constexpr int kMaxPhases = 2 * kMaxLevels + 1;

// The units of one class in one phase, all of about the same cost (relative work of one).
struct UnitGroup {
  double cost;
  std::vector<Unit> units;
};
using PhaseGroups = std::vector<UnitGroup>[kMaxPhases];

// Adds the units of one class whose items are offs[first .. first + items).
void add_units(const ClassHost& c, const SizeClass& d, int cls, int first, size_t items, PhaseGroups& per) {
  const int log2sub = d.L.log2n[d.d0];
  const double passes = c.key.dir == 3 ? 2 : 1;
  const uint16_t cl = (uint16_t)cls;
  const uint8_t dir = (uint8_t)c.key.dir;
  if (d.d0 == 0) {
    UnitGroup g{(double)c.tpc * (double)(1L << log2sub) * log2sub * passes, {}};
    g.units.reserve(items / (size_t)c.tpc + 1);
    for (size_t k = 0; k < items; k += (size_t)c.tpc)
      g.units.push_back(Unit{cl, (uint8_t)std::min<size_t>(c.tpc, items - k), dir, first + (int)k, -1, 0});
    per[kMaxLevels].push_back(std::move(g));
    return;
  }
  const int nsub = 1 << (d.log2n - log2sub), group = std::min(nsub, 1 << (kBatchSmemLog2 - log2sub));
  const int parts = 1 << std::max(0, d.log2n - kLevelUnitLog2);
  UnitGroup g{(double)group * (double)(1L << log2sub) * log2sub * passes, {}};
  g.units.reserve(items * (size_t)(nsub / group));
  for (size_t k = 0; k < items; ++k)
    for (int t = 0; t < nsub; t += group) g.units.push_back(Unit{cl, (uint8_t)group, dir, first + (int)k, -1, t});
  per[kMaxLevels].push_back(std::move(g));
  for (int l = 0; l < d.d0; ++l)
    for (int way : {1, 2}) {
      if (!(c.key.dir & way)) continue;
      UnitGroup lg{(double)d.L.log2r[l], {}};
      lg.units.reserve(items * (size_t)parts);
      for (size_t k = 0; k < items; ++k)
        for (int p = 0; p < parts; ++p) lg.units.push_back(Unit{cl, 1, (uint8_t)way, first + (int)k, l, p});
      per[way == 1 ? l : 2 * kMaxLevels - l].push_back(std::move(lg));
    }
}

// Longest units first in each phase.
Phases order_units(PhaseGroups& per) {
  Phases ph;
  for (auto& groups : per) {
    if (groups.empty()) continue;
    std::stable_sort(groups.begin(), groups.end(), [](const UnitGroup& x, const UnitGroup& y) { return x.cost > y.cost; });
    const size_t before = ph.units.size();
    for (const UnitGroup& g : groups) ph.units.insert(ph.units.end(), g.units.begin(), g.units.end());
    ph.count.push_back((int)(ph.units.size() - before));
  }
  return ph;
}

cfft_status batch_attr() {
  return ensure_smem((const void*)batch_kernel, 2 * (1 << kBatchSmemLog2) * sizeof(double2));
}

}  // namespace

struct cfft_batch {
  std::vector<ClassHost> classes;
  size_t units = 0;
  std::vector<int> phase;  // units of each launch
  SizeClass* d_classes = nullptr;
  uint64_t* d_offs = nullptr;
  Unit* d_units = nullptr;
  unsigned int* d_head = nullptr;  // one counter per phase
  int grid = 0;
  size_t total_points = 0;
  // graph cache: one captured launch per (stream, data pointer)
  std::mutex mu;
  cudaStream_t g_stream = nullptr;
  double* g_data = nullptr;
  cudaGraphExec_t g_exec = nullptr;
  // pipelined host runs: the items split into data-contiguous chunks, each
  // with its own units and work counter (built on first use)
  struct Chunk {
    uint64_t lo = 0, hi = 0;  // point range [lo, hi) covered by the chunk's items
    uint64_t* d_offs = nullptr;
    Unit* d_units = nullptr;
    std::vector<int> phase;
  };
  std::vector<cfft_batch_item> items;
  std::vector<Chunk> chunks;
  unsigned int* d_heads = nullptr;
  cudaStream_t pstream[3] = {};
  cudaEvent_t pevent[4] = {};
};

namespace {

cfft_status launch_phases(cfft_batch* b, double2* data, const uint64_t* offs, const Unit* units,
                          const std::vector<int>& phase, unsigned int* heads, cudaStream_t s) {
  CFFT_CUDA_TRY(cudaMemsetAsync(heads, 0, kMaxPhases * sizeof(unsigned int), s));
  const size_t smem = 2 * (1 << kBatchSmemLog2) * sizeof(double2);
  for (size_t p = 0; p < phase.size(); ++p) {
    batch_kernel<<<std::min(b->grid, phase[p]), kBatchThreads, smem, s>>>(data, b->d_classes, offs, units, phase[p],
                                                                         heads + p);
    units += phase[p];
  }
  CFFT_CHECK_LAUNCH();
  return CFFT_OK;
}
cfft_status launch_batch(cfft_batch* b, double2* data, cudaStream_t s) {
  return launch_phases(b, data, b->d_offs, b->d_units, b->phase, b->d_head, s);
}

void free_batch_device(cfft_batch* b) {
  if (b->d_classes) cudaFree(b->d_classes);
  if (b->d_offs) cudaFree(b->d_offs);
  if (b->d_units) cudaFree(b->d_units);
  b->d_classes = nullptr;
  b->d_offs = nullptr;
  b->d_units = nullptr;
}

// Builds units and uploads class descriptors, offsets and units.
cfft_status finalize(cfft_batch* b) {
  free_batch_device(b);
  std::vector<uint64_t> offs;
  std::vector<SizeClass> dcls;
  PhaseGroups per;
  for (size_t ci = 0; ci < b->classes.size(); ++ci) {
    ClassHost& c = b->classes[ci];
    dcls.push_back(device_class(c));
    const int first = (int)offs.size();
    offs.insert(offs.end(), c.items.begin(), c.items.end());
    add_units(c, dcls.back(), (int)ci, first, c.items.size(), per);
  }
  const Phases ph = order_units(per);
  b->units = ph.units.size();
  b->phase = ph.count;
  cfft_status st = upload(dcls.data(), dcls.size(), &b->d_classes);
  if (st == CFFT_OK) st = upload(offs.data(), offs.size(), &b->d_offs);
  if (st == CFFT_OK) st = upload(ph.units.data(), ph.units.size(), &b->d_units);
  return st;
}

// FP64 operations (additions, products, FMAs) of one unordered transform of 2^log2n points
// with the given base, wherever they run: the outer levels' radix-r butterflies plus r - 1 twiddle
// products each, the base's radix-R passes likewise, and its end butterfly.
double fp64_ops_per_point(int log2n, int base_log2, int algo) {
  auto core = [](int r) { return r == 2 ? 4.0 : r == 4 ? 16.0 : r == 8 ? 56.0 : 168.0; };
  const LevelDesc lv = make_levels(size_t(1) << log2n, size_t(1) << base_log2);
  double ops = 0;
  for (int l = 0; l < lv.nlevels; ++l) {
    const int r = 1 << lv.log2r[l];
    ops += (core(r) + 4.0 * (r - 1)) / r;
  }
  const int lr = ilog2((size_t)algo_radix(algo));
  int rem = base_log2;
  while (rem > lr) {
    rem -= lr;
    ops += (core(1 << lr) + 4.0 * ((1 << lr) - 1)) / (1 << lr);
  }
  if (rem > 0) ops += core(1 << rem) / (1 << rem);
  return ops;
}

// Times candidate schedules of one size class on a synthetic homogeneous batch.
// Among candidates timed within 3% of the fastest (short timings are that noisy)
// the one with the fewest FP64 operations per point wins, so that the choice
// does not hang on the noise, and the time decides between equal counts.
cfft_status tune_class(cfft_batch* b, size_t ci, double seconds) {
  ClassHost& c = b->classes[ci];
  const int log2n = c.key.log2n;
  std::vector<std::tuple<int, int, int>> cands;  // (algo, base_log2, tpc)
  std::vector<int> bases;
  if (c.key.kind == 0) bases.push_back(log2n);  // ordered: the base is the transform
  else
    for (int bl : {9, 10})
      if (bl <= log2n) bases.push_back(bl);
  if (bases.empty()) bases.push_back(log2n);
  for (int bl : bases)
    for (int algo : {2, 4})
      for (int tpc : {1, 2, 4, 8}) {
        if (log2n > kBatchSmemLog2 && tpc > 1) continue;
        if (log2n <= kBatchSmemLog2 && (tpc << log2n) > (1 << kBatchSmemLog2)) continue;
        cands.emplace_back(algo, bl, tpc);
      }
  const size_t n = size_t(1) << log2n;
  const size_t count = std::max<size_t>(b->grid * 2, (size_t(1) << 21) >> log2n);  // >= 2 units per CTA
  double2* buf = nullptr;
  CFFT_CUDA_TRY(cudaMalloc(&buf, count * n * sizeof(double2)));
  cfft_batch tb;
  tb.grid = b->grid;
  CFFT_CUDA_TRY(cudaMalloc(&tb.d_head, kMaxPhases * sizeof(unsigned int)));
  cudaStream_t s;
  CFFT_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  std::vector<double> times;
  cfft_status st = CFFT_OK;
  for (auto cand : cands) {
    ClassHost t;
    t.key = c.key;
    std::tie(t.algo, t.base_log2, t.tpc) = cand;
    for (size_t i = 0; i < count; ++i) t.items.push_back(i * n);
    st = build_tables(t);
    if (st != CFFT_OK) break;
    tb.classes.clear();
    tb.classes.push_back(t);
    st = finalize(&tb);
    if (st != CFFT_OK) break;
    // forward and inverse grow the data by log2 n bits each
    const int most = timing_reps_max((c.key.dir == 3 ? 2 : 1) * log2n);
    fill_timing_doubles((double*)buf, 2 * count * n, kTimingScale, s);
    launch_batch(&tb, buf, s);
    int reps = 1;
    double per = 0;
    for (;;) {
      fill_timing_doubles((double*)buf, 2 * count * n, kTimingScale, s);
      cudaEventRecord(e0, s);
      for (int r = 0; r < reps; ++r) launch_batch(&tb, buf, s);
      cudaEventRecord(e1, s);
      cudaEventSynchronize(e1);
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      per = ms / reps;
      if (ms * 1e-3 >= std::max(seconds, 5e-4) || reps >= std::min(64, most)) break;
      reps = std::min(2 * reps, most);
    }
    free_tables(tb.classes[0]);
    times.push_back(per);
  }
  free_batch_device(&tb);
  cudaFree(tb.d_head);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(s);
  cudaFree(buf);
  if (st != CFFT_OK) return st;
  const double fastest = *std::min_element(times.begin(), times.end());
  size_t pick = 0;
  double pick_ops = 1e30;
  for (size_t i = 0; i < cands.size(); ++i) {
    if (times[i] > 1.03 * fastest) continue;
    const double ops = fp64_ops_per_point(log2n, std::get<1>(cands[i]), std::get<0>(cands[i]));
    if (ops < pick_ops - 1e-9 || (ops < pick_ops + 1e-9 && times[i] < times[pick])) {
      pick = i;
      pick_ops = ops;
    }
  }
  std::tie(c.algo, c.base_log2, c.tpc) = cands[pick];
  return CFFT_OK;
}

void destroy_batch(cfft_batch* b) {
  if (!b) return;
  if (b->g_exec) cudaGraphExecDestroy(b->g_exec);
  for (auto& c : b->chunks) {
    if (c.d_offs) cudaFree(c.d_offs);
    if (c.d_units) cudaFree(c.d_units);
  }
  if (b->d_heads) cudaFree(b->d_heads);
  for (cudaStream_t st : b->pstream)
    if (st) cudaStreamDestroy(st);
  for (cudaEvent_t ev : b->pevent)
    if (ev) cudaEventDestroy(ev);
  for (auto& c : b->classes) free_tables(c);
  free_batch_device(b);
  if (b->d_head) cudaFree(b->d_head);
  delete b;
}

// Splits the items, in offset order, into about kChunks groups of equal
// points; each group gets the units of its items (same classes and
// schedules as the whole batch, longest first) and its own work counter.
constexpr int kChunks = 16;
cfft_status build_chunks(cfft_batch* b) {
  std::map<ClassKey, int> cls;
  for (size_t ci = 0; ci < b->classes.size(); ++ci) cls[b->classes[ci].key] = (int)ci;
  std::vector<size_t> order(b->items.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](size_t x, size_t y) { return b->items[x].offset < b->items[y].offset; });
  const size_t target = std::max<size_t>(1, b->total_points / kChunks);
  size_t i = 0;
  while (i < order.size()) {
    size_t j = i, pts = 0;
    while (j < order.size() && (pts < target || j == i)) pts += size_t(1) << b->items[order[j++]].log2n;
    cfft_batch::Chunk ch;
    ch.lo = b->items[order[i]].offset;
    ch.hi = b->items[order[j - 1]].offset + (uint64_t(1) << b->items[order[j - 1]].log2n);
    // per class, this chunk's items in offset order
    std::vector<std::vector<uint64_t>> per(b->classes.size());
    for (size_t k = i; k < j; ++k) {
      const cfft_batch_item& it = b->items[order[k]];
      per[cls[ClassKey{(int)it.kind, (int)it.log2n, (int)it.direction}]].push_back(it.offset);
    }
    std::vector<uint64_t> offs;
    PhaseGroups by_phase;
    for (size_t ci = 0; ci < per.size(); ++ci) {
      if (per[ci].empty()) continue;
      const int first = (int)offs.size();
      offs.insert(offs.end(), per[ci].begin(), per[ci].end());
      add_units(b->classes[ci], device_class(b->classes[ci]), (int)ci, first, per[ci].size(), by_phase);
    }
    const Phases ph = order_units(by_phase);
    const std::vector<Unit>& units = ph.units;
    ch.phase = ph.count;
    b->chunks.push_back(ch);
    cfft_status st = upload(offs.data(), offs.size(), &b->chunks.back().d_offs);
    if (st == CFFT_OK) st = upload(units.data(), units.size(), &b->chunks.back().d_units);
    if (st != CFFT_OK) return st;
    i = j;
  }
  CFFT_CUDA_TRY(cudaMalloc(&b->d_heads, b->chunks.size() * kMaxPhases * sizeof(unsigned int)));
  for (cudaStream_t& st : b->pstream) CFFT_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  for (cudaEvent_t& ev : b->pevent) CFFT_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  return CFFT_OK;
}

}  // namespace

extern "C" {

cfft_status cfft_batch_create(const cfft_batch_item* items, size_t count, double tune_seconds, cfft_batch** out) {
  if (!out || (!items && count)) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  std::map<ClassKey, std::vector<uint64_t>> groups;
  size_t total = 0;
  for (size_t i = 0; i < count; ++i) {
    const cfft_batch_item& it = items[i];
    if (it.kind > 1) return fail(CFFT_ERR_INVALID_ARGUMENT, "item kind must be 0 (ordered) or 1 (unordered)");
    if (it.direction < 1 || it.direction > 3) return fail(CFFT_ERR_INVALID_ARGUMENT, "item direction must be 1..3");
    if (it.log2n > 16 || (it.kind == 0 && it.log2n > 10))
      return fail(CFFT_ERR_INVALID_SIZE, "item size out of range (ordered <= 2^10, unordered <= 2^16)");
    if (it.log2n < 1) return fail(CFFT_ERR_INVALID_SIZE, "item size must be at least 2");
    groups[ClassKey{(int)it.kind, (int)it.log2n, (int)it.direction}].push_back(it.offset);
    total += size_t(1) << it.log2n;
  }
  cfft_status st = batch_attr();
  if (st != CFFT_OK) return st;
  auto* b = new cfft_batch();
  b->total_points = total;
  b->items.assign(items, items + count);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel, kBatchThreads,
                                                2 * (1 << kBatchSmemLog2) * sizeof(double2));
  b->grid = sm_count() * std::max(per_sm, 1);
  st = cudaMalloc(&b->d_head, kMaxPhases * sizeof(unsigned int)) == cudaSuccess ? CFFT_OK : CFFT_ERR_OUT_OF_MEMORY;
  for (auto& g : groups) {
    if (st != CFFT_OK) break;
    ClassHost c;
    c.key = g.first;
    c.items = std::move(g.second);
    // default schedule: Dif4 over a base of 1024 (or the whole ordered/small transform)
    c.algo = 2;
    c.base_log2 = c.key.kind == 0 ? c.key.log2n : std::min(c.key.log2n, 10);
    c.tpc = c.key.log2n <= kBatchSmemLog2 ? std::max(1, (1 << kBatchSmemLog2) >> c.key.log2n) : 1;
    c.tpc = std::min(c.tpc, 8);
    b->classes.push_back(std::move(c));
  }
  if (st == CFFT_OK && tune_seconds > 0)
    for (size_t ci = 0; ci < b->classes.size() && st == CFFT_OK; ++ci) st = tune_class(b, ci, tune_seconds);
  for (size_t ci = 0; ci < b->classes.size() && st == CFFT_OK; ++ci) st = build_tables(b->classes[ci]);
  if (st == CFFT_OK) st = finalize(b);
  if (st != CFFT_OK) {
    destroy_batch(b);
    return st;
  }
  *out = b;
  return CFFT_OK;
}

void cfft_batch_destroy(cfft_batch* batch) { destroy_batch(batch); }

size_t cfft_batch_units(const cfft_batch* batch) { return batch ? batch->units : 0; }

cfft_status cfft_batch_schedule(const cfft_batch* batch, uint32_t kind, uint32_t log2n, uint32_t direction,
                                cfft_algo* base_algo, size_t* base_n, uint32_t* per_unit) {
  if (!batch) return fail(CFFT_ERR_INVALID_ARGUMENT, "null batch");
  for (const auto& c : batch->classes)
    if (c.key.kind == (int)kind && c.key.log2n == (int)log2n && c.key.dir == (int)direction) {
      if (base_algo) *base_algo = (cfft_algo)c.algo;
      if (base_n) *base_n = size_t(1) << c.base_log2;
      if (per_unit) *per_unit = (uint32_t)c.tpc;
      return CFFT_OK;
    }
  return fail(CFFT_ERR_INVALID_ARGUMENT, "no such size class in the batch");
}

cfft_status cfft_batch_run(cfft_batch* b, double* data, void* stream) {
  if (!b || !data) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (b->units == 0) return CFFT_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (s == nullptr) return launch_batch(b, (double2*)data, s);  // the legacy stream cannot be captured
  std::lock_guard<std::mutex> lk(b->mu);
  if (!b->g_exec || b->g_stream != s || b->g_data != data) {
    if (b->g_exec) {
      cudaGraphExecDestroy(b->g_exec);
      b->g_exec = nullptr;
    }
    cudaGraph_t graph;
    CFFT_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cfft_status st = launch_batch(b, (double2*)data, s);
    cudaError_t e = cudaStreamEndCapture(s, &graph);
    if (st != CFFT_OK) return st;
    if (e != cudaSuccess) return fail(CFFT_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&b->g_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail(CFFT_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    b->g_stream = s;
    b->g_data = data;
  }
  CFFT_CUDA_TRY(cudaGraphLaunch(b->g_exec, s));
  return CFFT_OK;
}

cfft_status cfft_batch_run_host(cfft_batch* b, double* host, double* dev, void* stream) {
  if (!b || !host || !dev) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (b->units == 0) return CFFT_OK;
  std::lock_guard<std::mutex> lk(b->mu);
  if (b->chunks.empty()) {
    cfft_status st = build_chunks(b);
    if (st != CFFT_OK) return st;
  }
  cudaStream_t s = (cudaStream_t)stream;
  CFFT_CUDA_TRY(cudaEventRecord(b->pevent[3], s));
  for (cudaStream_t ps : b->pstream) CFFT_CUDA_TRY(cudaStreamWaitEvent(ps, b->pevent[3], 0));
  for (size_t k = 0; k < b->chunks.size(); ++k) {
    const cfft_batch::Chunk& c = b->chunks[k];
    cudaStream_t ps = b->pstream[k % 3];
    const size_t bytes = (size_t)(c.hi - c.lo) * sizeof(double2);
    double* hp = host + 2 * c.lo;
    double* dp = dev + 2 * c.lo;
    CFFT_CUDA_TRY(cudaMemcpyAsync(dp, hp, bytes, cudaMemcpyHostToDevice, ps));
    const cfft_status st =
        launch_phases(b, (double2*)dev, c.d_offs, c.d_units, c.phase, b->d_heads + k * kMaxPhases, ps);
    if (st != CFFT_OK) return st;
    CFFT_CUDA_TRY(cudaMemcpyAsync(hp, dp, bytes, cudaMemcpyDeviceToHost, ps));
  }
  for (int i = 0; i < 3; ++i) {
    CFFT_CUDA_TRY(cudaEventRecord(b->pevent[i], b->pstream[i]));
    CFFT_CUDA_TRY(cudaStreamWaitEvent(s, b->pevent[i], 0));
  }
  return CFFT_OK;
}

}  // extern "C"
