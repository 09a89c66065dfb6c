// Host side of the batching form: mixed-shape, mixed-direction batches in one persistent
// launch (k_ragged), and the per-array launch loop it is compared against.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/bridct_b200.h"
#include "bridct_internal.h"
#include "ragged.cuh"

// One shape class of a ragged batch: every array of one (height, width, mode), with the device
// table of their offsets and the schedule that runs them.
struct RaggedClass {
  int h = 0, w = 0, mode = 0;
  std::vector<int> arrays;            // indices into the item list
  long long* d_offs = nullptr;        // offsets (floats) of those arrays
  size_t floats = 0;                  // elements of the class
  int schedule = BRIDCT_RAGGED_QUEUE;
  bool merged = false;                // its arrays are in the merged passes
};

constexpr int kRaggedMaxStreams = 8;

// A merged pass: every column strip (col) or row block of the MERGED classes whose line lengths share a
// kernel (merged.cu), as one launch over a device table of units.
struct MergedPass {
  int cls = 0, mode = 0;              // mode -1: every unit its own
  bool col = true;
  bridct::MergedUnit* d_units = nullptr;
  long long n = 0;
  size_t floats = 0;
};

// What a batch's schedule runs: the queue and the merged passes, on the host and on the device.
struct RaggedTables {
  std::vector<bridct::RaggedArray> arrays;
  std::vector<bridct::RaggedUnit> units;
  bridct::RaggedArray* d_arrays = nullptr;
  bridct::RaggedUnit* d_units = nullptr;
  std::vector<MergedPass> merged;       // column passes first, then row passes
};

struct bridct_ragged {
  int device = 0;
  bridct::DeviceCtx* dev = nullptr;
  std::vector<bridct_ragged_item> items;
  RaggedTables tables;
  unsigned int* d_counters = nullptr;   // [0] queue head, [1..n] strips done per array
  int* d_err = nullptr;
  size_t span = 0;                      // floats covered by the batch (max offset + size)
  int grid = 0;
  unsigned spin_limit = bridct::kRaggedSpin;
  bridct_ragged_tuning tuning{};
  std::map<int, bridct_plan*> plans;    // per-array launch loop: one plan per shape
  // shape classes, in decreasing size; classes scheduled as their own launches run on `streams`
  // side streams forked from and joined back into the caller's stream
  std::vector<RaggedClass> classes;
  int streams = 4;
  cudaStream_t aux[kRaggedMaxStreams] = {};
  cudaEvent_t fork_ev = nullptr, join_ev[kRaggedMaxStreams] = {};
  cudaEvent_t mid_ev[kRaggedMaxStreams] = {}, mid_fork = nullptr;   // between merged column and row passes
};

namespace bridct {
namespace {

int lg(int n) {
  int k = 0;
  while ((8 << k) < n) ++k;
  return k;
}

// Smallest number of lines of a unit (1 for register lines).
int lines_per_warp(int n) { return n >= 128 ? 1024 / n : 1; }

int pow2_floor(int v) {
  int p = 1;
  while (p * 2 <= v) p *= 2;
  return p;
}

// Columns per strip: a power of two dividing w, >= 4 (float4 rows), >= lines_per_warp(h),
// and h * columns <= budget unless the minimum forces more.
int strip_cols(int h, int w, int budget) {
  const int want = pow2_floor(std::max(1, std::min(w, budget / h)));
  return std::min(w, std::max(want, std::max(4, lines_per_warp(h))));
}

// Whether an array is one unit.
bool one_unit(int h, int w, const bridct_ragged_tuning& t) { return h * w <= t.tile_floats && ragged_fits(h, w); }

// Rows per row block: a power of two dividing h, >= lines_per_warp(w).
int block_rows(int h, int w, int budget) {
  const int want = pow2_floor(std::max(1, std::min(h, budget / w)));
  return std::min(h, std::max(want, lines_per_warp(w)));
}

// Queued arrays that run in the merged passes where a batch has them: those that the queue takes through
// its two passes because no sub-block holds them, with lines that the merged kernels know.  The
// queue takes about three times as long for them: batches of mixed arrays, queued / joined, us a call:
// 640 up to 256 x 256 42 / 34, 200 up to 1024 x 1024 81 / 74, 1024 of them 296 / 280.  Below kJoinFloats
// elements the launches they add cost more (200 up to 256 x 256 27.8 / 29.7, 64 of them 26.9 / 30.9).
constexpr size_t kJoinFloats = (size_t)1 << 21;
bool may_join(const RaggedClass& c) {
  return c.schedule == BRIDCT_RAGGED_QUEUE && !ragged_fits(c.h, c.w) && c.h >= 32 && c.w >= 32;
}

// Queue order of items a and b: large arrays first (the small ones fill the tail), arrays of one shape
// and mode together, so that the CTAs of an SM run the same few line programs at a time (in submission
// order the kernel spent a third of its time waiting for instructions).
bool queue_before(const bridct_ragged_item* items, int a, int b) {
  const bridct_ragged_item &p = items[a], &q = items[b];
  const long long ep = (long long)p.height * p.width, eq = (long long)q.height * q.width;
  if (ep != eq) return ep > eq;
  if (p.height != q.height) return p.height > q.height;
  if (p.mode != q.mode) return p.mode < q.mode;
  return a < b;
}

// The queue of the classes' present schedules.
void build_units(const bridct_ragged* r, RaggedTables& tables) {
  bridct_ragged_tuning t = r->tuning;
  t.strip_floats = std::min(t.strip_floats, kRaggedUnit);
  t.row_floats = std::min(t.row_floats, kRaggedUnit);
  std::vector<int> big, small;
  std::vector<char> queued(r->items.size(), 1);
  for (const RaggedClass& c : r->classes)
    if (c.schedule != BRIDCT_RAGGED_QUEUE || c.merged)
      for (int i : c.arrays) queued[i] = 0;
  for (size_t i = 0; i < r->items.size(); ++i) {
    const bridct_ragged_item& it = r->items[i];
    RaggedArray a{(long long)it.offset, (short)it.height, (short)it.width, (short)it.mode, 0};
    if (!queued[i]) {
      // run by its class's own launch: not in the queue
    } else if (one_unit(it.height, it.width, t)) {
      small.push_back((int)i);
    } else {
      a.nstrips = (short)(it.width / strip_cols(it.height, it.width, t.strip_floats));
      big.push_back((int)i);
    }
    tables.arrays.push_back(a);
  }
  auto order = [&](int a, int b) { return queue_before(r->items.data(), a, b); };
  std::sort(big.begin(), big.end(), order);
  std::sort(small.begin(), small.end(), order);
  auto cols = [&](int i) {
    const RaggedArray& a = tables.arrays[i];
    const int tc = a.w / a.nstrips;
    for (int s = 0; s < a.nstrips; ++s) tables.units.push_back(RaggedUnit{i, UNIT_COLSTRIP, s * tc, tc});
  };
  auto rows = [&](int i) {
    const RaggedArray& a = tables.arrays[i];
    const int rb = block_rows(a.h, a.w, t.row_floats);
    for (int r0 = 0; r0 < a.h; r0 += rb) tables.units.push_back(RaggedUnit{i, UNIT_ROWBLOCK, r0, rb});
  };
  // Column strips of array k+lookahead are queued ahead of the row blocks of array k, so a
  // row block usually finds its strips finished; small arrays fill the tail.
  const int la = std::max(1, t.lookahead);
  for (size_t k = 0; k < big.size() + la; ++k) {
    if (k < big.size()) cols(big[k]);
    if (k >= (size_t)la) rows(big[k - la]);
  }
  for (int i : small) tables.units.push_back(RaggedUnit{i, UNIT_TILE, 0, 0});
}

// Groups the items into shape classes (height, width, mode), largest first, and uploads each
// class's offset table.
int build_classes(bridct_ragged* r) {
  std::map<std::tuple<int, int, int>, size_t> index;
  for (size_t i = 0; i < r->items.size(); ++i) {
    const bridct_ragged_item& it = r->items[i];
    const auto key = std::make_tuple(it.height, it.width, it.mode);
    auto f = index.find(key);
    if (f == index.end()) {
      f = index.emplace(key, r->classes.size()).first;
      RaggedClass c;
      c.h = it.height;
      c.w = it.width;
      c.mode = it.mode;
      r->classes.push_back(c);
    }
    RaggedClass& c = r->classes[f->second];
    c.arrays.push_back((int)i);
    c.floats += (size_t)it.height * it.width;
  }
  std::stable_sort(r->classes.begin(), r->classes.end(),
                   [](const RaggedClass& a, const RaggedClass& b) { return a.floats > b.floats; });
  for (RaggedClass& c : r->classes) {
    std::vector<long long> offs;
    for (int i : c.arrays) offs.push_back((long long)r->items[i].offset);
    cudaError_t e = cudaMalloc((void**)&c.d_offs, offs.size() * sizeof(long long));
    if (e == cudaSuccess) e = upload_table(c.d_offs, offs.data(), offs.size() * sizeof(long long));
    if (e != cudaSuccess) return cuda_fail(e, "ragged class tables");
  }
  cudaError_t e = cudaEventCreateWithFlags(&r->fork_ev, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&r->mid_fork, cudaEventDisableTiming);
  for (int i = 0; e == cudaSuccess && i < kRaggedMaxStreams; ++i) {
    e = cudaStreamCreateWithFlags(&r->aux[i], cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&r->join_ev[i], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&r->mid_ev[i], cudaEventDisableTiming);
  }
  return e == cudaSuccess ? BRIDCT_OK : cuda_fail(e, "ragged streams");
}

// Merged batches up to this many elements take all modes in one launch: the launches bound them (81
// against 88 us a call at 12 M elements, 192 against 182 at 37 M; merged.cu).
constexpr size_t kMergedAllModes = (size_t)1 << 24;

void free_tables(RaggedTables& tables) {
  cudaFree(tables.d_arrays);
  cudaFree(tables.d_units);
  for (MergedPass& m : tables.merged) cudaFree(m.d_units);
  tables = RaggedTables{};
}

// Unit tables of the merged passes: column strips of the MERGED classes grouped by the kernel of their
// column length, row blocks by that of their row length, each group largest first.  Within a group the
// units go by line length and mode, so that the CTAs of an SM run few line programs at a time.
int build_merged(const bridct_ragged* r, RaggedTables& tables) {
  size_t floats = 0;
  for (const RaggedClass& c : r->classes) floats += c.merged ? c.floats : 0;
  const bool all_modes = floats <= kMergedAllModes;
  for (int pass = 0; pass < 2; ++pass) {
    const bool col = pass == 0;
    std::map<std::pair<int, int>, std::vector<MergedUnit>> groups;
    for (const RaggedClass& c : r->classes) {
      if (!c.merged) continue;
      std::vector<MergedUnit>& g = groups[{merged_class(col, col ? c.h : c.w), all_modes ? -1 : c.mode}];
      const int step = col ? merged_strip_cols(c.h) : merged_block_rows(c.w), end = col ? c.w : c.h;
      for (int i : c.arrays)
        for (int k = 0; k < end; k += step)
          g.push_back(MergedUnit{(long long)r->items[i].offset + (long long)k * (col ? 1 : c.w), c.w,
                                 (short)(col ? c.h : c.w), (short)c.mode});
    }
    const size_t first = tables.merged.size();
    for (auto& kv : groups) {
      std::vector<MergedUnit>& g = kv.second;
      std::stable_sort(g.begin(), g.end(), [](const MergedUnit& a, const MergedUnit& b) {
        return a.n != b.n ? a.n > b.n : a.mode < b.mode;
      });
      MergedPass m;
      m.cls = kv.first.first;
      m.mode = kv.first.second;
      m.col = col;
      m.n = (long long)g.size();
      for (const MergedUnit& u : g) m.floats += (size_t)u.n * (col ? merged_strip_cols(u.n) : merged_block_rows(u.n));
      cudaError_t e = cudaMalloc((void**)&m.d_units, g.size() * sizeof(MergedUnit));
      if (e == cudaSuccess) e = upload_table(m.d_units, g.data(), g.size() * sizeof(MergedUnit));
      if (e != cudaSuccess) {
        cudaFree(m.d_units);
        return cuda_fail(e, "merged pass tables");
      }
      tables.merged.push_back(m);
    }
    std::stable_sort(tables.merged.begin() + first, tables.merged.end(),
                     [](const MergedPass& a, const MergedPass& b) { return a.floats > b.floats; });
  }
  return BRIDCT_OK;
}

int launch_merged(bridct_ragged* r, const MergedPass& m, const float* x, float* y, cudaStream_t st) {
  // column passes read x and write y; row passes transform y in place
  cudaError_t e = launch_merged_pass(r->dev, m.col, m.cls, m.mode, m.d_units, m.n, m.col ? x : y, y, st);
  return e == cudaSuccess ? BRIDCT_OK : cuda_fail(e, "merged pass launch");
}

// One class as its own plain-form launch over the class's offset table.
int launch_class(bridct_ragged* r, const RaggedClass& c, int schedule, const float* x, float* y, cudaStream_t st) {
  BatchLayout l;
  l.offs = c.d_offs;
  l.ld = c.w;
  l.small_units = schedule == BRIDCT_RAGGED_CLASS_LAUNCH_SMALL;
  return launch_plain_layout(r->dev, c.h, c.w, c.mode, x, y, (long long)c.arrays.size(), &l, &l, st);
}

int upload(RaggedTables& t) {
  cudaError_t e = cudaMalloc((void**)&t.d_arrays, t.arrays.size() * sizeof(RaggedArray));
  if (e == cudaSuccess) e = cudaMalloc((void**)&t.d_units, std::max<size_t>(1, t.units.size()) * sizeof(RaggedUnit));
  if (e == cudaSuccess)
    e = upload_table(t.d_arrays, t.arrays.data(), t.arrays.size() * sizeof(RaggedArray));
  if (e == cudaSuccess && !t.units.empty())
    e = upload_table(t.d_units, t.units.data(), t.units.size() * sizeof(RaggedUnit));
  return e == cudaSuccess ? BRIDCT_OK : cuda_fail(e, "ragged upload");
}

// The tables of the classes' present schedules, in place of the batch's: all of them, or on failure none (the batch
// keeps the old ones).
int replace_tables(bridct_ragged* r) {
  RaggedTables t;
  build_units(r, t);
  int s = upload(t);
  if (!s) s = build_merged(r, t);
  if (s) {
    free_tables(t);
    return s;
  }
  std::swap(r->tables, t);
  free_tables(t);
  return BRIDCT_OK;
}

}  // namespace
}  // namespace bridct

using namespace bridct;

extern "C" {

BRIDCT_API void bridct_ragged_default_tuning(bridct_ragged_tuning* t) {
  if (!t) return;
  t->tile_floats = 16384;
  t->strip_floats = 16384;
  t->row_floats = 16384;
  t->lookahead = 32;   // 2, 16, 32: 2.65, 2.26, 2.24 ms (4096 mixed arrays; an earlier queue kernel of whole-array units)
}

BRIDCT_API bridct_ragged* bridct_ragged_create(const bridct_ragged_item* items, size_t count) {
  bridct_ragged_tuning t;
  bridct_ragged_default_tuning(&t);
  return bridct_ragged_create_tuned(items, count, &t);
}

BRIDCT_API bridct_ragged* bridct_ragged_create_tuned(const bridct_ragged_item* items, size_t count,
                                                     const bridct_ragged_tuning* tuning) {
  if (!items || count == 0 || count > 0x7FFFFFFF || !tuning) {
    set_error("bridct_ragged_create: empty or NULL item list");
    return nullptr;
  }
  const bridct_ragged_tuning& t = *tuning;
  if (t.tile_floats < 64 || t.tile_floats > 16384 || t.strip_floats < 64 || t.strip_floats > 16384 ||
      t.row_floats < 64 || t.row_floats > 16384 || t.lookahead < 1 || t.lookahead > 64) {
    set_error("bridct_ragged_create: tuning out of range");
    return nullptr;
  }
  std::vector<std::pair<size_t, size_t>> spans;
  size_t span = 0;
  for (size_t i = 0; i < count; ++i) {
    const bridct_ragged_item& it = items[i];
    if (!bridct_supported(it.height, it.width) || it.mode < 0 || it.mode > 2 || it.offset % 4) {
      set_error("bridct_ragged_create: item " + std::to_string(i) +
                " has an unsupported shape, mode, or an offset that is not a multiple of 4 floats");
      return nullptr;
    }
    const size_t e = (size_t)it.height * it.width;
    spans.push_back({it.offset, it.offset + e});
    span = std::max(span, it.offset + e);
  }
  std::sort(spans.begin(), spans.end());
  for (size_t i = 1; i < spans.size(); ++i)
    if (spans[i].first < spans[i - 1].second) {
      set_error("bridct_ragged_create: arrays overlap");
      return nullptr;
    }
  int dev = 0;
  if (current_device(&dev) != BRIDCT_OK) return nullptr;
  DeviceCtx* d = device_ctx(dev);
  if (!d) return nullptr;
  bridct_ragged* r = new bridct_ragged();
  r->device = dev;
  r->dev = d;
  r->items.assign(items, items + count);
  r->span = span;
  r->tuning = t;
  if (build_classes(r) != BRIDCT_OK) {
    bridct_ragged_destroy(r);
    return nullptr;
  }
  cudaError_t e = cudaMalloc((void**)&r->d_counters, (count + 1) * sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMalloc((void**)&r->d_err, sizeof(int));
  const int zero = 0;
  if (e == cudaSuccess) e = upload_table(r->d_err, &zero, sizeof(int));
  if (e != cudaSuccess || replace_tables(r) != BRIDCT_OK) {
    if (e != cudaSuccess) cuda_fail(e, "bridct_ragged_create");
    bridct_ragged_destroy(r);
    return nullptr;
  }
  const int bps = kernel_setup(reinterpret_cast<const void*>(k_ragged), kRaggedSmem, kRaggedThreads);
  if (bps <= 0) {
    cuda_fail(cudaErrorInvalidConfiguration, "k_ragged occupancy");
    bridct_ragged_destroy(r);
    return nullptr;
  }
  r->grid = std::min<long long>((long long)d->sm_count * bps, std::max<size_t>(1, r->tables.units.size()));
  return r;
}

BRIDCT_API void bridct_ragged_destroy(bridct_ragged* r) {
  if (!r) return;
  free_tables(r->tables);
  cudaFree(r->d_counters);
  cudaFree(r->d_err);
  for (auto& kv : r->plans) bridct_plan_destroy(kv.second);
  for (RaggedClass& c : r->classes) cudaFree(c.d_offs);
  for (int i = 0; i < kRaggedMaxStreams; ++i) {
    if (r->aux[i]) cudaStreamDestroy(r->aux[i]);
    if (r->join_ev[i]) cudaEventDestroy(r->join_ev[i]);
    if (r->mid_ev[i]) cudaEventDestroy(r->mid_ev[i]);
  }
  if (r->fork_ev) cudaEventDestroy(r->fork_ev);
  if (r->mid_fork) cudaEventDestroy(r->mid_fork);
  delete r;
}

BRIDCT_API size_t bridct_ragged_units(const bridct_ragged* r) { return r ? r->tables.units.size() : 0; }

BRIDCT_API int bridct_ragged_apply_device(bridct_ragged* r, const float* x, float* y, void* stream) {
  if (!r || !x || !y) return BRIDCT_INVALID_ARGUMENT;
  const size_t bytes = r->span * sizeof(float);
  const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
  if ((a <= b ? b - a : a - b) < bytes) return BRIDCT_OVERLAPPING_BUFFERS;
  if ((a | b) % 16) return BRIDCT_BAD_ALIGNMENT;
  DeviceGuard guard(r->device);
  if (guard.status != cudaSuccess) return cuda_fail(guard.status, "cudaSetDevice(batch device)");
  cudaStream_t st = (cudaStream_t)stream;
  // Classes with their own launches run on side streams forked from the caller's stream (largest
  // class first, round robin) and joined back into it; the queue's persistent kernel runs on the
  // caller's stream meanwhile.  Capturable: the fork and join are events on captured streams.
  // MERGED classes run as merged column passes, then (after every column pass has finished) merged
  // row passes, spread over the side streams; classes with their own launches follow on the same
  // streams.
  std::vector<const RaggedClass*> own;
  for (const RaggedClass& c : r->classes)
    if (c.schedule == BRIDCT_RAGGED_CLASS_LAUNCH || c.schedule == BRIDCT_RAGGED_CLASS_LAUNCH_SMALL) own.push_back(&c);
  size_t ncol = 0;
  for (const MergedPass& m : r->tables.merged) ncol += m.col ? 1 : 0;
  const size_t nrow = r->tables.merged.size() - ncol;
  const size_t widest = std::max(own.size(), std::max(ncol, nrow));
  cudaError_t e = cudaSuccess;
  const int nst = std::max(1, std::min(r->streams, (int)widest));
  const bool fork = !own.empty() || !r->tables.merged.empty();
  if (fork) {
    e = cudaEventRecord(r->fork_ev, st);
    for (int i = 0; e == cudaSuccess && i < nst; ++i) e = cudaStreamWaitEvent(r->aux[i], r->fork_ev, 0);
    if (e != cudaSuccess) return cuda_fail(e, "ragged fork");
  }
  if (!r->tables.merged.empty()) {
    for (size_t k = 0; k < ncol; ++k) {
      const int s = launch_merged(r, r->tables.merged[k], x, y, r->aux[k % nst]);
      if (s) return s;
    }
    // every row block needs its array's column strips: all side streams meet here
    for (int i = 1; e == cudaSuccess && i < nst; ++i) {
      e = cudaEventRecord(r->mid_ev[i], r->aux[i]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(r->aux[0], r->mid_ev[i], 0);
    }
    if (e == cudaSuccess) e = cudaEventRecord(r->mid_fork, r->aux[0]);
    for (int i = 1; e == cudaSuccess && i < nst; ++i) e = cudaStreamWaitEvent(r->aux[i], r->mid_fork, 0);
    if (e != cudaSuccess) return cuda_fail(e, "ragged merged barrier");
    for (size_t k = 0; k < nrow; ++k) {
      const int s = launch_merged(r, r->tables.merged[ncol + k], x, y, r->aux[k % nst]);
      if (s) return s;
    }
  }
  for (size_t k = 0; k < own.size(); ++k) {
    const int s = launch_class(r, *own[k], own[k]->schedule, x, y, r->aux[k % nst]);
    if (s) return s;
  }
  if (!r->tables.units.empty()) {
    e = cudaMemsetAsync(r->d_counters, 0, (r->items.size() + 1) * sizeof(unsigned int), st);
    if (e != cudaSuccess) return cuda_fail(e, "ragged reset");
    RaggedArgs args;
    args.x = x;
    args.y = y;
    args.arrays = r->tables.d_arrays;
    args.units = r->tables.d_units;
    args.nunits = (int)r->tables.units.size();
    args.next = r->d_counters;
    args.done = r->d_counters + 1;
    args.err = r->d_err;
    args.spin_limit = r->spin_limit;
    for (int i = 0; i < 4; ++i) args.tab[i] = r->dev->split[i];
    k_ragged<<<r->grid, kRaggedThreads, kRaggedSmem, st>>>(args);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "k_ragged launch");
  }
  for (int i = 0; fork && i < nst; ++i) {
    e = cudaEventRecord(r->join_ev[i], r->aux[i]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, r->join_ev[i], 0);
    if (e != cudaSuccess) return cuda_fail(e, "ragged join");
  }
  return BRIDCT_OK;
}

BRIDCT_API size_t bridct_ragged_class_count(const bridct_ragged* r) { return r ? r->classes.size() : 0; }

BRIDCT_API size_t bridct_ragged_launch_count(const bridct_ragged* r) {
  if (!r) return 0;
  size_t n = r->tables.merged.size() + (r->tables.units.empty() ? 0 : 1);
  for (const RaggedClass& c : r->classes)
    if (c.schedule == BRIDCT_RAGGED_CLASS_LAUNCH || c.schedule == BRIDCT_RAGGED_CLASS_LAUNCH_SMALL)
      n += c.h * c.w <= 16384 ? 1 : 2;
  return n;
}

BRIDCT_API int bridct_ragged_class_info(const bridct_ragged* r, size_t cls, int* height, int* width, int* mode,
                                        size_t* arrays, int* schedule) {
  if (!r || cls >= r->classes.size()) return BRIDCT_INVALID_ARGUMENT;
  const RaggedClass& c = r->classes[cls];
  if (height) *height = c.h;
  if (width) *width = c.w;
  if (mode) *mode = c.mode;
  if (arrays) *arrays = c.arrays.size();
  if (schedule) *schedule = c.schedule;
  return BRIDCT_OK;
}

BRIDCT_API int bridct_ragged_set_schedule(bridct_ragged* r, const int* schedules, size_t count, int streams) {
  if (!r || count != r->classes.size() || (count && !schedules) || streams < 1 || streams > kRaggedMaxStreams)
    return BRIDCT_INVALID_ARGUMENT;
  for (size_t i = 0; i < count; ++i) {
    if (schedules[i] < BRIDCT_RAGGED_QUEUE || schedules[i] > BRIDCT_RAGGED_MERGED) {
      set_error("bridct_ragged_set_schedule: unknown schedule " + std::to_string(schedules[i]));
      return BRIDCT_INVALID_ARGUMENT;
    }
    const RaggedClass& c = r->classes[i];
    if (schedules[i] == BRIDCT_RAGGED_MERGED && !merged_route(c.h, c.w, c.mode)) {
      set_error("bridct_ragged_set_schedule: class " + std::to_string(i) + " is not a two-pass shape");
      return BRIDCT_INVALID_ARGUMENT;
    }
  }
  DeviceGuard guard(r->device);
  if (guard.status != cudaSuccess) return cuda_fail(guard.status, "cudaSetDevice(batch device)");
  cudaError_t e = cudaDeviceSynchronize();   // the old queue may still be in use
  if (e != cudaSuccess) return cuda_fail(e, "bridct_ragged_set_schedule");
  std::vector<std::pair<int, bool>> before;   // schedules and merged flags, kept if the tables cannot be made
  for (const RaggedClass& c : r->classes) before.push_back({c.schedule, c.merged});
  bool any_merged = false;
  size_t merged_floats = 0;   // with the queued classes that may join
  for (size_t i = 0; i < count; ++i) {
    RaggedClass& c = r->classes[i];
    c.schedule = schedules[i];
    any_merged |= c.schedule == BRIDCT_RAGGED_MERGED;
    if (c.schedule == BRIDCT_RAGGED_MERGED || may_join(c)) merged_floats += c.floats;
  }
  const bool join = any_merged && merged_floats >= kJoinFloats;
  for (RaggedClass& c : r->classes) c.merged = c.schedule == BRIDCT_RAGGED_MERGED || (join && may_join(c));
  const int s = replace_tables(r);
  if (s) {
    for (size_t i = 0; i < count; ++i) {
      r->classes[i].schedule = before[i].first;
      r->classes[i].merged = before[i].second;
    }
    return s;
  }
  r->streams = streams;
  const int bps = kernel_setup(reinterpret_cast<const void*>(k_ragged), kRaggedSmem, kRaggedThreads);
  r->grid = (int)std::min<long long>((long long)r->dev->sm_count * std::max(1, bps),
                                     std::max<size_t>(1, r->tables.units.size()));
  return BRIDCT_OK;
}

BRIDCT_API int bridct_ragged_apply_class_device(bridct_ragged* r, size_t cls, int schedule, const float* x, float* y,
                                                void* stream) {
  if (!r || !x || !y || cls >= r->classes.size() ||
      (schedule != BRIDCT_RAGGED_CLASS_LAUNCH && schedule != BRIDCT_RAGGED_CLASS_LAUNCH_SMALL))
    return BRIDCT_INVALID_ARGUMENT;
  const size_t bytes = r->span * sizeof(float);
  const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
  if ((a <= b ? b - a : a - b) < bytes) return BRIDCT_OVERLAPPING_BUFFERS;
  if ((a | b) % 16) return BRIDCT_BAD_ALIGNMENT;
  DeviceGuard guard(r->device);
  if (guard.status != cudaSuccess) return cuda_fail(guard.status, "cudaSetDevice(batch device)");
  return launch_class(r, r->classes[cls], schedule, x, y, (cudaStream_t)stream);
}

BRIDCT_API int bridct_ragged_set_wait_limit(bridct_ragged* r, unsigned polls) {
  if (!r) return BRIDCT_INVALID_ARGUMENT;
  r->spin_limit = polls;
  return BRIDCT_OK;
}

BRIDCT_API int bridct_ragged_timeout_flag(bridct_ragged* r) {
  if (!r) return 0;
  DeviceGuard guard(r->device);
  int v = 0;
  cudaMemcpy(&v, r->d_err, sizeof(int), cudaMemcpyDeviceToHost);
  const int zero = 0;
  if (v) upload_table(r->d_err, &zero, sizeof(int));
  return v;
}

BRIDCT_API int bridct_ragged_apply_loop_device(bridct_ragged* r, const float* x, float* y, void* stream) {
  if (!r || !x || !y) return BRIDCT_INVALID_ARGUMENT;
  const size_t bytes = r->span * sizeof(float);
  const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
  if ((a <= b ? b - a : a - b) < bytes) return BRIDCT_OVERLAPPING_BUFFERS;
  if ((a | b) % 16) return BRIDCT_BAD_ALIGNMENT;
  DeviceGuard guard(r->device);
  if (guard.status != cudaSuccess) return cuda_fail(guard.status, "cudaSetDevice(batch device)");
  // one launch per array, grouped by shape so consecutive launches reuse kernels
  std::vector<int> order(r->items.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) {
    const int kp = lg(r->items[p].height) * 8 + lg(r->items[p].width);
    const int kq = lg(r->items[q].height) * 8 + lg(r->items[q].width);
    return kp < kq;
  });
  for (int i : order) {
    const bridct_ragged_item& it = r->items[i];
    const int key = lg(it.height) * 8 + lg(it.width);
    bridct_plan*& p = r->plans[key];
    if (!p) {
      p = bridct_plan_create(it.height, it.width);
      if (!p) return BRIDCT_DEVICE_ERROR;
    }
    int s = launch_plain_form(p, it.mode, x + it.offset, y + it.offset, 1, (cudaStream_t)stream);
    if (s) return s;
  }
  return BRIDCT_OK;
}

}  // extern "C"

// ---- Ragged batch without any allocation ---------------------------------------------------
//
// Some callers cannot let a library allocate device memory: a framework whose caching
// allocator owns every byte of the GPU (any cudaMalloc outside it can fail or fragment its
// pool), a latency-bound loop where cudaMalloc/cudaFree's implicit device synchronisation is
// not acceptable, or an embedding that fixes the process's device footprint at start-up.
// bridct_ragged_apply_noalloc serves them: the caller passes the item list and the input and
// output buffers, and everything else the persistent kernel needs (work queue, per-array
// counters, error word, split-line tables) lives in one statically sized __device__ array below,
// which every GPU that loads this library holds until the process exits.  The host side builds
// the queue in static buffers as well, so a successful call allocates nothing.
namespace {

constexpr int kNaMaxArrays = 4096;    // items per call
constexpr int kNaMaxUnits = 49152;    // work units per call, counted in units of the default tuning's sizes
// The units queued are smaller: strips and row blocks by half, and a whole array that no sub-block
// holds becomes up to four of them.
constexpr int kNaQueue = 2 * kNaMaxUnits + 2 * kNaMaxArrays;

struct NaOff {
  static constexpr size_t arrays = 0;
  static constexpr size_t units = arrays + sizeof(bridct::RaggedArray) * kNaMaxArrays;
  static constexpr size_t counters = units + sizeof(bridct::RaggedUnit) * kNaQueue;
  static constexpr size_t err = counters + sizeof(unsigned int) * (kNaMaxArrays + 1);
  static constexpr size_t tabs = (err + sizeof(int) + 255) / 256 * 256;   // split-line tables, N = 128..1024
  static constexpr size_t bytes = tabs + sizeof(float) * bridct::kRaggedTabs;
};

}  // namespace

// About 0.95 MB: queue (arrays, units), counters, error word, split-line tables.  Host code must
// not use this name as a device address; the entry point resolves it per device below.
static __device__ __align__(256) unsigned char g_ragged_scratch[NaOff::bytes];

namespace {

std::mutex g_na_mutex;                                  // one call at a time (shared scratch)
bridct::RaggedArray g_na_arrays[kNaMaxArrays];
bridct::RaggedUnit g_na_units[kNaQueue];
int g_na_big[kNaMaxArrays];
int g_na_small[kNaMaxArrays];
int g_na_order[kNaMaxArrays];
float g_na_tabs[bridct::kRaggedTabs];                  // split-line tables, N = 128..1024
bool g_na_filled = false;
unsigned char* g_na_addr[64] = {};                      // scratch address per device

// First float of the tables of N = 128 << i.
size_t na_segment(int i) {
  return i == 0 ? 0 : i == 1 ? bridct::ragged_tab<256>() : i == 2 ? bridct::ragged_tab<512>() : bridct::ragged_tab<1024>();
}

}  // namespace

extern "C" BRIDCT_API int bridct_ragged_apply_noalloc(const bridct_ragged_item* items, size_t count,
                                                      const float* input, float* output, void* stream) {
  using namespace bridct;
  if (!items || !input || !output || count == 0) return BRIDCT_INVALID_ARGUMENT;
  if (count > (size_t)kNaMaxArrays) {
    set_error("bridct_ragged_apply_noalloc: at most 4096 arrays per call");
    return BRIDCT_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lock(g_na_mutex);
  // validation (as bridct_ragged_create): shapes, modes, 16-byte aligned offsets, no overlap
  size_t span = 0;
  for (size_t i = 0; i < count; ++i) {
    const bridct_ragged_item& it = items[i];
    if (!bridct_supported(it.height, it.width) || it.mode < 0 || it.mode > 2 || it.offset % 4) {
      set_error("bridct_ragged_apply_noalloc: unsupported shape or mode, or misaligned offset");
      return BRIDCT_INVALID_ARGUMENT;
    }
    span = std::max(span, it.offset + (size_t)it.height * it.width);
    g_na_order[i] = (int)i;
  }
  std::sort(g_na_order, g_na_order + count, [&](int a, int b) {
    return items[a].offset != items[b].offset ? items[a].offset < items[b].offset : a < b;
  });
  for (size_t i = 1; i < count; ++i) {
    const bridct_ragged_item& p = items[g_na_order[i - 1]];
    if (items[g_na_order[i]].offset < p.offset + (size_t)p.height * p.width) {
      set_error("bridct_ragged_apply_noalloc: arrays overlap");
      return BRIDCT_INVALID_ARGUMENT;
    }
  }
  const uintptr_t xa = (uintptr_t)input, ya = (uintptr_t)output;
  if ((xa <= ya ? ya - xa : xa - ya) < span * sizeof(float)) return BRIDCT_OVERLAPPING_BUFFERS;
  if ((xa | ya) % 16) return BRIDCT_BAD_ALIGNMENT;

  // work queue with the default unit geometry (same units as bridct_ragged_create)
  bridct_ragged_tuning t;
  bridct_ragged_default_tuning(&t);
  int nbig = 0, nsmall = 0;
  long long limit = 0;   // units of the tuning's sizes
  for (size_t i = 0; i < count; ++i) {
    const bridct_ragged_item& it = items[i];
    RaggedArray a{(long long)it.offset, (short)it.height, (short)it.width, (short)it.mode, 0};
    const bool tile = (long long)it.height * it.width <= t.tile_floats;
    limit += tile ? 1 : it.width / strip_cols(it.height, it.width, t.strip_floats) +
                            it.height / block_rows(it.height, it.width, t.row_floats);
    if (one_unit(it.height, it.width, t)) {
      g_na_small[nsmall++] = (int)i;
    } else {
      a.nstrips = (short)(it.width / strip_cols(it.height, it.width, std::min(t.strip_floats, kRaggedUnit)));
      g_na_big[nbig++] = (int)i;
    }
    g_na_arrays[i] = a;
  }
  auto order = [&](int a, int b) { return queue_before(items, a, b); };
  std::sort(g_na_big, g_na_big + nbig, order);
  std::sort(g_na_small, g_na_small + nsmall, order);
  int nunits = 0;
  bool full = limit > kNaMaxUnits;
  auto push = [&](RaggedUnit u) {
    if (nunits == kNaQueue) full = true;
    else g_na_units[nunits++] = u;
  };
  for (int k = 0; k < nbig + t.lookahead; ++k) {
    if (k < nbig) {
      const RaggedArray& a = g_na_arrays[g_na_big[k]];
      const int tc = a.w / a.nstrips;
      for (int s = 0; s < a.nstrips; ++s) push(RaggedUnit{g_na_big[k], UNIT_COLSTRIP, s * tc, tc});
    }
    if (k >= t.lookahead) {
      const int i = g_na_big[k - t.lookahead];
      const RaggedArray& a = g_na_arrays[i];
      const int rb = block_rows(a.h, a.w, std::min(t.row_floats, kRaggedUnit));
      for (int r0 = 0; r0 < a.h; r0 += rb) push(RaggedUnit{i, UNIT_ROWBLOCK, r0, rb});
    }
  }
  for (int k = 0; k < nsmall; ++k) push(RaggedUnit{g_na_small[k], UNIT_TILE, 0, 0});
  if (full) {
    set_error("bridct_ragged_apply_noalloc: the batch needs more than 49152 work units");
    return BRIDCT_INVALID_ARGUMENT;
  }

  // set-up, once per device, with that device current: resolve the scratch array's device
  // address (the host-side name is only a stand-in) and upload the split-line tables into it
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) {
    set_error("bridct_ragged_apply_noalloc: device index beyond 63");
    return BRIDCT_INVALID_ARGUMENT;
  }
  if (!g_na_filled) {
    for (int i = 0; i < 4; ++i) fill_split_tables(128 << i, g_na_tabs + na_segment(i));
    g_na_filled = true;
  }
  if (!g_na_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_ragged_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_ragged_scratch)");
    unsigned char* base = static_cast<unsigned char*>(p);
    e = upload_table(base + NaOff::tabs, g_na_tabs, sizeof(g_na_tabs));
    if (e != cudaSuccess) return cuda_fail(e, "scratch tables");
    g_na_addr[dev] = base;
  }
  const int bps = kernel_setup(reinterpret_cast<const void*>(k_ragged), kRaggedSmem, kRaggedThreads);
  int sms = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess || bps <= 0) return cuda_fail(e != cudaSuccess ? e : cudaErrorInvalidConfiguration, "k_ragged");
  unsigned char* base = g_na_addr[dev];
  cudaStream_t st = (cudaStream_t)stream;
  // The scratch keeps the previous call's contents: queue tables are overwritten, and the
  // counters and error word are cleared before the launch.
  e = cudaMemcpyAsync(base + NaOff::arrays, g_na_arrays, count * sizeof(RaggedArray), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(base + NaOff::units, g_na_units, (size_t)nunits * sizeof(RaggedUnit), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(base + NaOff::counters, 0, (count + 1) * sizeof(unsigned int), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(base + NaOff::err, 0, sizeof(int), st);
  if (e != cudaSuccess) return cuda_fail(e, "scratch upload");
  RaggedArgs args;
  args.x = input;
  args.y = output;
  args.arrays = reinterpret_cast<const RaggedArray*>(base + NaOff::arrays);
  args.units = reinterpret_cast<const RaggedUnit*>(base + NaOff::units);
  args.nunits = nunits;
  args.next = reinterpret_cast<unsigned int*>(base + NaOff::counters);
  args.done = args.next + 1;
  args.err = reinterpret_cast<int*>(base + NaOff::err);
  args.spin_limit = kRaggedSpin;
  for (int i = 0; i < 4; ++i) args.tab[i].t = reinterpret_cast<const float*>(base + NaOff::tabs) + na_segment(i);
  const int grid = (int)std::min<long long>((long long)sms * bps, nunits);
  k_ragged<<<grid, kRaggedThreads, kRaggedSmem, st>>>(args);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_ragged launch");
  // Synchronous: the shared scratch is free again when the call returns.
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "bridct_ragged_apply_noalloc");
  int flag = 0;
  e = cudaMemcpy(&flag, base + NaOff::err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "error word");
  return flag ? BRIDCT_TIMEOUT : BRIDCT_OK;
}
