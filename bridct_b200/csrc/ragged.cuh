// Batching form: one persistent launch over a mixed-shape, mixed-direction batch.
//
// The host turns the batch into a queue of work units:
//   TILE      one array up to the tuning's tile_floats that lies in a sub-block whole: both passes
//   COLSTRIP  h rows x some columns of a larger array: its column lines, x -> y
//   ROWBLOCK  some full rows of a larger array: its row lines, y -> y in place
// CTAs are persistent (one launch, grid = SMs x resident CTAs) and take units in queue order
// from an atomic counter.  A ROWBLOCK of array i needs every COLSTRIP of array i finished: each
// strip adds 1 to done[i] after a __threadfence, and the row block spins on done[i] with a
// bounded budget (nanosleep back-off).  Column strips never wait, and every unit that a waiting
// row block depends on was dequeued earlier by a running CTA, so the wait always ends; on budget
// expiry the unit is skipped and the error flag set instead (the host reports BRIDCT_TIMEOUT).
//
// Line lengths and modes vary per unit and are dispatched at run time to the line pairs of the
// fixed-shape kernels (sj_split.cuh).  A unit is worked through in sub-blocks of at most 9216 floats of
// shared memory, so that three CTAs of 128 threads (168 registers: 64-point leaves, two lines per thread)
// share an SM together with the tables of all four split lengths.  1024 mixed arrays up to 1024 x 1024: 590 us with
// one line per thread or line group per warp in 256-thread CTAs of 112 KB, 408 us this way.
#pragma once
#include "sj_kernels.cuh"
#include "sj_split.cuh"

namespace bridct {

enum UnitType { UNIT_TILE = 0, UNIT_COLSTRIP = 1, UNIT_ROWBLOCK = 2 };

struct RaggedArray {
  long long offset;   // first float of the array in x and y
  short h, w, mode;
  short nstrips;      // column strips of a two-pass array (0 for tile arrays)
};

// Eight bytes: the queue of the allocation-free entry point lies in static device memory.
struct RaggedUnit {
  int array;
  unsigned what;      // type, then 11 bits each of first and count
  RaggedUnit() = default;
  RaggedUnit(int array, UnitType type, int first, int count)
      : array(array), what((unsigned)type | (unsigned)first << 2 | (unsigned)count << 13) {}
  __host__ __device__ int type() const { return what & 3; }
  __host__ __device__ int first() const { return what >> 2 & 0x7FF; }    // first column (COLSTRIP) or row (ROWBLOCK)
  __host__ __device__ int count() const { return what >> 13; }           // columns or rows covered
};
static_assert(sizeof(RaggedUnit) == 8 && sizeof(RaggedArray) == 16, "queue entries");

struct RaggedArgs {
  const float* x;
  float* y;
  const RaggedArray* arrays;
  const RaggedUnit* units;
  int nunits;
  unsigned int* next;       // queue head (zeroed before the launch)
  unsigned int* done;       // finished column strips per array (zeroed before the launch)
  int* err;
  unsigned spin_limit;      // polls of a row block's dependency wait before it gives up
  SplitTables tab[4];       // N = 128, 256, 512, 1024
};

constexpr int kRaggedThreads = 128;
constexpr int kRaggedTile = 9216;                                   // floats of a sub-block
// Floats of a strip or row block at most: one sub-block's.  Units of 16384 floats, and whole arrays of
// that size as one unit, measured (before / after, us a call of mixed arrays): 16 up to 256 x 256 23 / 17,
// 200 up to 256 x 256 30 / 24, 64 up to 1024 x 1024 48 / 39, 640 up to 1024 x 1024 237 / 230.  Units of
// 4096: 15.5, 27, 51 and 353.
constexpr int kRaggedUnit = 8192;
constexpr int kRaggedTabs = SplitTab<128>::kFloats + SplitTab<256>::kFloats + SplitTab<512>::kFloats + SplitTab<1024>::kFloats;
constexpr int kRaggedSmem = (kRaggedTile + kRaggedTabs) * 4;
constexpr unsigned kRaggedSpin = 1u << 22;                          // x ~256 ns back-off

// Offset (floats) of the tables of length N among the staged ones.
template <int N> __host__ __device__ constexpr int ragged_tab() {
  return N <= 128   ? 0
         : N == 256 ? SplitTab<128>::kFloats
         : N == 512 ? SplitTab<128>::kFloats + SplitTab<256>::kFloats
                    : SplitTab<128>::kFloats + SplitTab<256>::kFloats + SplitTab<512>::kFloats;
}

// Line pairs of a group: strips of 8 columns and blocks of 8 rows for 1024-point lines.
template <int N> __host__ __device__ constexpr int ragged_col_pairs() { return N == 1024 ? 4 : N == 512 ? 8 : 16; }
template <int N> __host__ __device__ constexpr int ragged_row_pairs() { return N == 1024 ? 4 : 8; }
// Row pitch in shared memory (32 / pairs modulo 32 floats for split rows).
__host__ __device__ constexpr int ragged_pitch(int w) { return w == 1024 ? w + 8 : w + 4; }
// Whether an array's two passes run in one shared-memory tile.
__host__ __device__ constexpr bool ragged_fits(int h, int w) { return h <= 256 && h * ragged_pitch(w) <= kRaggedTile; }

// Columns of length H, x -> y, rows ld floats apart in both.
template <int H, int MODE>
__device__ __forceinline__ void ragged_cols(const float* x, float* y, int ld, int ncols, float* tile,
                                            const float* tabs) {
  if constexpr (H <= 64) {
    for (int p = threadIdx.x; p < ncols / 2; p += kRaggedThreads) {
      F2 v[H];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const float2 f = __ldg(reinterpret_cast<const float2*>(x + (long long)i * ld) + p);
        v[i] = f2_make(f.x, f.y);
      }
      pair_line<H, MODE>(v);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        float2 f;
        f2_split(v[i], f.x, f.y);
        reinterpret_cast<float2*>(y + (long long)i * ld)[p] = f;
      }
    }
  } else {
    constexpr int LP = ragged_col_pairs<H>(), TC = 2 * LP;
    for (int c0 = 0; c0 < ncols; c0 += TC) {
      const int nc = ncols - c0 < TC ? ncols - c0 : TC, q = nc >> 2;   // a power of two, at least 4 columns
      const int sh = 31 - __clz(q);
      for (int i = threadIdx.x; i < H * q; i += kRaggedThreads) {
        const int r = i >> sh, c = (i & (q - 1)) << 2;
        cp_async16(tile + strip_row<TC>(r) + c, x + (long long)r * ld + c0 + c);
      }
      cp_async_wait_all();
      __syncthreads();
      const int p = 2 * (threadIdx.x % LP);
      float* yt = y + c0 + p;
      split_lines<H, MODE, kRaggedThreads, 1, LP, false>(
          [&](int, int i) {
            const float2 v = *reinterpret_cast<const float2*>(tile + strip_row<TC>(i) + p);
            return f2_make(v.x, v.y);
          },
          [&](int, int i, F2 v) {
            float2 f;
            f2_split(v, f.x, f.y);
            *reinterpret_cast<float2*>(yt + (long long)i * ld) = f;
          },
          [&](int) { return tile + p; }, TC, tabs + ragged_tab<H>(), [&](int) { return p < nc; });
      __syncthreads();
    }
  }
}

// Columns of an array that lies in shared memory whole, rows P floats apart (H <= 256).
template <int H, int MODE>
__device__ __forceinline__ void ragged_tile_cols(float* tile, int P, int w, const float* tabs) {
  if constexpr (H <= 64) {
    for (int p = threadIdx.x; p < w / 2; p += kRaggedThreads) {
      F2 v[H];
#pragma unroll
      for (int i = 0; i < H; ++i) v[i] = *reinterpret_cast<const F2*>(tile + i * P + 2 * p);
      pair_line<H, MODE>(v);
#pragma unroll
      for (int i = 0; i < H; ++i) *reinterpret_cast<F2*>(tile + i * P + 2 * p) = v[i];
    }
  } else {
    for (int c0 = 0; c0 < w; c0 += 32) {
      const int p = c0 + 2 * (threadIdx.x % 16);
      split_lines<H, MODE, kRaggedThreads, 1, 16, true>(
          [&](int, int i) { return *reinterpret_cast<const F2*>(tile + i * P + p); },
          [&](int, int i, F2 v) { *reinterpret_cast<F2*>(tile + i * P + p) = v; }, [&](int) { return tile + p; }, P,
          tabs + ragged_tab<H>(), [&](int) { return p < w; });
    }
  }
  __syncthreads();
}

// nr rows of length W in shared memory, in place.  Split rows: up to the rows of one sub-block; the
// second row of a pair may lie beyond nr (its values are not stored).
template <int W, int MODE>
__device__ __forceinline__ void ragged_rows(float* tile, int nr, const float* tabs) {
  constexpr int P = ragged_pitch(W);
  if constexpr (W <= 64) {
    for (int l = threadIdx.x; l < (nr + 15) / 16 * 8; l += kRaggedThreads) {
      const int r = (l / 8) * 16 + l % 8;
      if (r < nr) pair_rows<W, MODE>(tile + r * P, tile + (r + 8 < nr ? r + 8 : r) * P);
    }
  } else {
    constexpr int LP = ragged_row_pairs<W>(), GROUPS = W <= 256 ? 2 : 1, GP = 2 * LP * P;
    const int p = threadIdx.x % LP;
    float* rows = tile + p * P;
    split_lines<W, MODE, kRaggedThreads, GROUPS, LP, true>(
        [&](int g, int i) { return f2_make(rows[g * GP + i], rows[g * GP + i + LP * P]); },
        [&](int g, int i, F2 v) { f2_split(v, rows[g * GP + i], rows[g * GP + i + LP * P]); },
        [&](int g) { return tile + g * GP + 2 * p; }, 2 * LP, tabs + ragged_tab<W>(),
        [&](int g) { return g * 2 * LP + p < nr; });
  }
  fence_async();
  __syncthreads();
}

// Run-time dispatch of F<N, MODE>(...) over the line length and mode.
#define BRIDCT_RAGGED_CASE(F, N, ...)                       \
  case N:                                                   \
    if (mode == LM_FWD) F<N, LM_FWD>(__VA_ARGS__);          \
    else if (mode == LM_INV) F<N, LM_INV>(__VA_ARGS__);     \
    else F<N, LM_RT>(__VA_ARGS__);                          \
    break;

__device__ __forceinline__ void ragged_cols_dyn(int h, int mode, const float* x, float* y, int ld, int ncols,
                                                float* tile, const float* tabs) {
  switch (h) {
    BRIDCT_RAGGED_CASE(ragged_cols, 8, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 16, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 32, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 64, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 128, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 256, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 512, x, y, ld, ncols, tile, tabs)
    BRIDCT_RAGGED_CASE(ragged_cols, 1024, x, y, ld, ncols, tile, tabs)
    default: break;
  }
}
__device__ __forceinline__ void ragged_tile_cols_dyn(int h, int mode, float* tile, int P, int w, const float* tabs) {
  switch (h) {
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 8, tile, P, w, tabs)
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 16, tile, P, w, tabs)
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 32, tile, P, w, tabs)
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 64, tile, P, w, tabs)
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 128, tile, P, w, tabs)
    BRIDCT_RAGGED_CASE(ragged_tile_cols, 256, tile, P, w, tabs)
    default: break;
  }
}
__device__ __forceinline__ void ragged_rows_dyn(int w, int mode, float* tile, int nr, const float* tabs) {
  switch (w) {
    BRIDCT_RAGGED_CASE(ragged_rows, 8, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 16, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 32, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 64, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 128, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 256, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 512, tile, nr, tabs)
    BRIDCT_RAGGED_CASE(ragged_rows, 1024, tile, nr, tabs)
    default: break;
  }
}
#undef BRIDCT_RAGGED_CASE

// Rows of one sub-block: what the threads have split-row tasks for, or 128 register rows.
__device__ __forceinline__ int ragged_block_rows(int w) { return w <= 64 ? 128 : w <= 256 ? 32 : w == 512 ? 16 : 8; }

// `rows` rows of width w to shared memory, pitch P, bypassing L1 (row blocks read data that other
// CTAs, or other threads of this one, wrote in this launch).
__device__ __forceinline__ void ragged_load(const float* g, int rows, int w, float* tile, int P) {
  const int sh = 29 - __clz(w);   // log2(w / 4)
  for (int i = threadIdx.x; i < rows << sh; i += kRaggedThreads) {
    const int r = i >> sh, c = (i & ((1 << sh) - 1)) << 2;
    cp_async16(tile + r * P + c, g + 4ll * i);
  }
  cp_async_wait_all();
  __syncthreads();
}

// The row lines of `rows` rows of width w at g; loaded: they already lie in the tile.
__device__ __forceinline__ void ragged_row_pass(float* g, int rows, int w, int mode, bool loaded, float* tile,
                                                const float* tabs) {
  const int P = ragged_pitch(w), step = ragged_block_rows(w), sh = 29 - __clz(w);
  for (int r0 = 0; r0 < rows; r0 += step) {
    const int nr = rows - r0 < step ? rows - r0 : step;
    float* t = loaded ? tile + r0 * P : tile;
    float* gr = g + (long long)r0 * w;
    if (!loaded) ragged_load(gr, nr, w, tile, P);
    ragged_rows_dyn(w, mode, t, nr, tabs);
    if (w >= 128) {
      if (threadIdx.x < nr) {
        bulk_store(gr + (long long)threadIdx.x * w, t + threadIdx.x * P, w * 4);
        bulk_commit_wait();
      }
    } else {
      for (int i = threadIdx.x; i < nr << sh; i += kRaggedThreads)
        *reinterpret_cast<float4*>(gr + 4 * i) =
            *reinterpret_cast<const float4*>(t + (i >> sh) * P + ((i & ((1 << sh) - 1)) << 2));
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kRaggedThreads, 3) k_ragged(RaggedArgs a) {
  extern __shared__ float smem[];
  float* tile = smem;
  float* tabs = smem + kRaggedTile;
  __shared__ int s_index;
  __shared__ RaggedUnit s_unit;
  __shared__ RaggedArray s_array;
  __shared__ int s_ok;
  split_stage_tables<128, kRaggedThreads>(a.tab[0], tabs + ragged_tab<128>());
  split_stage_tables<256, kRaggedThreads>(a.tab[1], tabs + ragged_tab<256>());
  split_stage_tables<512, kRaggedThreads>(a.tab[2], tabs + ragged_tab<512>());
  split_stage_tables<1024, kRaggedThreads>(a.tab[3], tabs + ragged_tab<1024>());
  cp_async_wait_all();
  // Thread 0 takes the next unit while the CTA works on the current one, as long as the queue is long
  // enough that no CTA runs dry for it; a held unit comes after the current one in the queue, so what
  // any row block waits for still makes progress.
  int ahead = -1;
  RaggedUnit next;
  for (;;) {
    if (threadIdx.x == 0) {
      int u = ahead;
      if (u < 0) {
        u = (int)atomicAdd(a.next, 1u);
        if (u < a.nunits) next = a.units[u];
      }
      s_index = u;
      if (u < a.nunits) {
        s_unit = next;
        s_array = a.arrays[next.array];
      }
    }
    __syncthreads();
    const int u = s_index;
    if (u >= a.nunits) break;
    const RaggedUnit unit = s_unit;
    const RaggedArray arr = s_array;
    if (threadIdx.x == 0) ahead = u + 4 * (int)gridDim.x < a.nunits ? (int)atomicAdd(a.next, 1u) : -1;
    auto fetch = [&] {
      if (threadIdx.x == 0 && ahead >= 0 && ahead < a.nunits) next = a.units[ahead];
    };
    const int h = arr.h, w = arr.w, mode = arr.mode;
    const float* xa = a.x + arr.offset;
    float* ya = a.y + arr.offset;
    const bool whole = unit.type() == UNIT_TILE;
    bool rows = unit.type() != UNIT_COLSTRIP;
    int first = 0, count = h;
    if (whole) {
      ragged_load(xa, h, w, tile, ragged_pitch(w));
      ragged_tile_cols_dyn(h, mode, tile, ragged_pitch(w), w, tabs);
      fetch();
    } else if (unit.type() == UNIT_COLSTRIP) {
      ragged_cols_dyn(h, mode, xa + unit.first(), ya + unit.first(), w, unit.count(), tile, tabs);
      fetch();
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) atomicAdd(a.done + unit.array, 1u);
    } else {
      if (threadIdx.x == 0) {
        int ok = 0;
        for (unsigned i = 0; i < a.spin_limit; ++i) {
          unsigned n;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(a.done + unit.array) : "memory");
          if (n >= (unsigned)arr.nstrips) {
            ok = 1;
            break;
          }
          __nanosleep(256);
        }
        if (!ok) atomicExch(a.err, 2);
        __threadfence();
        s_ok = ok;
      }
      fetch();
      __syncthreads();
      // The strips of this launch stored y through the generic proxy; the bulk stores below write the same
      // rows through the async proxy.  No grid boundary lies between, so order the two here.
      asm volatile("fence.proxy.async.global;" ::: "memory");
      rows = s_ok;
      first = unit.first();
      count = unit.count();
    }
    if (rows) ragged_row_pass(ya + (long long)first * w, count, w, mode, whole, tile, tabs);
    __syncthreads();
  }
}

}  // namespace bridct
