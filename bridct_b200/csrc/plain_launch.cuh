// Host-side launch logic of the plain form for one compile-time shape (H, W) and mode.
#pragma once
#include <cuda_runtime.h>
#include "sj_kernels.cuh"
#include "sj_blocks8.cuh"
#include "sj_split.cuh"

namespace bridct {

struct LaunchCtx {
  int sm_count;
};

// lx, ly: general layouts of x and y (both NULL: a contiguous batch).
using PlainLauncher = cudaError_t (*)(const float*, float*, long long, cudaStream_t,
                                      LineTables, const LaunchCtx&, const BatchLayout*, const BatchLayout*);

int kernel_setup(const void* kernel, int smem, int threads, bool all_shared = false);   // bridct_api.cu

// Blocks per SM for a kernel at a given dynamic shared-memory size (set up once per device).
template <typename Kernel>
static int kernel_blocks_per_sm(Kernel k, int smem, int threads) {
  return kernel_setup(reinterpret_cast<const void*>(k), smem, threads);
}

// Launches a plain-form kernel with programmatic stream serialization (see griddep_wait): its
// CTAs may be scheduled, and run up to their first global access, while the previous kernel in
// the stream finishes, which hides most of the launch gap between back-to-back launches (the two
// passes of a two-pass shape, or consecutive calls).
template <typename... Params, typename... Args>
static cudaError_t launch_pdl(void (*k)(Params...), unsigned grid, unsigned threads, int smem, cudaStream_t st,
                              Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// One CTA per strip or row block of a pass of split lines.  The table copy overlaps the previous
// kernel's end (programmatic dependent launch: +1% on 128 MiB batches, +0..4% on 16 MiB ones,
// -4% on 16 MiB of 512-point columns).
template <typename Kernel>
static cudaError_t launch_split(Kernel k, int smem, int threads, long long units, const SplitArgs& a, cudaStream_t st) {
  if (kernel_blocks_per_sm(k, smem, threads) <= 0) return cudaErrorInvalidConfiguration;
  if (units <= 0) return cudaSuccess;
  if (units > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
  return launch_pdl(k, (unsigned)units, (unsigned)threads, smem, st, a);
}

// Narrow units (strips of 8 columns, blocks of 8 rows) take about half the time of a wide one, so they
// pay where the wide ones leave SMs idle.  Measured on batches of 2^16..2^22 elements of nine shapes:
// row blocks of 8 are 10..40% faster below one wide block per SM and 5..25% slower above; strips of 8
// columns (32-byte row segments) are 2..10% faster up to 64 wide strips where the rows are few too,
// and 10..30% slower from 128 strips on.
template <int W> static bool few_rows(long long rows, const LaunchCtx& ctx) { return rows / RowGeo<W>::RB < ctx.sm_count; }

// Column pass x -> y of `batch` H x W arrays (H >= 128).
template <int H, int W, int MODE, bool GEN>
cudaError_t launch_split_cols(const float* x, float* y, long long batch, const BatchLayout& lx, const BatchLayout& ly,
                              SplitTables tab, const LaunchCtx& ctx, cudaStream_t st) {
  using Wide = ColGeo<H>;
  using Few = ColGeo<H, kFewPairs>;
  const SplitArgs a{x, y, tab, W, lx, ly};
  const long long units = batch * (W / Wide::TC);
  if ((units <= 64 && (W < 128 || few_rows<cmax(W, 128)>(batch * H, ctx))) || (GEN && lx.small_units))
    return launch_split(k_split_cols<H, GEN ? 0 : W, MODE, kFewPairs>, Few::kSmem, Few::T, batch * (W / Few::TC), a, st);
  return launch_split(k_split_cols<H, GEN ? 0 : W, MODE, col_pairs<H>()>, Wide::kSmem, Wide::T, units, a, st);
}

// Row pass in place in y (W >= 128).
template <int H, int W, int MODE, bool GEN>
cudaError_t launch_split_rows(float* y, long long batch, const BatchLayout& ly, SplitTables tab, const LaunchCtx& ctx,
                              cudaStream_t st) {
  using Wide = RowGeo<W>;
  using Few = RowGeo<W, kFewPairs>;
  const SplitArgs a{y, y, tab, W, ly, ly};
  if (few_rows<W>(batch * H, ctx) || (GEN && ly.small_units))
    return launch_split(k_split_rows<W, GEN ? H : 0, MODE, kFewPairs>, Few::kSmem, Few::T, batch * H / Few::RB, a, st);
  return launch_split(k_split_rows<W, GEN ? H : 0, MODE, 8>, Wide::kSmem, Wide::T, batch * H / Wide::RB, a, st);
}

// Arrays and threads per CTA, CTAs per SM that the registers are limited for, and whether short axes run one
// line per thread (SINGLE), of the whole-array tiles (k_pair_tile): the fastest of 3 to 10 combinations measured
// per shape.  Shapes up to 64 x 64 run one or two warps per CTA: 12 to 32 independent warps per SM overlap one
// another's loads, transforms and stores, where 128-thread CTAs of the same tiles measured 5..30% slower.  Up to
// 32 points a thread of a full batch runs a pair of lines (32 x 16 and 32 x 32 round trips +5..10% over
// single lines, the others equal).  With 64 points single lines are the faster ones at every size: a pair's 128 values leave the
// compiler no room to overlap anything, and a line at a time makes twice the warps (us a call on 2^25
// elements, pairs / single: 16x64 45.5 / 42.5, 64x32 45.4 / 42.9, round trips 54.1 / 49.0 and 52.0 / 52.1; on 2^20
// elements 4.26 / 3.02 and 3.80 / 3.07).  Shapes with a longer axis take the smallest tile that gives every
// thread a task of both stages, at the register limit that keeps 12 or more warps per SM.
//
// resident: at most so many CTAs share an SM (by the shared memory asked for, in the SM's largest
// configuration; 0: as many as fit).  Where the tiles of two launches fit side by side, each slows the other down,
// and whether they do depended on the configuration that the kernel before had left (2^21 elements of 16x32 in
// one-warp tiles 4.9 or 5.9 us).  16 for one-warp tiles measured fastest of 10 to 18 over 2^19 .. 2^23 elements
// (2^21, 2^21.5 and 2^22 elements of 16x64, no limit / 16: 5.6 / 5.6, 8.8 / 8.1 and 9.7 / 8.9 us), 8 and 10 for two warps
// (2^21.5 and 2^22 elements of 64x64 9.1 / 8.5 and 10.1 / 9.3, of 16x32 7.2 / 6.3 and 8.3 / 7.5).
struct TileCfg {
  int arrays, threads, blocks;
  bool single = false;
  int resident = 0;
};
__host__ __device__ constexpr TileCfg tile_cfg(int h, int w) {
  const int m = cmax(h, w);
  if (m <= 32) return {64 * m / (h * w), 32, m == 32 ? 20 : 24};
  if (m == 64) return h == w ? TileCfg{1, 64, 6, true, 8} : TileCfg{2048 / (h * w), 32, 12, true, 16};
  if (m == 128) {
    if (h <= 16) return {2048 / (h * w), 64, 16};
    if (w == 8) return {4, 64, 10};
    if (w == 16) return {2, 128, 8};
    if (h == 32 || w == 32) return {1, 64, 10};
    if (w == 64) return {1, 128, 3, true};   // 2^21 and 2^25 elements 9.0 / 7.2 and 61 / 57 us, pairs in 64 threads / this
    return {1, 64, 6};
  }
  if (m == 256) {
    if (h <= 16) return {4096 / (h * w), 64, 10};
    if (h == 64 || w == 64) return {1, 128, 3};
    return {h == 32 ? 1 : 32 / w, 128, 5};
  }
  if (m == 512) {
    if (h <= 16) return {8192 / (h * w), 128, 5};
    if (h == 32) return {1, 128, 3};
    if (w == 8) return {1, 64, 8};
    return {1, w == 32 ? 256 : 128, w == 32 ? 2 : 4};
  }
  return {w == 1024 ? 16 / h : 1, 128, 3};
}
// The same for batches that do not fill the GPU (few_tiles): smaller tiles or more threads for one, and single
// lines for short axes, since with about a warp per scheduler a line's instructions are the whole latency and
// a packed one takes two issue cycles (us a call on 2^19 elements, half tiles of pairs / these: 16x32 2.39 / 2.08,
// 32x32 2.53 / 2.05, round trips 2.79 / 2.30 and 3.02 / 2.33; 8x64 round trips 3.87 / 2.77, 16x64 3.16 / 2.28, 32x64
// round trips 4.81 / 2.78; 64x128 on 2^21 8.9 / 7.7).  One-warp tiles of 1024 floats measured up to 20% faster for 32
// points on 2^20.5 and 2^21 elements, but 20..40% slower on 2^20 and 2^21 in processes with many streams.
__host__ __device__ constexpr TileCfg tile_cfg_few(int h, int w) {
  const TileCfg c = tile_cfg(h, w);
  const int m = cmax(h, w);
  if (m <= 16) return {1024 / (h * w), 64, 16, true};
  if (m == 32) return {2048 / (h * w), 64, 8, true, 10};
  if (m == 64) return h == w ? c : TileCfg{2048 / (h * w), 64, 8, true, 10};
  if (m == 128) {
    if (h <= 16 || w == 16 || w == 64) return c;
    if (h == 64) return {1, 128, 3, true};
    if (h == 32) return {1, 128, 7};
    return {c.arrays, 128, 5};
  }
  if (m == 256) {
    if (w == 8) return c;
    if (w == 16) return {1, 128, 5};
    return {c.arrays, c.threads * 2, c.threads == 64 ? 5 : c.blocks == 3 ? 2 : 3};
  }
  if (m == 512) return h == 512 ? (w == 8 ? TileCfg{1, 128, 4} : c) : TileCfg{c.arrays, 256, c.blocks == 5 ? 3 : 2};
  return h == 8 ? TileCfg{1, 128, 3} : w == 8 ? TileCfg{1, 256, 2} : c;
}
// Whether a batch takes the tiles of tile_cfg_few.  waves: of full tiles.
//   * Axes up to 16 points, 32 x 128 and 64 x 128: below a wave, or 1.3 where the second one would be nearly empty
//     (2^22 elements of 8x16 9.4 / 7.9 us, 2^23 of 64x128 22.0 / 19.5; full / these).
//   * 64 points: up to two tiles per SM, and where the last one-warp tiles decide the time (2^21.5 elements of 16x64
//     7.9 / 6.9, 64x16 8.6 / 7.6; 2^21 5.6 / 6.1).
//   * 512x8, 1024x8 and 16x512: where their own wave is nearly full (2^21 elements 10.2 / 8.5 and 11.5 / 10.5; a
//     quarter fewer 7.3 / 7.9 and 9.1 / 9.9).
//   * Others: below a wave, except where the full tiles fit in less than half of the GPU's slots and the smaller ones
//     (twice the slots) do not: back-to-back launches then overlap (programmatic dependent launch), which is
//     worth more (+5..25% at 8 MiB).
static inline bool few_tiles(int h, int w, long long batch, const LaunchCtx& ctx) {
  const TileCfg c = tile_cfg(h, w), f = tile_cfg_few(h, w);
  const int m = cmax(h, w);
  const long long tiles = (batch + c.arrays - 1) / c.arrays, few = (batch + f.arrays - 1) / f.arrays;
  const double waves = (double)tiles / ((double)c.blocks * ctx.sm_count);
  if (m <= 16 || (w == 128 && (h == 32 || h == 64))) return waves < (h == 32 ? 1.0 : 1.3);
  if (m == 64) return tiles <= 2 * ctx.sm_count || (waves > 0.65 && waves < 1);
  if ((w == 8 && h >= 512) || (h == 16 && w == 512)) {
    const double own = (double)few / ((double)f.blocks * ctx.sm_count);
    return own > 0.75 && own <= 1;
  }
  return waves < 1 && (tiles <= ctx.sm_count || waves < 0.225 || waves > 0.45);
}
// Whole arrays up to 16384 floats, except 128 x 128 (register lines of one thread each, below: +15..20%
// over split lines there).
__host__ __device__ constexpr bool pair_tile_route(int h, int w) {
  return h * w <= 16384 && !(h == 128 && w == 128) && !(h == 8 && w == 8);
}

constexpr int kSmemPerSm = 228 * 1024;   // of which a CTA takes 1024 bytes besides its own
template <int H, int W, int MODE, bool GEN, int ARR, int T, int BLOCKS, bool SINGLE, int RESIDENT>
static cudaError_t launch_pair_tile(long long batch, TileArgs a, cudaStream_t st) {
  const auto k = k_pair_tile<H, W, ARR, MODE, T, BLOCKS, GEN, SINGLE>;
  constexpr int need = PairTileGeo<H, W, ARR>::kSmem;
  constexpr int smem = RESIDENT ? cmax(need, (kSmemPerSm / cmax(RESIDENT, 1) - 1024) / 128 * 128) : need;
  if (kernel_setup(reinterpret_cast<const void*>(k), smem, T, RESIDENT > 0) <= 0) return cudaErrorInvalidConfiguration;
  a.ntiles = (batch + ARR - 1) / ARR;
  if (a.ntiles > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
  return launch_pdl(k, (unsigned)a.ntiles, (unsigned)T, smem, st, a);
}

// The classes of a ragged batch that the merged passes take (bridct_ragged_set_schedule): shapes above
// 16384 floats, without the 32768-float arrays in the modes that ran as whole-array tiles before the
// passes of split lines overtook them (the schedules a caller may set stay the same).
__host__ __device__ constexpr bool merged_route(int H, int W, int MODE) {
  const bool whole = H * W == 32768 && (MODE == LM_INV || H == 1024 || H == 64 || (H == 32 && MODE == LM_FWD));
  return H * W > 16384 && !whole;
}

// GEN: the batch has general layouts (strided arrays or an offset table, BatchLayout); the same
// geometry choices run the GEN instantiations of the kernels, except that 8x8 arrays take the
// generic tile kernel instead of the dedicated one-thread-per-array kernels.
template <int H, int W, int MODE, bool GEN>
cudaError_t launch_plain_impl(const float* x, float* y, long long batch, cudaStream_t st,
                              LineTables tab, const LaunchCtx& ctx, const BatchLayout& lx,
                              const BatchLayout& ly) {
  if (batch <= 0) return cudaSuccess;
  if constexpr (H == 8 && W == 8 && !GEN) {
    // Measured on B200 (GB/s, device-resident, back-to-back launches): the double-buffered kernel
    // wins forward/inverse batches up to a few hundred thousand arrays (262,144: 5131 vs 4937)
    // and round trips from about 200,000 (524,288: 5655 vs 5130); the single-buffer kernel
    // wins larger forward batches (1,048,576: 5930 vs 5355) and small round trips.
    const bool db = MODE == LM_RT ? batch >= 196608 : batch <= 393216;
    if (db) {
      auto k = k_blocks8_db<MODE>;
      constexpr int smem = 2 * kB8dbChunks * 16;
      const int bps = kernel_blocks_per_sm(k, smem, kB8dbThreads);
      if (bps <= 0) return cudaErrorInvalidConfiguration;
      const long long ntiles = (batch + kB8dbThreads - 1) / kB8dbThreads;
      long long grid = (long long)ctx.sm_count * bps;
      if (grid > ntiles) grid = ntiles;
      return launch_pdl(k, (unsigned)grid, kB8dbThreads, smem, st, x, y, batch);
    }
    auto k = k_blocks8<MODE>;
    constexpr int smem = kB8Chunks * 16;
    const int bps = kernel_blocks_per_sm(k, smem, kB8Threads);
    if (bps <= 0) return cudaErrorInvalidConfiguration;
    const long long ntiles = (batch + kB8Threads - 1) / kB8Threads;
    long long grid = (long long)ctx.sm_count * bps;
    if (grid > ntiles) grid = ntiles;
    return launch_pdl(k, (unsigned)grid, kB8Threads, smem, st, x, y, batch);
  } else if constexpr (pair_tile_route(H, W)) {
    constexpr TileCfg c = tile_cfg(H, W), f = tile_cfg_few(H, W);
    constexpr bool has_few = f.arrays != c.arrays || f.threads != c.threads;
    const TileArgs a{x, y, 0, batch * H, tab, lx, ly};
    if (has_few && few_tiles(H, W, batch, ctx))
      return launch_pair_tile<H, W, MODE, GEN, f.arrays, f.threads, f.blocks, f.single, f.resident>(batch, a, st);
    return launch_pair_tile<H, W, MODE, GEN, c.arrays, c.threads, c.blocks, c.single, c.resident>(batch, a, st);
  } else if constexpr (H * W <= 16384) {
    // Register tiles, persistent CTAs.  The 128 x 128 round trip is given shared memory for two CTAs per
    // SM only, which measured 2-3% faster than three.
    constexpr int ARR = H == 8 ? 128 : 1, T = H == 8 ? 256 : 128;
    constexpr int smem = H == 128 && MODE == LM_RT ? 110 * 1024 : RegTileGeo<H, W, ARR>::kSmem;
    auto k = k_reg_tile<H, W, ARR, MODE, T, GEN>;
    const int bps = kernel_blocks_per_sm(k, smem, T);
    if (bps <= 0) return cudaErrorInvalidConfiguration;
    const long long tiles = (batch + ARR - 1) / ARR, slots = (long long)ctx.sm_count * bps;
    return launch_pdl(k, (unsigned)(tiles < slots ? tiles : slots), T, smem, st,
                      TileArgs{x, y, tiles, batch * H, tab, lx, ly});
  } else {
    // One column launch and one row launch over the whole batch.
    cudaError_t e;
    if constexpr (H >= 128) {
      e = launch_split_cols<H, W, MODE, GEN>(x, y, batch, lx, ly, tab.col, ctx, st);
    } else {
      using Geo = PairColGeo<H>;
      e = launch_split(k_pair_cols<H, MODE, GEN>, 0, Geo::T, batch * (W / Geo::TC), SplitArgs{x, y, {}, W, lx, ly},
                       st);
    }
    if (e != cudaSuccess) return e;
    if constexpr (W >= 128) {
      return launch_split_rows<H, W, MODE, GEN>(y, batch, ly, tab.row, ctx, st);
    } else {
      using Geo = PairRowGeo<W>;
      return launch_split(k_pair_rows<W, GEN ? H : 0, MODE>, Geo::kSmem, Geo::T, batch * H / Geo::RB,
                          SplitArgs{y, y, {}, W, ly, ly}, st);
    }
  }
}

template <int H, int W, int MODE>
cudaError_t launch_plain(const float* x, float* y, long long batch, cudaStream_t st, LineTables tab,
                         const LaunchCtx& ctx, const BatchLayout* lx, const BatchLayout* ly) {
  if (lx && ly) return launch_plain_impl<H, W, MODE, true>(x, y, batch, st, tab, ctx, *lx, *ly);
  return launch_plain_impl<H, W, MODE, false>(x, y, batch, st, tab, ctx, BatchLayout{}, BatchLayout{});
}

// Per-H instantiation units (plain_inst.cu compiled once per H) export this table row.
void plain_table_row(int h, PlainLauncher (*row)[3]);

}  // namespace bridct
