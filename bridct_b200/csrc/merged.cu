// Merged passes of a ragged batch: one launch over the column strips (or row blocks) of arrays of many
// shapes.  Each CTA takes the unit of its block index and runs the pass of that unit's line length, so a
// launch holds every length that needs about the same registers and shared memory: columns of 32 and 64
// points, of 128 to 512, and of 1024; rows of 32 and 64, of 128 and 256, of 512, and of 1024.  Batches whose
// launches cost the host more than the device take all modes in one launch too (3 + 4 launches at most
// instead of up to 21); larger ones a launch per mode, whose kernels are faster (fewer line programs in
// the instruction cache).  Batches of mixed arrays, merged, with one launch per length and mode / per
// group and mode / per group, us a call: 16 up to 256 x 256 29 / 31 / 20; 64 up to 1024 x 1024
// 71 / 61 / 43; 200 up to 1024 x 1024 104 / 88 / 81; 640 up to 1024 x 1024 202 / 182 / 192; 1024 of them
// (half in the queue beside) 305 / 296 / 325.
#include "bridct_internal.h"
#include "plain_launch.cuh"

namespace bridct {
namespace {

struct MergedArgs {
  const float* x;
  float* y;
  const MergedUnit* units;
  SplitTables tab[4];   // N = 128, 256, 512, 1024
};

template <bool COL, int N, int MODE>
__device__ __forceinline__ void merged_unit(const MergedArgs& a, const MergedUnit& u, float* smem) {
  const float* x = a.x + u.off;
  float* y = a.y + u.off;
  if constexpr (N >= 128) {
    constexpr int T = COL ? ColGeo<N>::T : RowGeo<N>::T;
    float* tab = smem + (COL ? ColGeo<N>::kTile : RowGeo<N>::kTile);
    split_stage_tables<N, T>(a.tab[N == 128 ? 0 : N == 256 ? 1 : N == 512 ? 2 : 3], tab);
    if constexpr (COL) split_col_unit<N, 0, MODE, col_pairs<N>()>(x, y, u.ld, u.ld, smem, tab);
    else split_row_unit<N, MODE, 8>([&](int r) { return x + r * N; }, [&](int r) { return y + r * N; }, smem, tab);
  } else if constexpr (COL) {
    pair_col_unit<N, MODE>(x, y, u.ld, u.ld);
  } else {
    pair_row_unit<N, MODE>([&](int r) { return y + r * N; }, smem);
  }
}

// Runs the unit if its lines have N points; MODE < 0: in the unit's mode.
template <bool COL, int N, int MODE>
__device__ __forceinline__ void merged_length(const MergedArgs& a, const MergedUnit& u, float* smem) {
  if (u.n != N) return;
  if (MODE >= 0) merged_unit<COL, N, MODE < 0 ? 0 : MODE>(a, u, smem);
  else if (u.mode == LM_FWD) merged_unit<COL, N, LM_FWD>(a, u, smem);
  else if (u.mode == LM_INV) merged_unit<COL, N, LM_INV>(a, u, smem);
  else merged_unit<COL, N, LM_RT>(a, u, smem);
}

template <bool COL, int MODE, int T, int BLOCKS, int... NS>
__global__ void __launch_bounds__(T, BLOCKS) k_merged(MergedArgs a) {
  extern __shared__ float smem[];
  const MergedUnit u = a.units[blockIdx.x];
  griddep_wait();
  griddep_trigger();
  (merged_length<COL, NS, MODE>(a, u, smem), ...);
}

template <bool COL, int N>
constexpr int merged_smem() {
  if constexpr (N >= 128) return COL ? ColGeo<N>::kSmem : RowGeo<N>::kSmem;
  else return COL ? 0 : PairRowGeo<N>::kSmem;
}
template <bool COL, int T, int BLOCKS, int... NS>
cudaError_t launch_merged_kernel(int mode, long long n, const MergedArgs& a, cudaStream_t st) {
  int smem = 0;   // the largest length's
  ((smem = cmax(smem, merged_smem<COL, NS>())), ...);
  const auto k = mode == LM_FWD   ? k_merged<COL, LM_FWD, T, BLOCKS, NS...>
                 : mode == LM_INV ? k_merged<COL, LM_INV, T, BLOCKS, NS...>
                 : mode == LM_RT  ? k_merged<COL, LM_RT, T, BLOCKS, NS...>
                                  : k_merged<COL, -1, T, BLOCKS, NS...>;
  if (kernel_setup(reinterpret_cast<const void*>(k), smem, T) <= 0) return cudaErrorInvalidConfiguration;
  return launch_pdl(k, (unsigned)n, (unsigned)T, smem, st, a);
}

}  // namespace

int merged_class(bool col, int n) { return col ? (n <= 64 ? 0 : n <= 512 ? 1 : 2) : n <= 64 ? 0 : n <= 256 ? 1 : n == 512 ? 2 : 3; }

int merged_strip_cols(int h) {
  return h <= 64 ? PairColGeo<64>::TC : h == 128 ? ColGeo<128>::TC : h == 256 ? ColGeo<256>::TC
         : h == 512 ? ColGeo<512>::TC : ColGeo<1024>::TC;
}
int merged_block_rows(int w) {
  return w <= 64 ? PairRowGeo<64>::RB : w == 128 ? RowGeo<128>::RB : w == 256 ? RowGeo<256>::RB
         : w == 512 ? RowGeo<512>::RB : RowGeo<1024>::RB;
}

cudaError_t launch_merged_pass(const DeviceCtx* d, bool col, int cls, int mode, const MergedUnit* units, long long n, const float* x,
                               float* y, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (n > 0x7FFFFFFFLL) return cudaErrorInvalidValue;
  const MergedArgs a{x, y, units, {d->split[0], d->split[1], d->split[2], d->split[3]}};
  if (col) {
    if (cls == 0) return launch_merged_kernel<true, 32, 12, 64, 32>(mode, n, a, st);
    if (cls == 1) return launch_merged_kernel<true, 128, 5, 512, 256, 128>(mode, n, a, st);
    return launch_merged_kernel<true, 128, 3, 1024>(mode, n, a, st);
  }
  if (cls == 0) return launch_merged_kernel<false, 32, 12, 64, 32>(mode, n, a, st);
  if (cls == 1) return launch_merged_kernel<false, 64, 10, 256, 128>(mode, n, a, st);
  if (cls == 2) return launch_merged_kernel<false, 128, 5, 512>(mode, n, a, st);
  return launch_merged_kernel<false, 128, 3, 1024>(mode, n, a, st);
}

}  // namespace bridct
