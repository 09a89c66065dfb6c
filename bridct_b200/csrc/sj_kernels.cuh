// Shared pieces of the plain (Shao-Johnson FP32) kernels, and the tile kernel of register lines.
//
// Shape classes (h, w powers of two in [8, 1024]; plain_launch.cuh picks the kernel):
//   8 x 8            sj_blocks8.cuh, one thread per array
//   h*w <= 16384     k_pair_tile (sj_split.cuh): a CTA holds whole arrays in shared memory, runs every
//                    column line, then every row line; one HBM read and one write per element.
//                    128 x 128, and 8 x 8 arrays in general layouts, run k_reg_tile (here).
//   h*w >  16384     two passes, columns x -> y, then rows in place in y, one launch each over the whole
//                    batch (k_split_cols, k_split_rows, k_pair_cols, k_pair_rows; the reference's rect
//                    route does the same pair of passes, vertical then bands, src/generated/rect.c:5-23).
#pragma once
#include "sj_lines.cuh"

namespace bridct {

// Rotation tables of the split lines (sj_split.cuh), in global memory.
struct SplitTables {
  const float* t = nullptr;   // tw, then post (SplitTab<N>::kFloats floats, 16-byte aligned)
};

struct LineTables {
  SplitTables col;   // for line length h (used when h >= 128)
  SplitTables row;   // for line length w (used when w >= 128)
};

// Where the arrays of a launch live in a general layout (kernels instantiated with GEN): array b
// starts at offs[b] when an offset table is given (the shape classes of a ragged batch), else at
// b * bs (a strided batch), and its rows are ld floats apart.  Array starts and ld are multiples of
// 4 floats, so every row is 16-byte aligned.  Contiguous batches (array b at b*h*w, rows w apart)
// use the kernels' fixed addressing instead.
struct BatchLayout {
  const long long* offs = nullptr;
  long long bs = 0;
  long long ld = 0;
  int small_units = 0;   // two-pass shapes: force the narrow strips and row blocks
};

struct TileArgs {
  const float* x;
  float* y;
  long long ntiles;
  long long rows_total;   // rows of the (batch*h) x w matrix covered by this launch
  LineTables tab;
  BatchLayout lx, ly;     // layouts of x and y (GEN kernels only)
};

// Offset (floats) of row g of the (batch*H) x W row matrix in a general layout.
template <int H>
__device__ __forceinline__ long long layout_row(const BatchLayout& l, long long g) {
  const long long b = g / H;
  const int r = (int)(g % H);
  return (l.offs ? __ldg(l.offs + b) : b * l.bs) + (long long)r * l.ld;
}

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int cmin(int a, int b) { return a < b ? a : b; }
// Asynchronous global -> shared copies (cp.async, 16 bytes, through L2 only).  The issuing thread waits with cp_async_wait_all; a barrier then publishes the data.
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Runs `nlines` lines of length N, one thread per line; line l starts at tile + off(l), elements at
// stride es.
template <int N, int MODE, typename Off>
__device__ __forceinline__ void run_lines(float* tile, int nlines, int es, const Off& off) {
  for (int l = threadIdx.x; l < nlines; l += blockDim.x) reg_line<N, MODE>(tile + off(l), es);
}

// Tiles of whole arrays whose lines run in one thread's registers, scalar: ARR arrays of H x W, rows
// W + 4 floats apart.  128 x 128: 128-point lines (168 registers), 128 threads, one array per CTA.
// 8 x 8 in general layouts: the line programs of the contiguous 8 x 8 kernels, hence their bits; arrays
// 8 (mod 32) floats apart, so that the column walks of the four arrays under a warp differ in banks.
template <int H, int W, int ARR> struct RegTileGeo {
  static constexpr int P = W + 4;
  static constexpr int AP = W == 8 ? H * P + (40 - H * P % 32) % 32 : H * P;
  static constexpr int kSmem = ARR * AP * 4;
};
template <int H, int W, int ARR, int MODE, int T, bool GEN>
__global__ void __launch_bounds__(T) k_reg_tile(TileArgs a) {
  using Geo = RegTileGeo<H, W, ARR>;
  constexpr int P = Geo::P, AP = Geo::AP, TR = ARR * H, Q = W / 4;
  extern __shared__ float smem[];
  griddep_wait();
  auto srow = [](int r) { return (r / H) * AP + (r % H) * P; };
  for (long long t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    if (t + gridDim.x >= a.ntiles) griddep_trigger();   // this CTA's last tile
    const long long first = t * TR;
    const int rows = a.rows_total - first < TR ? (int)(a.rows_total - first) : TR;
    for (int i = threadIdx.x; i < rows * Q; i += T) {
      const int r = i / Q, c = (i % Q) * 4;
      cp_async16(smem + srow(r) + c, GEN ? a.x + layout_row<H>(a.lx, first + r) + c : a.x + (first + r) * W + c);
    }
    cp_async_wait_all();
    __syncthreads();
    run_lines<H, MODE>(smem, ARR * W, P, [](int l) { return (l / W) * AP + (l % W); });
    __syncthreads();
    run_lines<W, MODE>(smem, TR, 1, srow);
    __syncthreads();
    for (int i = threadIdx.x; i < rows * Q; i += T) {
      const int r = i / Q, c = (i % Q) * 4;
      *reinterpret_cast<float4*>(GEN ? a.y + layout_row<H>(a.ly, first + r) + c : a.y + (first + r) * W + c) =
          *reinterpret_cast<const float4*>(smem + srow(r) + c);
    }
    __syncthreads();
  }
}

}  // namespace bridct
