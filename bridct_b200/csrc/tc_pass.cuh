// Tensor-core precision forms for arrays of any supported shape but 8x8 (tcgen05 + TMEM + TMA).
//
// A 2D transform Y = C_H X C_W^T is computed as two row passes.  A row pass takes a matrix of
// contiguous rows of length L (rows grouped into arrays of R rows), multiplies every row by
// C_L^T (forward) or C_L (inverse) on the tensor cores, and writes every array's result
// transposed:
//     pass 1: rows of X (R = H, L = W)      -> T_b = (X_b C_W^T)^T   (W x H per array)
//     pass 2: rows of T (R = W, L = H)      -> Y_b = (T_b C_H^T)^T = C_H X_b C_W^T
// so the second pass is again a plain row pass.  The host runs the passes over chunks of up to
// 1 GB of arrays (T is plan-owned scratch).
//
// One pass is a GEMM with M = rows (tiles of 128), N = L, K = L.  Each CTA owns one N-block of
// 64 output columns: its slice of C_L (64 x L, split into bf16 or tf32 parts, in the K-major
// 128-byte-swizzled image the UMMA B operand reads) is loaded into shared memory once (L <= 256)
// or arrives chunk by chunk with the ring (L = 512, 1024), and the CTA streams M-tiles through a
// TMA ring in K-chunks (64 FP32 per row for BF16x3, 32 for TF32x3 and for short folded rows).  Rows of 8, 16 or 32 points
// run as 64-float super-rows against a block-diagonal B (SUB).
// Rows of 128 points and more use the symmetry of C_L (PassFold), which halves the products, and for
// every output also the loads and splits:
//   forward  u[j] = (x[j] + x[L-1-j]) / 2 and v[j] = (x[j] - x[L-1-j]) / 2, j < L/2, give the even and the
//            odd coefficients as products of length L/2 with 2 C_L; an N-block is 64 even or 64 odd columns, and the
//            split groups fold the row while they split it
//   inverse  e[j] = sum over even k, o[j] = sum over odd k of C[k][j] X[k], j < L/2, give
//            y[j] = e + o and y[L-1-j] = e - o; the split groups put the even elements of a K-chunk
//            first, e and o accumulate apart, and the epilogue stores 128 columns per N-block
// Split precision as in the 8x8 forms: BF16x3 = six products of 3-way splits, TF32x3 = three
// products of 2-way splits, all accumulated in FP32 in TMEM.
//
// Warp roles (512 threads):
//   warp 0 lane 0  TMA producer: ring stage s <- K-chunk of an M-tile (+ the B chunk when
//                  streamed; waits stage_free)
//   warp 1 lane 0  MMA issuer: TMEM acc set t += splits(stage s, A buffer a) . B slice; commits
//                  stage_free/a_free per chunk and acc_full after an M-tile's last chunk
//   warp 2         TMEM allocator
//   warps 4-7      split group 0 (even K-chunks), warps 8-11 split group 1 (odd K-chunks):
//                  stage s (FP32) -> hi/mid in place + lo into A buffer j % 2
//   warps 12-15    epilogue: sum of acc set t, 16 columns at a time -> transposed stores,
//                  then frees set t
// Every wait is bounded; on expiry the CTA sets *err and all roles leave their loops.
#pragma once
#include "tc_blocks8.cuh"

namespace bridct {
namespace tc {

template <int FORM> struct PassForm;
template <> struct PassForm<BF16X3> {
  static constexpr int kKC = 64;                         // FP32 row elements per K-chunk
  static constexpr int kSplits = 3;
  static constexpr int kStageBytes = kRows * kKC * 4;    // 32 KB (two 32-wide boxes)
  static constexpr int kABufBytes = kRows * kKC * 2;     // Xl (bf16)
};
template <> struct PassForm<TF32X3> {
  static constexpr int kKC = 32;
  static constexpr int kSplits = 2;
  static constexpr int kStageBytes = kRows * kKC * 4;    // 16 KB (one box)
  static constexpr int kABufBytes = kRows * kKC * 4;     // Xl (tf32)
};

constexpr int kBAtom = 64 * 128;         // one K-major SW128 atom column of 64 B rows
constexpr int kPassSmemMax = 232448;     // opt-in shared memory per block
constexpr int kPassMaxStages = 6;
constexpr int kPassThreads = 512;

constexpr int pass_min(int a, int b) { return a < b ? a : b; }

enum PassFold { FOLD_NONE = 0, FOLD_FWD = 1, FOLD_INV = 2 };

// Output columns per CTA (MMA N).  Folded forward passes of 256 points take 128, all columns of one
// parity: with 64, every M-tile crosses from L2 four times, and that traffic (4.9 TB/s) bounds the pass.
// NARROW: half as many, for calls whose wide CTAs would leave half of the SMs idle.  An accumulator's
// products and their order are the same either way (PassAccs), so a row's results have the same
// bits in a call of any size.
__host__ __device__ constexpr int pass_nblock(int L, int fold) { return fold == FOLD_FWD && L == 256 ? 128 : 64; }
__host__ __device__ constexpr bool pass_has_narrow(int L, int fold) {
  return fold == FOLD_INV || (fold == FOLD_FWD && L == 256);
}

// Folded BF16x3 forward passes of 128 and 256 points run K-chunks of 32: the same ring then holds twice
// the stages, and loads, splits and products of one M-tile overlap more finely (16 M elements at 256 x 256:
// 96.4 -> 91.9 us).  512 points measured 221 us that way, 210 with chunks of 64.
__host__ __device__ constexpr bool pass_half(int form, int L, int fold) {
  return form == BF16X3 && fold == FOLD_FWD && L <= 256;
}

// Shared-memory plan of one row pass.  The CTA's slice of the coefficient matrix stays resident when it
// fits beside a two-stage ring; otherwise every ring stage carries the slice's K-chunk next to the A
// chunk (STREAM_B), brought in by a bulk copy from the pre-split image in global memory (L2-resident:
// 0.2-1.5 MB per form and direction).  Narrow inverse passes always stream: their CTAs see one or two M-tiles,
// and loading the slice first would stand before them (512x512 inverse on 2^20 elements 31.1 -> 28.0 us).  A
// folded forward stage holds both halves of the row's chunk, and
// the split parts fill it in place, so that it needs no A buffers.
template <int FORM, int L, int FOLD = FOLD_NONE, bool NARROW = false>
struct PassLayout {
  using F = PassForm<FORM>;
  static constexpr bool kHalf = pass_half(FORM, L, FOLD);
  static constexpr int kKC = kHalf ? 32 : F::kKC;                          // products per K-chunk
  static constexpr int kK = FOLD == FOLD_FWD ? L / 2 : L;                  // products per output
  static constexpr int kChunks = kK / kKC;
  static constexpr int kStageBytes = kRows * kKC * 4;
  static constexpr int kNBlock = pass_nblock(L, FOLD) / (NARROW ? 2 : 1);
  static constexpr int kBlocks = (FOLD == FOLD_INV ? L / 2 : L) / kNBlock;
  static constexpr int kBPart = kBAtom * kNBlock / 64;            // one split part of a K-chunk
  static constexpr int kBBytes = F::kSplits * (kK / F::kKC) * kBPart;   // this CTA's slice of C_L
  static constexpr int kBChunk = F::kSplits * kBPart;             // F::kKC products' part of the slice
  static constexpr int kABufs = FOLD == FOLD_FWD ? 0 : 2;
  static constexpr int kABytes = (FOLD == FOLD_FWD ? 2 : 1) * kStageBytes;   // A data of a stage
  static constexpr int kBarBytes = 1024;
  static constexpr bool kStreamB = (NARROW && FOLD == FOLD_INV) || kBBytes + kABufs * F::kABufBytes + kBarBytes + 1024 + 2 * kABytes > kPassSmemMax;
  static constexpr int kResident = kStreamB ? 0 : kBBytes;
  static constexpr int kStageStride = kABytes + (kStreamB ? kBChunk : 0);
  static constexpr int kStageTx = kStageStride;                  // bytes a stage's loads deliver
  static constexpr int kFixed = kResident + kABufs * F::kABufBytes + kBarBytes + 1024;
  static constexpr int kStages = pass_min(kPassMaxStages, (kPassSmemMax - kFixed) / kStageStride);
  static_assert(kStages >= 2, "pass ring needs two stages");
  static constexpr int kAOff = kStages * kStageStride;
  static constexpr int kBOff = kAOff + kABufs * F::kABufBytes;
  static constexpr int kBarOff = kBOff + kResident;
  static constexpr int kDynamic = kBarOff + kBarBytes + 1024;      // + 1024-byte alignment slack
  static_assert(kDynamic <= kPassSmemMax, "shared memory budget");
  // where the split parts lie: hi at the stage, mid (BF16x3) and lo at these offsets, lo in the A buffer
  // unless folded forward
  static constexpr int kMidOff = kHalf ? 64 : FOLD == FOLD_FWD ? 49152 : 16384;
  static_assert(!kHalf || !kStreamB, "half chunks: resident coefficients");
  static constexpr int kLoOff = 16384;
};

// Bulk copy of `bytes` (a multiple of 16) from global memory into shared memory, completing on bar.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// a_full: one per A buffer, or folded forward (no A buffers) one per stage.
constexpr int kPassTmemSlot = 24 * kPassMaxStages + 48;
struct PassBars {
  uint32_t stage_full, stage_free, a_full, a_free, acc_full, acc_free;
  __device__ explicit PassBars(uint32_t b)
      : stage_full(b), stage_free(b + 8 * kPassMaxStages), a_full(b + 16 * kPassMaxStages),
        a_free(b + 24 * kPassMaxStages), acc_full(b + 24 * kPassMaxStages + 16),
        acc_free(b + 24 * kPassMaxStages + 32) {}
};

// TF32 split of a one-box stage (128 rows x 32 FP32): Xh in place, Xl into the A buffer.
__device__ __forceinline__ void split_box_tf32(uint8_t* stage, uint8_t* abuf, uint32_t r) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t off = sw128(r, j);
    uint4 h, l;
    split_tf32x2(*reinterpret_cast<const float4*>(stage + off), h, l);
    *reinterpret_cast<uint4*>(stage + off) = h;
    *reinterpret_cast<uint4*>(abuf + off) = l;
  }
}

// Folded splits: element i of the folded chunk is (a[i] + sign * b[last - i]) / 2, with a the chunk's row of
// the first half of the matrix row and b that of the mirrored chunk.  Halved, because the sum itself leaves
// FP32's range for inputs above half of it, whose transform does not; the coefficient images hold
// twice the matrix, and both scalings are exact.
// The halving is packed: one instruction for two values.
__device__ __forceinline__ float4 half4(float4 v) {
  asm("{\n .reg .b64 a, h;\n mov.b64 h, {%4, %4};\n"
      " mov.b64 a, {%0, %1};\n mul.rn.f32x2 a, a, h;\n mov.b64 {%0, %1}, a;\n"
      " mov.b64 a, {%2, %3};\n mul.rn.f32x2 a, a, h;\n mov.b64 {%2, %3}, a;\n}\n"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "f"(0.5f));
  return v;
}
// BF16x3: boxes a0, a1, b0, b1 of 16 KB.  hi goes to a0, lo to a1, mid to b1; each half of the chunk
// reads its two source rows completely before it writes there, and lo of the first half, which would
// overwrite a1, waits in registers.
__device__ __forceinline__ void split_fold_bf16(uint8_t* stage, uint32_t r, float hs) {
  uint32_t lo0[4][4];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float x[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 u = half4(*reinterpret_cast<const float4*>(stage + half * 16384u + sw128(r, c)));
      const float4 w = *reinterpret_cast<const float4*>(stage + (half ? 32768u : 49152u) + sw128(r, 7 - c));
      x[4 * c] = fmaf(hs, w.w, u.x);
      x[4 * c + 1] = fmaf(hs, w.z, u.y);
      x[4 * c + 2] = fmaf(hs, w.y, u.z);
      x[4 * c + 3] = fmaf(hs, w.x, u.w);
    }
#pragma unroll
    for (int jq = 0; jq < 4; ++jq) {
      uint32_t hi[4], mid[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) split_bf16x3_pair(x[8 * jq + 2 * e], x[8 * jq + 2 * e + 1], hi[e], mid[e], lo[e]);
      const uint32_t off = sw128(r, half * 4 + jq);
      *reinterpret_cast<uint4*>(stage + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(stage + 49152u + off) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
      if (half) {
        *reinterpret_cast<uint4*>(stage + 16384u + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) lo0[jq][e] = lo[e];
      }
    }
  }
#pragma unroll
  for (int jq = 0; jq < 4; ++jq)
    *reinterpret_cast<uint4*>(stage + 16384u + sw128(r, jq)) =
        make_uint4(lo0[jq][0], lo0[jq][1], lo0[jq][2], lo0[jq][3]);
}
// BF16x3, K-chunks of 32: boxes a, b; a row of box a becomes hi (64 bytes) and mid, that of box b lo.
__device__ __forceinline__ void split_fold_bf16_half(uint8_t* stage, uint32_t r, float hs) {
  float4 w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(stage + 16384u + sw128(r, j));
  uint32_t mid[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {   // elements 8q .. 8q + 7
    const float4 u0 = half4(*reinterpret_cast<const float4*>(stage + sw128(r, 2 * q)));
    const float4 u1 = half4(*reinterpret_cast<const float4*>(stage + sw128(r, 2 * q + 1)));
    const float4 w0 = w[7 - 2 * q], w1 = w[6 - 2 * q];
    uint32_t hi[4], lo[4];
    split_bf16x3_pair(fmaf(hs, w0.w, u0.x), fmaf(hs, w0.z, u0.y), hi[0], mid[q][0], lo[0]);
    split_bf16x3_pair(fmaf(hs, w0.y, u0.z), fmaf(hs, w0.x, u0.w), hi[1], mid[q][1], lo[1]);
    split_bf16x3_pair(fmaf(hs, w1.w, u1.x), fmaf(hs, w1.z, u1.y), hi[2], mid[q][2], lo[2]);
    split_bf16x3_pair(fmaf(hs, w1.y, u1.z), fmaf(hs, w1.x, u1.w), hi[3], mid[q][3], lo[3]);
    *reinterpret_cast<uint4*>(stage + sw128(r, q)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(stage + 16384u + sw128(r, q)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<uint4*>(stage + sw128(r, 4 + q)) = make_uint4(mid[q][0], mid[q][1], mid[q][2], mid[q][3]);
}
// TF32x3: boxes a, b; hi goes to a, lo to b.
__device__ __forceinline__ void split_fold_tf32(uint8_t* stage, uint32_t r, float hs) {
  float4 w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(stage + 16384u + sw128(r, j));
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t off = sw128(r, j);
    const float4 u = half4(*reinterpret_cast<const float4*>(stage + off));
    uint4 h, l;
    split_tf32x2(make_float4(fmaf(hs, w[7 - j].w, u.x), fmaf(hs, w[7 - j].z, u.y), fmaf(hs, w[7 - j].y, u.z),
                             fmaf(hs, w[7 - j].x, u.w)),
                 h, l);
    *reinterpret_cast<uint4*>(stage + off) = h;
    *reinterpret_cast<uint4*>(stage + 16384u + off) = l;
  }
}
// Deinterleaving splits (inverse): the chunk's even elements go to K positions 0.., the odd ones to the
// second half.  BF16x3: as split_tile<BF16X3>, with half `half` of the row giving 16 even elements
// (16-byte pieces 2 half, 2 half + 1) and 16 odd ones (pieces 4 + 2 half, ...).
__device__ __forceinline__ void split_deint_bf16(uint8_t* stage, uint8_t* abuf, uint32_t r) {
  uint32_t mid0[4][4];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float x[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 u = *reinterpret_cast<const float4*>(stage + half * 16384u + sw128(r, c));
      x[4 * c] = u.x; x[4 * c + 1] = u.y; x[4 * c + 2] = u.z; x[4 * c + 3] = u.w;
    }
#pragma unroll
    for (int jq = 0; jq < 4; ++jq) {
      const int odd = jq >> 1, piece = odd * 4 + half * 2 + (jq & 1);
      uint32_t hi[4], mid[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = (jq & 1) * 16 + 4 * e + odd;   // elements i and i + 2 of this half
        split_bf16x3_pair(x[i], x[i + 2], hi[e], mid[e], lo[e]);
      }
      const uint32_t off = sw128(r, piece);
      *reinterpret_cast<uint4*>(stage + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(abuf + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      if (half) {
        *reinterpret_cast<uint4*>(stage + 16384u + off) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) mid0[jq][e] = mid[e];
      }
    }
  }
#pragma unroll
  for (int jq = 0; jq < 4; ++jq)
    *reinterpret_cast<uint4*>(stage + 16384u + sw128(r, (jq >> 1) * 4 + (jq & 1))) =
        make_uint4(mid0[jq][0], mid0[jq][1], mid0[jq][2], mid0[jq][3]);
}
// TF32x3: 32 elements of a row, even ones to 16-byte pieces 0..3, odd ones to 4..7.
__device__ __forceinline__ void split_deint_tf32(uint8_t* stage, uint8_t* abuf, uint32_t r) {
  float x[32];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float4 u = *reinterpret_cast<const float4*>(stage + sw128(r, c));
    x[4 * c] = u.x; x[4 * c + 1] = u.y; x[4 * c + 2] = u.z; x[4 * c + 3] = u.w;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int i = (j & 3) * 8 + (j >> 2);
    uint4 h, l;
    split_tf32x2(make_float4(x[i], x[i + 2], x[i + 4], x[i + 6]), h, l);
    const uint32_t off = sw128(r, j);
    *reinterpret_cast<uint4*>(stage + off) = h;
    *reinterpret_cast<uint4*>(abuf + off) = l;
  }
}

// Accumulator set of one M-tile (N-block TMEM columns per block: NB = 64 or 128).  The FP32 accumulation of an MMA
// into a large accumulator loses the addends' low bits toward zero, so the dominant Xh.Ch
// product accumulates apart from the small products (whose own losses are then negligible),
// and over long K it is spread over kBig group accumulators by K-chunk, each receiving few
// MMAs.  Products sharing an A split go into one MMA with the B splits stacked along N:
//   BF16x3 blocks [big0 | small | smaller | big1]:
//     Xh.[Ch|Cm|Cl] -> [big0|small|smaller] (group 0) or Xh.Ch -> big1, Xh.[Cm|Cl] -> [small|smaller]
//     Xm.[Ch|Cm] -> [small|smaller],  Xl.Ch -> small
//   TF32x3 blocks [big0 | small | big1 | big2]:
//     Xh.[Ch|Cl] -> [big0|small] (group 0) or Xh.Ch -> big_g, Xh.Cl -> small;  Xl.Ch -> small
// The epilogue adds the blocks in FP32.
// SETS accumulator sets share the 512 TMEM columns (PassSets): two, so that the epilogue of one M-tile
// overlaps the MMAs of the next, for rows up to 256 points; one for 512- and 1024-point rows, whose long K
// needs more group accumulators than two sets leave room for (TF32x3 round trips of 1024-point
// axes exceeded 3e-6 with three groups; one set holds seven for TF32x3, six for BF16x3).
// PARS = 2 (folded inverse): a set holds the blocks of e, then those of o, half as many for each.
// MERGE: BF16x3 adds all small products in one block, [big0 | small | big1 ..].  This makes room for the
// second set of a 128-column N-block (forward, 256 points: 91.9 -> 67 us per call on 16 M elements, with
// the errors of one K = 128 group per output, as in the unfolded pass) and of the inverses up to 256
// points (104 -> 95 us; 128 points 73 -> 59; 86.5 and 56 with the products issued as in issue_merged_mmas), and at 512 and 1024 points keeps a big group to no more MMAs
// than in an unfolded pass (errors against float64 1.75e-7 -> 1.57e-7 at 512 x 512, 2.77e-7 -> 2.65e-7 at
// 1024 x 1024; with two groups 2.01e-7 and 3.73e-7).  TF32x3 has nothing to give up: its folded passes of
// 256 points forward and 128 and 256 inverse keep one set, and its inverses of 512 and 1024 points are not
// folded (launch_pass).
// WIDE: the N-block that the number of group accumulators is counted for (NB, or twice NB in a narrow pass, so
// that both spread a product over the same groups).
template <int FORM, int CHUNKS, int SETS, int PARS, int NB, int WIDE, bool MERGE>
struct PassAccs {
  static constexpr int kNBlock = NB;
  static constexpr bool kMerge = MERGE;
  static constexpr int kSmallBlocks = FORM == BF16X3 && !MERGE ? 2 : 1;
  static constexpr int kMaxBig = 512 / (SETS * PARS * WIDE) - kSmallBlocks;
  static constexpr int kBig = CHUNKS < kMaxBig ? CHUNKS : kMaxBig;
  static constexpr int kPerParity = (1 + kSmallBlocks + (kBig - 1)) * NB;
  static constexpr int kPerTile = PARS * kPerParity;                               // columns
  static constexpr int kExtraBig = (1 + kSmallBlocks) * NB;                        // big1 column
  static constexpr int kAlloc = SETS * kPerTile <= 256 ? 256 : 512;
  static_assert(kBig >= 1 && SETS * kPerTile <= 512, "TMEM columns");
  __host__ __device__ static constexpr int group(int kc) { return kc * kBig / CHUNKS; }
};

// Accumulator sets, and whether the small products share a block (see PassAccs).
template <int FORM, int L, int FOLD> struct PassSets {
  static constexpr bool kMerge = FORM == BF16X3 && ((FOLD == FOLD_FWD && L == 256) || FOLD == FOLD_INV);
  static constexpr int value = L >= 512                                   ? 1
                               : FORM == BF16X3 || FOLD == FOLD_NONE      ? 2
                               : FOLD == FOLD_FWD && L == 128             ? 2
                                                                          : 1;
};

// Descriptor of the operand `bytes` (a multiple of 16) after that of d: the start address lies in the low
// bits of the low word, which shared memory's size keeps from overflowing.
__device__ __forceinline__ uint64_t desc_at(uint64_t d, uint32_t bytes) {
  return (d & 0xFFFFFFFF00000000ull) | ((uint32_t)d + (bytes >> 4));
}

// The products of a chunk with the small ones merged (PassAccs::kMerge).  One thread issues them, and its
// instructions bound the long inverse passes: descriptors by an addition each, and no choice within the
// chunk (16 M elements, inverse: 1024x1024 412 -> 346 us, 512x512 208 -> 179; 2^18 of 512x512 28.3 -> 26.8).  The
// products that are not merged gain nothing that way (512x512 forward 210 -> 213).  FIRST (group 0): the big block and the small one lie side by side, so one product reads Xh for both.
template <typename A, int PARS, int NB, int STEPS, bool FIRST>
__device__ __forceinline__ void issue_merged_mmas(uint32_t hi, uint32_t mid, uint32_t lo, uint32_t bchunk, int kc,
                                                  uint32_t tmem) {
  constexpr uint32_t kPart = kBAtom * NB / 64, i1 = instr_desc(1, NB);
  constexpr int kSteps = STEPS / PARS;
  const uint64_t dh = sw128_desc(hi), dm = sw128_desc(mid), dl = sw128_desc(lo), db = sw128_desc(bchunk);
  const int g = A::group(kc);
  const uint32_t clear = FIRST ? (kc != 0) : A::group(kc - 1) == g;
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    const uint32_t t = tmem + (uint32_t)(k / kSteps) * A::kPerParity;
    const uint32_t c = k % kSteps == 0 ? clear : 1u;
    const uint64_t bd = desc_at(db, k * 32u), bm = desc_at(db, kPart + k * 32u), ah = desc_at(dh, k * 32u);
    if constexpr (FIRST) {
      umma(t, ah, bd, instr_desc(1, 2 * NB), c, BF16X3);
    } else {
      umma(t + A::kExtraBig + (uint32_t)(g - 1) * NB, ah, bd, i1, c, BF16X3);
      umma(t + NB, ah, bm, i1, 1u, BF16X3);
    }
    umma(t + NB, ah, desc_at(db, 2 * kPart + k * 32u), i1, 1u, BF16X3);
    umma(t + NB, desc_at(dm, k * 32u), bd, i1, 1u, BF16X3);
    umma(t + NB, desc_at(dm, k * 32u), bm, i1, 1u, BF16X3);
    umma(t + NB, desc_at(dl, k * 32u), bd, i1, 1u, BF16X3);
  }
}

// Split products of K-chunk kc (one thread): hi, mid, lo: shared addresses of the A parts (mid: BF16x3
// only).  bchunk: shared address of the chunk's B splits, laid out [split][8 KB atom column of 64 rows].
// tmem: column 0 of this M-tile's set.  With PARS = 2 the first half of a chunk's steps are e's.
// STEPS: K steps of a chunk (two in half chunks).
template <int FORM, typename A, int PARS, int NB, int STEPS>
__device__ __forceinline__ void issue_pass_mmas(uint32_t hi, uint32_t mid, uint32_t lo, uint32_t bchunk, int kc,
                                                uint32_t tmem) {
  if constexpr (A::kMerge) {
    if (A::kBig == 1 || A::group(kc) == 0) issue_merged_mmas<A, PARS, NB, STEPS, true>(hi, mid, lo, bchunk, kc, tmem);
    else issue_merged_mmas<A, PARS, NB, STEPS, false>(hi, mid, lo, bchunk, kc, tmem);
    return;
  }
  constexpr uint32_t kPart = kBAtom * NB / 64;
  const int g = A::group(kc);
  const bool big_first = kc == 0 || A::group(kc - 1) != g;
  constexpr int kSteps = STEPS / PARS;   // K steps of one parity in a chunk
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {   // 32 bytes of a row per MMA: 16 bf16 or 8 tf32
    const uint32_t t = tmem + (uint32_t)(k / kSteps) * A::kPerParity;
    const uint32_t big_g = t + A::kExtraBig + (uint32_t)(g - 1) * NB;
    const bool first = k % kSteps == 0;
    const uint64_t bd = sw128_desc(bchunk + k * 32u);
    const uint64_t ah = sw128_desc(hi + k * 32u);
    const uint32_t clear = (kc == 0 && first) ? 0u : 1u, clear_g = (big_first && first) ? 0u : 1u;
    if constexpr (FORM == BF16X3) {
      constexpr uint32_t i3 = instr_desc(1, NB == 64 ? 192 : 256), i2 = instr_desc(1, 2 * NB), i1 = instr_desc(1, NB);
      if (g == 0 && NB == 64) {
        umma(t, ah, bd, i3, clear, BF16X3);
      } else if (g == 0) {   // N = 384 does not fit one MMA
        umma(t, ah, bd, i2, clear, BF16X3);
        umma(t + 2 * NB, ah, sw128_desc(bchunk + 2 * kPart + k * 32u), i1, clear, BF16X3);
      } else {
        umma(big_g, ah, bd, i1, clear_g, BF16X3);
        umma(t + NB, ah, sw128_desc(bchunk + kPart + k * 32u), i2, 1u, BF16X3);
      }
      umma(t + NB, sw128_desc(mid + k * 32u), bd, i2, 1u, BF16X3);   // Xm
      umma(t + NB, sw128_desc(lo + k * 32u), bd, i1, 1u, BF16X3);    // Xl
    } else {
      constexpr uint32_t i2 = instr_desc(2, 2 * NB), i1 = instr_desc(2, NB);
      if (g == 0) {
        umma(t, ah, bd, i2, clear, TF32X3);
      } else {
        umma(big_g, ah, bd, i1, clear_g, TF32X3);
        umma(t + NB, ah, sw128_desc(bchunk + kPart + k * 32u), i1, 1u, TF32X3);
      }
      umma(t + NB, sw128_desc(lo + k * 32u), bd, i1, 1u, TF32X3);   // Xl
    }
  }
}

// Columns q*16 .. q*16+15 of one parity's accumulator blocks at taddr: the sum of the big groups and that
// of the small products.
template <typename ACC>
__device__ __forceinline__ void load_parts(uint32_t taddr, int q, float (&big)[16], float (&sm)[16]) {
  float w[16];
  tmem_ld16(taddr + q * 16, big);
  tmem_ld16(taddr + ACC::kNBlock + q * 16, sm);
  tmem_wait_ld();
#pragma unroll
  for (int a = 0; a < ACC::kSmallBlocks - 1; ++a) {
    tmem_ld16(taddr + (2 + a) * ACC::kNBlock + q * 16, w);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) sm[i] += w[i];
  }
#pragma unroll
  for (int a = 1; a < ACC::kBig; ++a) {
    tmem_ld16(taddr + ACC::kExtraBig + (a - 1) * ACC::kNBlock + q * 16, w);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) big[i] += w[i];
  }
}

// xmap: the (nrows x L) FP32 row matrix (box 32 x 128, SWIZZLE_128B).  out: destination of
// the transposed arrays (R rows per array, rshift = log2 R).  bimage: kBlocks slices of
// PassLayout::kBBytes.  Grid: a multiple of kBlocks CTAs; CTA c computes N-block c % kBlocks.
// SUB > 1 (rows of LS = 64 / SUB = 8, 16 or 32 points): L = 64 and every matrix row holds SUB
// consecutive rows of length LS (a super-row); B is block-diagonal (SUB copies of C_LS), so
// column n = j * LS + c of super-row g is output column c of row g * SUB + j, and nrows counts
// super-rows.
// FOLD: see the file comment (L >= 128).  Folded forward, N-block i holds the columns
// 2 (NB (i / 2) + n) + i % 2 (NB columns); folded inverse, the columns NB i + n and L - 1 - (NB i + n).
template <int FORM, int L, int SUB = 1, int FOLD = FOLD_NONE, bool NARROW = false>
__global__ void __launch_bounds__(kPassThreads, 1)
    k_tcpass(const __grid_constant__ CUtensorMap xmap, float* __restrict__ out,
             const uint4* __restrict__ bimage, long long nrows, int rshift, int* __restrict__ err) {
  static_assert(SUB == 1 || L == 64, "super-rows are 64 floats");
  static_assert(FOLD == FOLD_NONE || (SUB == 1 && L >= 128), "folded rows");
  constexpr int LS = L / SUB;   // points per original row
  using PL = PassLayout<FORM, L, FOLD, NARROW>;
  using F = PassForm<FORM>;
  constexpr int kStages = PL::kStages;
  constexpr int kChunks = PL::kChunks;
  constexpr int kSets = PassSets<FORM, L, FOLD>::value;
  constexpr int kPars = FOLD == FOLD_INV ? 2 : 1;
  using ACC = PassAccs<FORM, kChunks, kSets, kPars, PL::kNBlock, pass_nblock(L, FOLD), PassSets<FORM, L, FOLD>::kMerge>;
  constexpr uint32_t kTileCols = ACC::kPerTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(base);
  const PassBars bars(sbase + PL::kBarOff);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base + PL::kBarOff + kPassTmemSlot);
  __shared__ volatile int s_abort;
  __shared__ volatile int s_group_ok[3];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int nblk = blockIdx.x % PL::kBlocks;
  const long long slot = blockIdx.x / PL::kBlocks;
  const long long nslots = gridDim.x / PL::kBlocks;
  const long long mtiles = (nrows + kRows - 1) / kRows;
  const long long ntile_local = slot < mtiles ? (mtiles - 1 - slot) / nslots + 1 : 0;
  const long long nchunk_local = ntile_local * kChunks;

  if (tid == 0) {
    s_abort = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bars.stage_full + 8 * i, 1);
      mbar_init(bars.stage_free + 8 * i, 1);
      mbar_init(bars.a_full + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars.a_free + 8 * i, 1);
      mbar_init(bars.acc_full + 8 * i, 1);
      mbar_init(bars.acc_free + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(ACC::kAlloc));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if constexpr (!PL::kStreamB) {
    const uint4* src = bimage + (size_t)nblk * (PL::kBBytes / 16);
    uint4* dst = reinterpret_cast<uint4*>(base + PL::kBOff);
    for (int i = tid; i < PL::kBBytes / 16; i += kPassThreads) dst[i] = __ldg(src + i);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  // Launched with programmatic stream serialization: the prologue above (barriers, TMEM, the
  // coefficient image, which no kernel writes) overlaps the previous grid's tail; the data is
  // touched only after the wait.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0 && lane == 0) {
    for (long long j = 0; j < nchunk_local && ok && !s_abort; ++j) {
      const int s = (int)(j % kStages);
      ok = mbar_wait(bars.stage_free + 8 * s, ((uint32_t)(j / kStages) & 1u) ^ 1u);
      if (!ok) break;
      const long long m = slot + (j / kChunks) * nslots;
      const int kc = (int)(j % kChunks);
      const uint32_t dst = sbase + s * PL::kStageStride;
      mbar_expect_tx(bars.stage_full + 8 * s, PL::kStageTx);
      tma_load_2d(dst, &xmap, kc * PL::kKC, (int)(m * kRows), bars.stage_full + 8 * s);
      if constexpr (PL::kKC == 64)
        tma_load_2d(dst + 16384u, &xmap, kc * PL::kKC + 32, (int)(m * kRows), bars.stage_full + 8 * s);
      if constexpr (FOLD == FOLD_FWD) {   // the mirrored chunk
#pragma unroll
        for (int b = 0; b < PL::kKC / 32; ++b)
          tma_load_2d(dst + PL::kStageBytes + b * 16384u, &xmap, L - (kc + 1) * PL::kKC + b * 32, (int)(m * kRows),
                      bars.stage_full + 8 * s);
      }
      if constexpr (PL::kStreamB)
        bulk_load(dst + PL::kABytes,
                  reinterpret_cast<const uint8_t*>(bimage) + (size_t)nblk * PL::kBBytes + (size_t)kc * PL::kBChunk,
                  PL::kBChunk, bars.stage_full + 8 * s);
    }
  } else if (warp == 1 && lane == 0) {
    for (long long j = 0; j < nchunk_local && ok && !s_abort; ++j) {
      const int s = (int)(j % kStages), a = (int)(j & 1);
      const long long jt = j / kChunks;
      const int kc = (int)(j % kChunks), t = (int)(jt % kSets);
      ok = FOLD == FOLD_FWD ? mbar_wait(bars.a_full + 8 * s, (uint32_t)(j / kStages) & 1u)
                            : mbar_wait(bars.a_full + 8 * a, (uint32_t)(j >> 1) & 1u);
      if (ok && kc == 0) ok = mbar_wait(bars.acc_free + 8 * t, ((uint32_t)(jt / kSets) & 1u) ^ 1u);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sstage = sbase + s * PL::kStageStride;
      const uint32_t bchunk = PL::kStreamB ? sstage + PL::kABytes
                              : PL::kHalf  ? sbase + PL::kBOff + (uint32_t)(kc >> 1) * PL::kBChunk + (uint32_t)(kc & 1) * 64u
                                           : sbase + PL::kBOff + (uint32_t)kc * PL::kBChunk;
      issue_pass_mmas<FORM, ACC, kPars, PL::kNBlock, PL::kHalf ? 2 : 4>(
          sstage, sstage + PL::kMidOff,
          FOLD == FOLD_FWD ? sstage + PL::kLoOff : sbase + PL::kAOff + a * F::kABufBytes, bchunk, kc,
          tmem_base + t * kTileCols);
      umma_commit(bars.stage_free + 8 * s);
      if (FOLD != FOLD_FWD) umma_commit(bars.a_free + 8 * a);
      if (kc == kChunks - 1) umma_commit(bars.acc_full + 8 * t);
    }
    if (ok && nchunk_local > 0) {   // the last MMAs must finish before TMEM is freed
      const long long j = nchunk_local - 1;
      ok = mbar_wait(bars.stage_free + 8 * (int)(j % kStages), (uint32_t)(j / kStages) & 1u);
    }
  } else if (warp >= 4 && warp < 12) {
    const int grp = (warp - 4) >> 2;              // 0: even K-chunks, 1: odd K-chunks
    const uint32_t r = tid - 128 - 128 * grp;
    const int bar_id = grp ? 3 : 1, ok_slot = grp ? 2 : 0;
    for (long long j = grp; j < nchunk_local; j += 2) {
      const int s = (int)(j % kStages), a = (int)(j & 1);
      if (r == 0) {
        bool g = !s_abort && ring_wait<kStages>(bars.stage_full + 8 * s, bars.stage_free + 8 * s, (uint32_t)(j / kStages));
        if (FOLD != FOLD_FWD && g) g = mbar_wait(bars.a_free + 8 * a, ((uint32_t)(j >> 1) & 1u) ^ 1u);
        s_group_ok[ok_slot] = g ? 1 : 0;
      }
      named_sync(bar_id, 128);
      if (!s_group_ok[ok_slot]) {
        ok = r != 0;
        break;
      }
      uint8_t* stage = base + s * PL::kStageStride;
      uint8_t* abuf = base + PL::kAOff + a * F::kABufBytes;
      if constexpr (FOLD == FOLD_FWD) {
        const float hs = nblk & 1 ? -0.5f : 0.5f;
        if constexpr (PL::kHalf) split_fold_bf16_half(stage, r, hs);
        else if constexpr (FORM == BF16X3) split_fold_bf16(stage, r, hs);
        else split_fold_tf32(stage, r, hs);
      } else if constexpr (FOLD == FOLD_INV) {
        if constexpr (FORM == BF16X3) split_deint_bf16(stage, abuf, r);
        else split_deint_tf32(stage, abuf, r);
      } else {
        if constexpr (FORM == BF16X3) split_tile<BF16X3>(stage, abuf, r);
        else split_box_tf32(stage, abuf, r);
      }
      fence_async_smem();
      named_sync(bar_id, 128);
      if (r == 0) mbar_arrive(bars.a_full + 8 * (FOLD == FOLD_FWD ? s : a));
    }
  } else if (warp >= 12) {
    const uint32_t r = tid - 384;                 // tile row = TMEM lane
    const uint32_t quarter = (uint32_t)(warp & 3) * 32u;
    const long long rmask = (1ll << rshift) - 1;
    for (long long jt = 0; jt < ntile_local; ++jt) {
      const int t = (int)(jt % kSets);
      if (r == 0)
        s_group_ok[1] = (!s_abort && mbar_wait(bars.acc_full + 8 * t, (uint32_t)(jt / kSets) & 1u)) ? 1 : 0;
      named_sync(2, 128);
      if (!s_group_ok[1]) {
        ok = r != 0;
        break;
      }
      tc_fence_after();
      // row g = (array b, row h of that array); its column n goes to out[b][n][h].  With
      // super-rows, column n = j * LS + c of super-row g goes to out[b][c][h0 + j], h0 = g * SUB
      // within its array (SUB divides R, so a super-row lies in one array).
      const long long g = (slot + jt * nslots) * kRows + r;
      const bool live = g < nrows;
      const long long g0 = g * SUB;
      const long long b = g0 >> rshift, h = g0 & rmask;
      const uint32_t taddr = tmem_base + t * kTileCols + (quarter << 16);
      float* arr = out + ((b * LS) << rshift) + h;
      if constexpr (FOLD == FOLD_INV) {
        float* lo = arr + ((long long)(nblk * PL::kNBlock) << rshift);
        float* hi = arr + ((long long)(L - 1 - nblk * PL::kNBlock) << rshift);
#pragma unroll
        for (int q = 0; q < PL::kNBlock / 16; ++q) {
          float e[16], o[16], es[16], os[16];
          load_parts<ACC>(taddr, q, e, es);
          load_parts<ACC>(taddr + ACC::kPerParity, q, o, os);
          if (live) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const long long c = (long long)(q * 16 + i) << rshift;
              // the small sums join the smaller addend first: one rounding less at the size of the result
              lo[c] = e[i] + (o[i] + (os[i] + es[i]));
              hi[-c] = e[i] - (o[i] + (os[i] - es[i]));
            }
          }
        }
      } else {
        float* dst = arr + ((long long)(FOLD == FOLD_FWD ? (nblk >> 1) * 2 * PL::kNBlock + (nblk & 1)
                                                         : nblk * PL::kNBlock) << rshift);
#pragma unroll
        for (int q = 0; q < PL::kNBlock / 16; ++q) {
          float v[16], sm[16];
          load_parts<ACC>(taddr, q, v, sm);
          if (live) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              constexpr int kLS = LS;
              const int n = q * 16 + i, j = n / kLS, c = n % kLS * (FOLD == FOLD_FWD ? 2 : 1);
              dst[((long long)c << rshift) + j] = v[i] + sm[i];
            }
          }
        }
      }
      tc_fence_before();
      named_sync(2, 128);
      if (r == 0) mbar_arrive(bars.acc_free + 8 * t);
    }
  }
  if (!ok) {
    s_abort = 1;
    atomicExch(err, 1);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(ACC::kAlloc));
  }
}

}  // namespace tc
}  // namespace bridct
