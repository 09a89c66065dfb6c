// Long lines (128..1024 points) of the plain form, two lines per thread.
//
// A line of N = A * B points is split in two stages: stage 1 runs, for each residue b < B, the
// SJ scaled real FFT of length A of v[B a + b] (v: Makhoul's reorder of x); stage 2 runs, for each
// column c < A / 2, the SJ scaled complex FFT of length B over the twiddled stage-1 outputs and the
// post rotation that gives y[c + A d] and y[N - c - A d].  The real columns 0 and A/2 make one
// stage-2 task together (sjp_special), so a line has B stage-1 and A/2 stage-2 tasks of 2B values.
//
// What bounds long lines is instruction issue (about 35 thread instructions per element and pass
// when one warp holds whole lines and each thread one value at a time), so here
//   * a thread runs the same task of TWO lines in packed f32x2 arithmetic (F2): one issue slot does
//     two additions or multiply-adds, and one 64-bit access moves two values.  The packed
//     instructions run at half the rate of the scalar ones, so the arithmetic pipe is as busy as
//     before and half the issue slots are free for everything else;
//   * the lanes of a warp hold different lines at the same (or a few adjacent) b or c, so twiddles
//     and post coefficients are broadcast loads, offsets are compile-time constants and nothing is
//     conflicted or gathered;
//   * column lines come from and go to global memory directly (a row of the strip is one coalesced
//     segment): shared memory carries the stage-1 / stage-2 exchange only, one write and one read
//     per element instead of six.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "sj_kernels.cuh"

namespace bridct {

// ---- value types of the packed programs --------------------------------------------------------
struct F2 {
  unsigned long long v = 0;
};
__device__ __forceinline__ F2 f2_make(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vsub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 vneg(F2 a) {
  float x, y;
  f2_split(a, x, y);
  return f2_make(-x, -y);
}
__device__ __forceinline__ F2 vmul(F2 a, float c) { return vmul(a, f2_make(c, c)); }
__device__ __forceinline__ F2 vfma(F2 a, float c, F2 b) { return vfma(a, f2_make(c, c), b); }
__device__ __forceinline__ F2 vfms(F2 a, float c, F2 b) { return vfma(a, f2_make(c, c), vneg(b)); }
// The same operations on one line.  The intrinsics round once each and are never contracted, so one line at
// a time gives the bits of two at a time.
struct F1 {
  float v = 0.0f;
};
__device__ __forceinline__ F1 vadd(F1 a, F1 b) { return F1{__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vsub(F1 a, F1 b) { return F1{__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vmul(F1 a, float c) { return F1{__fmul_rn(a.v, c)}; }
__device__ __forceinline__ F1 vneg(F1 a) { return F1{-a.v}; }
__device__ __forceinline__ F1 vfma(F1 a, float c, F1 b) { return F1{__fmaf_rn(a.v, c, b.v)}; }
__device__ __forceinline__ F1 vfms(F1 a, float c, F1 b) { return F1{__fmaf_rn(a.v, c, -b.v)}; }

}  // namespace bridct

#include "sj_packed.cuh"

namespace bridct {

// ---- split geometry and tables ------------------------------------------------------------
template <int N> struct Split;
template <> struct Split<128> { static constexpr int A = 16, B = 8; };
template <> struct Split<256> { static constexpr int A = 32, B = 8; };
template <> struct Split<512> { static constexpr int A = 32, B = 16; };
// 64 * 16 rather than 32 * 32: the real columns' task, which one warp runs besides its own, is then
// short (32 M elements of 1024-point columns 53.7 -> 49.9 us, rows 60.5 -> 58.2, round trips -5..8%).
template <> struct Split<1024> { static constexpr int A = 64, B = 16; };

template <int A> struct Leaf;
template <> struct Leaf<16> {
  static __device__ __forceinline__ void fwd(const F2 (&x)[16], F2 (&w)[16]) { sjp_rfft_16<F2>(x, w); }
  static __device__ __forceinline__ void tr(const F2 (&w)[16], F2 (&x)[16]) { sjp_rfft_16_t<F2>(w, x); }
};
template <> struct Leaf<32> {
  static __device__ __forceinline__ void fwd(const F2 (&x)[32], F2 (&w)[32]) { sjp_rfft_32<F2>(x, w); }
  static __device__ __forceinline__ void tr(const F2 (&w)[32], F2 (&x)[32]) { sjp_rfft_32_t<F2>(w, x); }
};
template <> struct Leaf<64> {
  static __device__ __forceinline__ void fwd(const F2 (&x)[64], F2 (&w)[64]) { sjp_rfft_64<F2>(x, w); }
  static __device__ __forceinline__ void tr(const F2 (&w)[64], F2 (&x)[64]) { sjp_rfft_64_t<F2>(w, x); }
};
template <int B> struct Stage2;
#define BRIDCT_STAGE2(B)                                                                       \
  template <> struct Stage2<B> {                                                               \
    static __device__ __forceinline__ void fwd(F2 (&z)[2 * B]) { sjp_cfft_##B<F2>(z); }        \
    static __device__ __forceinline__ void tr(F2 (&z)[2 * B]) { sjp_cfft_##B##_t<F2>(z); }     \
    static __device__ __forceinline__ void sfwd(F2 (&z)[2 * B]) { sjp_special_##B<F2>(z); }    \
    static __device__ __forceinline__ void str(F2 (&z)[2 * B]) { sjp_special_##B##_t<F2>(z); } \
  };
BRIDCT_STAGE2(8)
BRIDCT_STAGE2(16)
#undef BRIDCT_STAGE2

// Rotations of one line length, A/2 * B of each kind:
//   tw[c * B + b]          (x, y) = w_N^{b c} s(A, c), c = 1..A/2-1
//   post[j * A/2 + c]      (P, Q): y[k] = P vr + Q vi and y[N-k] = Q vr - P vi for complex stage-2
//     output j of task c (k = c + A j; task 0: see sjp_special, its output 0 is y[0] = P vr and
//     y[N/2] = Q vi)
// Each CTA keeps them in shared memory: read through L1 they cost the row pass a third of its time.
// Up to 512 points every coefficient is stored twice, so that one 128-bit load gives two packed
// operands without a move per coefficient; 1024-point lines have no room for that.
template <int N> struct SplitTab {
  static constexpr bool kDup = N <= 512;
  static constexpr int kEntries = Split<N>::A / 2 * Split<N>::B;   // of each kind
  static constexpr int kWords = kDup ? 4 : 2;                      // floats of an entry
  static constexpr int kFloats = 2 * kEntries * kWords;
};
// Starts copying the tables to shared memory (cp.async: the caller waits and synchronizes).
template <int N, int T>
__device__ __forceinline__ void split_stage_tables(SplitTables tab, float* s) {
  for (int i = threadIdx.x; i < SplitTab<N>::kFloats / 4; i += T) cp_async16(s + 4 * i, tab.t + 4 * i);
}
// Entry i of the tables at t (shared memory) as two packed operands.
template <int N>
__device__ __forceinline__ void split_coef(const float* t, int i, F2& a, F2& b) {
  if constexpr (SplitTab<N>::kDup) {
    const float4 v = *reinterpret_cast<const float4*>(t + 4 * i);
    a = f2_make(v.x, v.y);
    b = f2_make(v.z, v.w);
  } else {
    const float2 v = *reinterpret_cast<const float2*>(t + 2 * i);
    a = f2_make(v.x, v.x);
    b = f2_make(v.y, v.y);
  }
}

// Stage-1 tail: the twiddled columns 1..A/2-1 and the two real columns into the exchange slots
// ex(c, part), part 0 = re and 1 = im (task 0: columns 0 and A/2).
template <int N, typename Put>
__device__ __forceinline__ void split_put(const F2 (&w)[Split<N>::A], int b, const float* tab, const Put& put) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  put(0, 0, w[0]);
  put(0, 1, w[A / 2]);
#pragma unroll
  for (int c = 1; c < A / 2; ++c) {
    F2 tx, ty;
    split_coef<N>(tab, c * B + b, tx, ty);
    const F2 wr = w[c], wi = w[A / 2 + c];
    put(c, 0, vfma(vneg(wi), ty, vmul(wr, tx)));
    put(c, 1, vfma(wi, tx, vmul(wr, ty)));
  }
}
// Its transpose.
template <int N, typename Get>
__device__ __forceinline__ void split_get(F2 (&w)[Split<N>::A], int b, const float* tab, const Get& get) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  w[0] = get(0, 0);
  w[A / 2] = get(0, 1);
#pragma unroll
  for (int c = 1; c < A / 2; ++c) {
    F2 tx, ty;
    split_coef<N>(tab, c * B + b, tx, ty);
    const F2 tr = get(c, 0), ti = get(c, 1);
    w[c] = vfma(ti, ty, vmul(tr, tx));
    w[A / 2 + c] = vfma(vneg(tr), ty, vmul(ti, tx));
  }
}

// Stage 2 of task c on its 2B exchange values z, with the post rotation: on return z[2j] and z[2j+1]
// are y[k_j] and y[N - k_j] (y[0] and y[N/2] for j = 0 of task 0).
template <int N>
__device__ __forceinline__ void split_stage2(F2 (&z)[2 * Split<N>::B], int c, const float* tab) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  if (c == 0) Stage2<B>::sfwd(z);
  else Stage2<B>::fwd(z);
  const float* post = tab + SplitTab<N>::kEntries * SplitTab<N>::kWords;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    F2 p, q;
    split_coef<N>(post, j * (A / 2) + c, p, q);
    const F2 vr = z[2 * j], vi = z[2 * j + 1];
    z[2 * j] = vmul(vr, p);
    z[2 * j + 1] = vmul(j == 0 && c == 0 ? vi : vr, q);
    if (j > 0 || c != 0) {
      z[2 * j] = vfma(vi, q, z[2 * j]);
      z[2 * j + 1] = vfma(vneg(vi), p, z[2 * j + 1]);
    }
  }
}
// Its transpose: z holds y[k_j], y[N - k_j] on entry and the adjoint exchange values on return.
template <int N>
__device__ __forceinline__ void split_stage2_t(F2 (&z)[2 * Split<N>::B], int c, const float* tab) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  const float* post = tab + SplitTab<N>::kEntries * SplitTab<N>::kWords;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    F2 p, q;
    split_coef<N>(post, j * (A / 2) + c, p, q);
    const F2 yk = z[2 * j], yn = z[2 * j + 1];
    z[2 * j] = vmul(yk, p);
    z[2 * j + 1] = vmul(j == 0 && c == 0 ? yn : yk, q);
    if (j > 0 || c != 0) {
      z[2 * j] = vfma(yn, q, z[2 * j]);
      z[2 * j + 1] = vfma(vneg(yn), p, z[2 * j + 1]);
    }
  }
  if (c == 0) Stage2<B>::str(z);
  else Stage2<B>::tr(z);
}

// Calls f(slot, k): z[slot] of task c is y[k].
template <int N, typename Fn>
__device__ __forceinline__ void split_outputs(int c, const Fn& f) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  if (c == 0) {
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int k = j < B / 2 ? A * j : A / 2 + 2 * A * (j - B / 2);
      f(2 * j, k);
      f(2 * j + 1, j == 0 ? N / 2 : N - k);
    }
  } else {
#pragma unroll
    for (int j = 0; j < B; ++j) {
      f(2 * j, c + A * j);
      f(2 * j + 1, N - A * j - c);
    }
  }
}

// Source row (Makhoul) of element a of residue b: v[n], n = B a + b.
template <int N>
__device__ __forceinline__ int split_src(int a, int b) {
  constexpr int A = Split<N>::A, B = Split<N>::B;
  return a < A / 2 ? 2 * B * a + 2 * b : 2 * N - 1 - 2 * B * a - 2 * b;
}

// ---- the lines of a tile in shared memory ---------------------------------------------------------
// GROUPS groups of LP line pairs, T threads: thread t holds pair t % LP and tasks t / LP, ... (group
// major) of either stage.  get(g, i) is element i of the thread's pair of group g, put(g, i, v) takes
// the result, ex(g) is the thread's place in the first of the group's N exchange slots, which lie ES
// floats apart.  The exchange may overlie what get() reads: a barrier lies between.  IN_PLACE: put()
// may also overlie the exchange.
// Slot (c, part, b) is number c * 2B + part * B + (b ^ (c % S)), S = 16 / LP: where a half-warp spans
// several tasks c, their slots of one b then lie in different banks.  Threads with on(g) false (pairs
// that a short unit does not have) only take part in the barriers.
struct AllPairs {
  __device__ __forceinline__ bool operator()(int) const { return true; }
};
template <int N, int MODE, int T, int GROUPS, int LP, bool IN_PLACE, typename Get, typename Put, typename Ex,
          typename On = AllPairs>
__device__ __forceinline__ void split_lines(const Get& get, const Put& put, const Ex& ex, int ES, const float* tab,
                                            const On& on = On()) {
  constexpr int A = Split<N>::A, B = Split<N>::B, S = LP < 16 ? 16 / LP : 1;
  auto at = [](float* e) -> F2& { return *reinterpret_cast<F2*>(e); };
  constexpr int N1 = GROUPS * B * LP, N2 = GROUPS * (A / 2) * LP;   // threads' tasks of the two stages
  constexpr int R1 = (N1 + T - 1) / T, R2 = (N2 + T - 1) / T;
  static_assert(N1 % 32 == 0 && N2 % 32 == 0, "whole warps");
  const int t = threadIdx.x / LP;
  constexpr int TP = T / LP;
  auto on1 = [&](int r) { return (N1 % T == 0 || (int)threadIdx.x + r * T < N1) && on((t + r * TP) / B); };
  auto on2 = [&](int r) { return (N2 % T == 0 || (int)threadIdx.x + r * T < N2) && on((t + r * TP) / (A / 2)); };
  if constexpr (MODE != LM_INV) {
    F2 w[R1][A];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int i = t + r * TP, g = i / B, b = i % B;
      if (on1(r)) {
        F2 v[A];
#pragma unroll
        for (int e = 0; e < A; ++e) v[e] = get(g, split_src<N>(e, b));
        Leaf<A>::fwd(v, w[r]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int i = t + r * TP, g = i / B, b = i % B;
      if (on1(r)) {
        float* e = ex(g);
        split_put<N>(w[r], b, tab, [&](int c, int part, F2 val) {
          at(e + (b ^ (c % S)) * ES + (c * 2 + part) * (B * ES)) = val;
        });
      }
    }
    __syncthreads();
    F2 z[IN_PLACE && MODE == LM_FWD ? R2 : 1][2 * B];
#pragma unroll
    for (int r = 0; r < R2; ++r) {
      const int i = t + r * TP, g = i / (A / 2), c = i % (A / 2);
      F2(&zr)[2 * B] = z[IN_PLACE && MODE == LM_FWD ? r : 0];
      if (on2(r)) {
        float* e = ex(g) + c * (2 * B * ES);
#pragma unroll
        for (int q = 0; q < B; ++q) {
          float* eq = e + ((q % S) ^ (c % S)) * ES + (q - q % S) * ES;
          zr[2 * q] = at(eq);
          zr[2 * q + 1] = at(eq + B * ES);
        }
        split_stage2<N>(zr, c, tab);
        if constexpr (MODE == LM_RT) {
          split_stage2_t<N>(zr, c, tab);
#pragma unroll
          for (int q = 0; q < B; ++q) {
            float* eq = e + ((q % S) ^ (c % S)) * ES + (q - q % S) * ES;
            at(eq) = zr[2 * q];
            at(eq + B * ES) = zr[2 * q + 1];
          }
        } else if constexpr (!IN_PLACE) {
          split_outputs<N>(c, [&](int j, int k) { put(g, k, zr[j]); });
        }
      }
    }
    if constexpr (MODE == LM_RT || IN_PLACE) __syncthreads();
    if constexpr (MODE == LM_FWD && IN_PLACE) {
#pragma unroll
      for (int r = 0; r < R2; ++r) {
        const int i = t + r * TP, g = i / (A / 2), c = i % (A / 2);
        if (on2(r)) split_outputs<N>(c, [&](int j, int k) { put(g, k, z[r][j]); });
      }
    }
  } else {
    F2 z[R2][2 * B];
#pragma unroll
    for (int r = 0; r < R2; ++r) {
      const int i = t + r * TP, g = i / (A / 2), c = i % (A / 2);
      if (on2(r)) {
        split_outputs<N>(c, [&](int j, int k) { z[r][j] = get(g, k); });
        split_stage2_t<N>(z[r], c, tab);
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R2; ++r) {
      const int i = t + r * TP, g = i / (A / 2), c = i % (A / 2);
      if (on2(r)) {
        float* e = ex(g) + c * (2 * B * ES);
#pragma unroll
        for (int q = 0; q < B; ++q) {
          float* eq = e + ((q % S) ^ (c % S)) * ES + (q - q % S) * ES;
          at(eq) = z[r][2 * q];
          at(eq + B * ES) = z[r][2 * q + 1];
        }
      }
    }
    __syncthreads();
  }
  if constexpr (MODE != LM_FWD) {
    F2 v[IN_PLACE ? R1 : 1][A];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int i = t + r * TP, g = i / B, b = i % B;
      F2(&vr)[A] = v[IN_PLACE ? r : 0];
      if (on1(r)) {
        float* e = ex(g);
        F2 w[A];
        split_get<N>(w, b, tab, [&](int c, int part) {
          return at(e + (b ^ (c % S)) * ES + (c * 2 + part) * (B * ES));
        });
        Leaf<A>::tr(w, vr);
        if constexpr (!IN_PLACE) {
#pragma unroll
          for (int e2 = 0; e2 < A; ++e2) put(g, split_src<N>(e2, b), vr[e2]);
        }
      }
    }
    if constexpr (IN_PLACE) {
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        const int i = t + r * TP, g = i / B, b = i % B;
        if (on1(r)) {
#pragma unroll
          for (int e = 0; e < A; ++e) put(g, split_src<N>(e, b), v[r][e]);
        }
      }
    }
  }
}

// ---- column pass -------------------------------------------------------------------------------
struct SplitArgs {
  const float* x;
  float* y;
  SplitTables tab;
  int width;              // run-time layouts: columns of an array
  BatchLayout lx, ly;     // run-time layouts
};

// A strip of TC columns is copied to shared memory (cp.async: loads into registers would be limited
// by the L1 that the exchange leaves), transformed, and stored from registers, each row of the strip
// one coalesced segment.  A thread holds two adjacent columns.  Strips of 16 columns are 64 bytes
// wide: rows 2k and 2k + 1 share a 128-byte line and swap places in every other line, so that the
// rows 2b, 2b + 2 (stage 1) and c, c + 1 (stage 2) which a half-warp reads lie in different banks.
// Calls on a few arrays take strips of 8 columns (LP = 4), so that they spread over more SMs.
template <int N> __host__ __device__ constexpr int col_pairs() { return N >= 512 ? 8 : 16; }
constexpr int kFewPairs = 4;
template <int N, int LP = col_pairs<N>()> struct ColGeo {
  static constexpr int TC = 2 * LP;
  static constexpr int T = 128;
  // resident CTAs that the registers are limited for (32 M elements of 512-point columns: 45.6 us, 52.0
  // unlimited; 1024: 49.9 and 60.2; 256-point round trips 51.7 and 61.8)
  static constexpr int kBlocks = LP == kFewPairs ? 1 : N == 128 ? 8 : N == 256 ? 6 : N == 512 ? 5 : 3;
  static constexpr int kTile = N * TC;   // the strip, then the exchange
  static constexpr int kSmem = (kTile + SplitTab<N>::kFloats) * 4;
};
template <int TC>
__device__ __forceinline__ int strip_row(int r) {
  return TC == 16 ? (r >> 1) * 32 + (((r ^ (r >> 1)) & 1) << 4) : r * TC;
}

// One strip: x and y at its first element, rows xp / yp floats apart (W > 0: W apart).
template <int N, int W, int MODE, int LP>
__device__ __forceinline__ void split_col_unit(const float* x, float* y, long long xp, long long yp, float* smem,
                                               const float* tab) {
  using Geo = ColGeo<N, LP>;
  constexpr int TC = Geo::TC, Q = TC / 4, T = Geo::T;
#pragma unroll
  for (int k = 0; k < N * Q / T; ++k) {
    const int i = threadIdx.x + k * T, r = i / Q, c = (i % Q) * 4;
    cp_async16(smem + strip_row<TC>(r) + c, x + (W > 0 ? (long long)(r * W) : r * xp) + c);
  }
  cp_async_wait_all();
  __syncthreads();
  const int p = 2 * (threadIdx.x % LP);
  float* yt = y + p;
  split_lines<N, MODE, T, 1, LP, false>(
      [&](int, int i) {
        const float2 v = *reinterpret_cast<const float2*>(smem + strip_row<TC>(i) + p);
        return f2_make(v.x, v.y);
      },
      [&](int, int i, F2 v) {
        float2 f;
        f2_split(v, f.x, f.y);
        *reinterpret_cast<float2*>(yt + (W > 0 ? (long long)(i * W) : i * yp)) = f;
      },
      [&](int) { return smem + p; }, TC, tab);
}

// W > 0: strips of contiguous N x W arrays; W = 0: run-time layouts.
template <int N, int W, int MODE, int LP>
__global__ void __launch_bounds__(ColGeo<N, LP>::T, ColGeo<N, LP>::kBlocks) k_split_cols(SplitArgs a) {
  using Geo = ColGeo<N, LP>;
  constexpr int TC = Geo::TC;
  extern __shared__ float smem[];
  float* tab = smem + Geo::kTile;
  split_stage_tables<N, Geo::T>(a.tab, tab);
  griddep_wait();
  griddep_trigger();
  if constexpr (W > 0) {
    constexpr int S = W / TC;
    const unsigned arr = blockIdx.x / S, s = blockIdx.x % S;
    const long long off = (long long)arr * N * W + s * TC;
    split_col_unit<N, W, MODE, LP>(a.x + off, a.y + off, W, W, smem, tab);
  } else {
    const unsigned S = a.width / TC, arr = blockIdx.x / S, s = blockIdx.x % S;
    split_col_unit<N, 0, MODE, LP>(a.x + layout_row<N>(a.lx, (long long)arr * N) + s * TC,
                                   a.y + layout_row<N>(a.ly, (long long)arr * N) + s * TC, a.lx.ld, a.ly.ld, smem, tab);
  }
}

// ---- row pass ----------------------------------------------------------------------------------
// Rows are staged whole in shared memory in groups of 2 LP, at pitch N + 32 / LP floats: a thread holds
// rows p and p + LP of a group, and a warp LP such pairs at 32 / LP adjacent c's (or b's), so the
// scalar walks along the rows hit bank (32 / LP) p + c in stage 2: conflict-free.  Stage 1 walks every
// second sample (bank (32 / LP) p + 2 b), two lanes to a bank.
// One group per CTA: 64 threads give 128- and 256-point lines a stage-1 task each, and ten to sixteen
// such CTAs per SM hide one another's barriers and copies (32 M elements of 256-point rows: 49.7 us,
// 53.7 as two groups in 128 threads, 63.1 without the register limit; 128: 48.8, 512: 52.0, 1024: 58.2).
template <int N, int LP = 8> struct RowGeo {
  static constexpr int P = N + 32 / LP;
  static constexpr int T = LP == 8 && N <= 256 ? 64 : 128;
  static constexpr int kBlocks = LP != 8 ? 1 : N == 128 ? 16 : N == 256 ? 10 : N == 512 ? 5 : 3;
  static constexpr int RB = 2 * LP;
  static constexpr int kTile = RB * P;
  static constexpr int kSmem = (kTile + SplitTab<N>::kFloats) * 4;
};

// All rows of a tile of GROUPS groups of 2 LP rows at pitch P.
template <int N, int MODE, int T, int GROUPS, int LP>
__device__ __forceinline__ void split_rows(float* tile, const float* tab) {
  constexpr int P = N + 32 / LP, GP = 2 * LP * P;
  const int p = threadIdx.x % LP;
  float* rows = tile + p * P;
  split_lines<N, MODE, T, GROUPS, LP, true>(
      [&](int g, int i) { return f2_make(rows[g * GP + i], rows[g * GP + i + LP * P]); },
      [&](int g, int i, F2 v) { f2_split(v, rows[g * GP + i], rows[g * GP + i + LP * P]); },
      [&](int g) { return tile + g * GP + 2 * p; }, 2 * LP, tab);
}

// Stores `bytes` (a multiple of 16) of shared memory to global memory asynchronously.
__device__ __forceinline__ void bulk_store(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(static_cast<unsigned>(__cvta_generic_to_shared(src))), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_wait() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Orders this thread's shared-memory writes before bulk stores that read them.  The global side needs
// no fence where a grid boundary lies between the ordinary stores to the rows and the bulk stores to
// them (the two passes, whole-array tiles); the queue of a ragged batch adds its own (ragged.cuh).
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// RB rows, row r at xrow(r) and yrow(r), in place or x -> y.
template <int N, int MODE, int LP, typename XRow, typename YRow>
__device__ __forceinline__ void split_row_unit(const XRow& xrow, const YRow& yrow, float* smem, const float* tab) {
  using Geo = RowGeo<N, LP>;
  constexpr int P = Geo::P, RB = Geo::RB, T = Geo::T, Q = N / 4;
  auto srow = [&](int r) { return smem + r * P; };
#pragma unroll
  for (int k = 0; k < RB * Q / T; ++k) {
    const int i = threadIdx.x + k * T, r = i / Q, c = (i % Q) * 4;
    cp_async16(srow(r) + c, xrow(r) + c);
  }
  cp_async_wait_all();
  __syncthreads();
  split_rows<N, MODE, T, Geo::RB / (2 * LP), LP>(smem, tab);
  fence_async();
  __syncthreads();
  if (threadIdx.x < RB) {
    bulk_store(yrow(threadIdx.x), srow(threadIdx.x), N * 4);
    bulk_commit_wait();
  }
}

// RB consecutive rows of a (batch * H) x N matrix per CTA.  H = 0: contiguous rows; H > 0: run-time
// layouts of arrays of H rows.
template <int N, int H, int MODE, int LP>
__global__ void __launch_bounds__(RowGeo<N, LP>::T, RowGeo<N, LP>::kBlocks) k_split_rows(SplitArgs a) {
  using Geo = RowGeo<N, LP>;
  extern __shared__ float smem[];
  float* tab = smem + Geo::kTile;
  split_stage_tables<N, Geo::T>(a.tab, tab);
  griddep_wait();
  griddep_trigger();
  const long long first = (long long)blockIdx.x * Geo::RB;
  if constexpr (H == 0) {
    split_row_unit<N, MODE, LP>([&](int r) { return a.x + (first + r) * N; },
                                [&](int r) { return a.y + (first + r) * N; }, smem, tab);
  } else {
    split_row_unit<N, MODE, LP>([&](int r) { return a.x + layout_row<H>(a.lx, first + r); },
                                [&](int r) { return a.y + layout_row<H>(a.ly, first + r); }, smem, tab);
  }
}

// ---- lines of 64 points and fewer: two per thread (V = F2) or one (V = F1) in registers --------
template <int N, int MODE, typename V>
__device__ __forceinline__ void pair_line(V (&v)[N]) {
  static_assert(N <= 64, "register lines");
  if constexpr (N == 8) MODE == LM_FWD ? sjp_fwd_8<V>(v) : MODE == LM_INV ? sjp_inv_8<V>(v) : sjp_rt_8<V>(v);
  if constexpr (N == 16) MODE == LM_FWD ? sjp_fwd_16<V>(v) : MODE == LM_INV ? sjp_inv_16<V>(v) : sjp_rt_16<V>(v);
  if constexpr (N == 32) MODE == LM_FWD ? sjp_fwd_32<V>(v) : MODE == LM_INV ? sjp_inv_32<V>(v) : sjp_rt_32<V>(v);
  if constexpr (N == 64) MODE == LM_FWD ? sjp_fwd_64<V>(v) : MODE == LM_INV ? sjp_inv_64<V>(v) : sjp_rt_64<V>(v);
}
// Two rows in shared memory, in place: 128-bit accesses (8 consecutive rows at a pitch of 4 mod 32
// floats are 4 banks apart).
template <int N, int MODE>
__device__ __forceinline__ void pair_rows(float* r0, float* r1) {
  F2 v[N];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 p = *reinterpret_cast<const float4*>(r0 + i), q = *reinterpret_cast<const float4*>(r1 + i);
    v[i] = f2_make(p.x, q.x);
    v[i + 1] = f2_make(p.y, q.y);
    v[i + 2] = f2_make(p.z, q.z);
    v[i + 3] = f2_make(p.w, q.w);
  }
  pair_line<N, MODE>(v);
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    float4 p, q;
    f2_split(v[i], p.x, q.x);
    f2_split(v[i + 1], p.y, q.y);
    f2_split(v[i + 2], p.z, q.z);
    f2_split(v[i + 3], p.w, q.w);
    *reinterpret_cast<float4*>(r0 + i) = p;
    *reinterpret_cast<float4*>(r1 + i) = q;
  }
}

// One row in shared memory, in place.
template <int N, int MODE>
__device__ __forceinline__ void single_row(float* r) {
  F1 v[N];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 p = *reinterpret_cast<const float4*>(r + i);
    v[i].v = p.x;
    v[i + 1].v = p.y;
    v[i + 2].v = p.z;
    v[i + 3].v = p.w;
  }
  pair_line<N, MODE>(v);
#pragma unroll
  for (int i = 0; i < N; i += 4)
    *reinterpret_cast<float4*>(r + i) = make_float4(v[i].v, v[i + 1].v, v[i + 2].v, v[i + 3].v);
}

// Column pass of 32- and 64-point columns: a thread holds two adjacent columns, straight from and to
// global memory (a warp's row segment is 256 bytes).
template <int N> struct PairColGeo {
  static constexpr int T = 32;
  static constexpr int TC = 2 * T;
};
template <int N, int MODE>
__device__ __forceinline__ void pair_col_unit(const float* x, float* y, long long xp, long long yp) {
  x += 2 * threadIdx.x;
  y += 2 * threadIdx.x;
  F2 v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    // not __ldg: the previous kernel of the stream may still be writing x until griddep_wait() returns
    const float2 f = *reinterpret_cast<const float2*>(x + i * xp);
    v[i] = f2_make(f.x, f.y);
  }
  pair_line<N, MODE>(v);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float2 f;
    f2_split(v[i], f.x, f.y);
    *reinterpret_cast<float2*>(y + i * yp) = f;
  }
}
template <int N, int MODE, bool GEN>
__global__ void __launch_bounds__(32) k_pair_cols(SplitArgs a) {
  constexpr int TC = PairColGeo<N>::TC;
  griddep_wait();
  griddep_trigger();
  const unsigned S = a.width / TC, arr = blockIdx.x / S, s = blockIdx.x % S;
  if constexpr (GEN) {
    pair_col_unit<N, MODE>(a.x + layout_row<N>(a.lx, (long long)arr * N) + s * TC,
                           a.y + layout_row<N>(a.ly, (long long)arr * N) + s * TC, a.lx.ld, a.ly.ld);
  } else {
    const long long off = (long long)arr * N * a.width + s * TC;
    pair_col_unit<N, MODE>(a.x + off, a.y + off, a.width, a.width);
  }
}

// Row pass of 32- and 64-point rows in place: 64 rows per warp, staged in shared memory.
template <int N> struct PairRowGeo {
  static constexpr int T = 32;
  static constexpr int RB = 64;
  static constexpr int P = N + 4;
  static constexpr int kSmem = RB * P * 4;
};
template <int N, int MODE, typename Row>
__device__ __forceinline__ void pair_row_unit(const Row& row, float* smem) {
  using Geo = PairRowGeo<N>;
  constexpr int P = Geo::P, Q = N / 4;
#pragma unroll 8
  for (int i = threadIdx.x; i < Geo::RB * Q; i += 32) cp_async16(smem + i / Q * P + i % Q * 4, row(i / Q) + i % Q * 4);
  cp_async_wait_all();
  __syncwarp();
  const int r = (threadIdx.x / 8) * 16 + threadIdx.x % 8;
  pair_rows<N, MODE>(smem + r * P, smem + (r + 8) * P);
  __syncwarp();
#pragma unroll 8
  for (int i = threadIdx.x; i < Geo::RB * Q; i += 32)
    *reinterpret_cast<float4*>(row(i / Q) + i % Q * 4) = *reinterpret_cast<const float4*>(smem + i / Q * P + i % Q * 4);
}
template <int N, int H, int MODE>
__global__ void __launch_bounds__(32) k_pair_rows(SplitArgs a) {
  extern __shared__ float smem[];
  griddep_wait();
  griddep_trigger();
  const long long first = (long long)blockIdx.x * PairRowGeo<N>::RB;
  pair_row_unit<N, MODE>(
      [&](int r) -> float* { return H == 0 ? a.y + (first + r) * N : a.y + layout_row<cmax(H, 1)>(a.ly, first + r); },
      smem);
}

// ---- whole arrays in one tile ------------------------------------------------------------------
// ARR arrays of H x W in shared memory, row pitch W + 4 and arrays AP floats apart (8- and 16-column
// arrays are padded so that the 4 or 2 arrays which a half-warp's 16 column pairs span lie in different
// banks).  Columns: adjacent columns make a pair (64-bit accesses, a half-warp reads 128 contiguous
// bytes); a split line's exchange slots are the rows of its own columns.  Rows: rows r and r + 8 of 16
// make a pair.
template <int H, int W, int ARR> struct PairTileGeo {
  static constexpr int kRowPairs = ARR * H % 16 == 0 ? 8 : 4;   // split rows: pairs of a group
  static constexpr int P = W >= 128 ? W + 32 / kRowPairs : W + 4;
  static constexpr int AP = W == 8 ? H * P + (40 - H * P % 32) % 32 : W == 16 ? H * P + (48 - H * P % 32) % 32 : H * P;
  static constexpr int TR = ARR * H;
  static constexpr int kTile = ARR * AP;
  static constexpr int kTabC = H >= 128 ? SplitTab<cmax(H, 128)>::kFloats : 0;
  static constexpr int kTabR = W >= 128 && W != H ? SplitTab<cmax(W, 128)>::kFloats : 0;
  static constexpr int kSmem = (kTile + kTabC + kTabR) * 4;
};

// SINGLE: a thread runs one line of a short axis at a time instead of two, for batches that leave most of
// the GPU's issue slots idle (tile_cfg_few).
template <int H, int W, int ARR, int MODE, int T, int MINB, bool GEN, bool SINGLE>
__global__ void __launch_bounds__(T, MINB) k_pair_tile(TileArgs a) {
  using Geo = PairTileGeo<H, W, ARR>;
  constexpr int P = Geo::P, AP = Geo::AP, TR = Geo::TR;
  extern __shared__ float smem[];
  float* tcol = smem + Geo::kTile;
  float* trow = H == W ? tcol : tcol + Geo::kTabC;
  if constexpr (H >= 128) split_stage_tables<H, T>(a.tab.col, tcol);
  if constexpr (W >= 128 && W != H) split_stage_tables<W, T>(a.tab.row, trow);
  griddep_wait();
  griddep_trigger();
  const long long first = (long long)blockIdx.x * TR;
  const int rows = a.rows_total - first < TR ? (int)(a.rows_total - first) : TR;
  auto srow = [](int r) { return (r / H) * AP + (r % H) * P; };
  constexpr int Q = W / 4;
  // rows beyond the batch stay as they are: lines do not mix, and they are not stored
#pragma unroll 8
  for (int i = threadIdx.x; i < rows * Q; i += T) {
    const int r = i / Q, c = (i % Q) * 4;
    cp_async16(smem + srow(r) + c, GEN ? a.x + layout_row<H>(a.lx, first + r) + c : a.x + first * W + 4 * i);
  }
  cp_async_wait_all();
  __syncthreads();
  if constexpr (H >= 128) {
    constexpr int LP = cmin(16, ARR * W / 2), G = ARR * W / (2 * LP);   // groups of LP column pairs
    static_assert(G * 2 * LP == ARR * W, "whole groups");
    const int p = threadIdx.x % LP;
    auto base = [&](int g) {
      const int c = (g * LP + p) * 2;
      return smem + c / W * AP + c % W;
    };
    split_lines<H, MODE, T, G, LP, true>(
        [&](int g, int i) {
          const float2 v = *reinterpret_cast<const float2*>(base(g) + i * P);
          return f2_make(v.x, v.y);
        },
        [&](int g, int i, F2 v) { *reinterpret_cast<F2*>(base(g) + i * P) = v; }, base, P, tcol);
  } else if constexpr (SINGLE) {
    for (int l = threadIdx.x; l < ARR * W; l += T) {
      float* c = smem + (l / W) * AP + l % W;
      F1 v[H];
#pragma unroll
      for (int i = 0; i < H; ++i) v[i].v = c[i * P];
      pair_line<H, MODE>(v);
#pragma unroll
      for (int i = 0; i < H; ++i) c[i * P] = v[i].v;
    }
  } else {
    for (int l = threadIdx.x; l < ARR * W / 2; l += T) {
      float* c = smem + (l / (W / 2)) * AP + 2 * (l % (W / 2));
      F2 v[H];
#pragma unroll
      for (int i = 0; i < H; ++i) v[i] = *reinterpret_cast<const F2*>(c + i * P);
      pair_line<H, MODE>(v);
#pragma unroll
      for (int i = 0; i < H; ++i) *reinterpret_cast<F2*>(c + i * P) = v[i];
    }
  }
  __syncthreads();
  if constexpr (W >= 128) {
    split_rows<W, MODE, T, TR / (2 * Geo::kRowPairs), Geo::kRowPairs>(smem, trow);
  } else if constexpr (SINGLE) {
    for (int l = threadIdx.x; l < TR; l += T) single_row<W, MODE>(smem + srow(l));
  } else {
    for (int l = threadIdx.x; l < TR / 2; l += T) {
      const int r = (l / 8) * 16 + l % 8;
      pair_rows<W, MODE>(smem + srow(r), smem + srow(r + 8));
    }
  }
  if constexpr (W >= 128) {
    fence_async();
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += T)
      bulk_store(GEN ? a.y + layout_row<H>(a.ly, first + r) : a.y + (first + r) * W, smem + srow(r), W * 4);
    bulk_commit_wait();
  } else {
    __syncthreads();
#pragma unroll 8
    for (int i = threadIdx.x; i < rows * Q; i += T) {
      const int r = i / Q, c = (i % Q) * 4;
      *reinterpret_cast<float4*>(GEN ? a.y + layout_row<H>(a.ly, first + r) + c : a.y + first * W + 4 * i) =
          *reinterpret_cast<const float4*>(smem + srow(r) + c);
    }
  }
}

}  // namespace bridct
