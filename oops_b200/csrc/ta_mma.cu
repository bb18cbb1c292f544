// Triangle attention of 16-bit operands at head sizes and layouts the tcgen05 kernels do not take (head size up to 64
// other than 32 in f16, under a mask or in calls of few columns, strides or addresses that are no multiples of 16 bytes, an f32
// bias): register-level matrix products (mma.sync m16n8k16, f32 accumulation), operands staged by cp.async.  Definition as in the reference's kernels
// (oops/attention/triangle/triton/kernel.py:128-147, :250-261, :499-564, :682-714, :856).
//
// Calls of this kind are small -- token attention, odd head sizes -- and bound by latency and by the element-wise work
// on the scores, not by the tensor pipe; fragments go from product to softmax to product in registers, which needs no
// tensor-memory round trips, no 16-byte rules and no padding of the head size beyond 16.
// The path it takes over kept probabilities and dS in f32; here they enter their products as a pair of 16-bit numbers (value
// and remainder: 16 digits in bf16, 22 in f16), well below the rounding of the results.  f16 lacks the exponents of f32:
// its probabilities are raised by 2^14 and its rows of dS scaled by a running power of two (RowScale).
//
//   forward   CTA = (batch, row, head, 64 queries), four warps of 16 queries, 64-key steps, online softmax.
//   reverse   one launch, three kinds of CTA: dQ of 64 queries; dK and dV of 64 keys (scores transposed, a warp owns 16
//             keys); a 64 x 64 tile of the row-shared bias gradient, rows innermost, summed in registers.  Each makes the
//             scores it needs again (9 products instead of 5): token attention has too few rows and heads to give a
//             CTA a whole row, and nothing has to be added across CTAs, so results are reproducible.
// 4 samples, 16 heads of 64 channels, 512 tokens, f16: 35 us forward and 144 us reverse (bf16 with a mask 37 and 143; without one it goes to the
// tcgen05 kernels), against 1178 us in 9 launches with scores in memory.  Bound by latency at twelve to sixteen warps per SM, element-wise work and
// products in turn (counters of the bf16 call while it came here: issue slots 50 % and the tensor pipe 38 % busy forward, 36 and 33 %
// in the reverse, HBM idle): packed f32 arithmetic, no tests on kept keys where a tile keeps all, first products without a zeroed accumulator,
// and, in the reverse, row operands read again from shared memory instead of held in 64 registers (238 -> 168 registers, two -> three
// CTAs per SM) took 45 and 171 us to 35 and 136 in bf16.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "ta_internal.h"

namespace oops_ta {
namespace {

constexpr int kT = 64;          // rows and columns of a tile
constexpr int kThreads = 128;   // four warps of 16 tile rows
constexpr float kLog2e = 1.4426950408889634f;

struct MmaProblem {
  oops_ta_pair q, k, v, out, dout, dq, dk, dv;
  const uint8_t* mask;
  int64_t m_sb, m_sr, m_sc;
  const void* bias;
  int64_t b_sb, b_sg, b_sh, b_sq, b_sk;
  int batch, rows, cols, heads, dim, bias_groups;
  float scale;
  int vec, bias_vec;  // 16-byte words throughout the pair tensors / the bias rows
  float* lse;
  float* delta;
  void* dbias;        // shared gradient (one part), or the per-row gradient
  float* parts;       // [parts][batch][heads][cols][cols] (several parts)
  int64_t db_sb, db_sg, db_sh, db_sq, db_sk;
  int dbias_f32, num_parts, rows_per_part;
  int dq_ctas, dkv_ctas;
};

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_at(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// kWide: the type has the exponents of f32.  kUp: exponent that probabilities are raised by before they are split (f16 ends at
// 2^-24, which would cut those below 2^-10 of the largest short of 16 digits; 2^14 leaves room below 65504 for rounding).
template <typename T>
struct Pair16;
template <>
struct Pair16<__nv_bfloat16> {
  static constexpr bool kWide = true;
  static constexpr float kUp = 0.f;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 widen(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ void mma_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {  // c = a b
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  }
};
template <>
struct Pair16<__half> {
  static constexpr bool kWide = false;
  static constexpr float kUp = 14.f;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 widen(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ void mma_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {  // c = a b
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  }
};

// Rows of a tile are 16 bytes more than the padded head size: an odd number of 16-byte words, so that the eight rows of
// an 8 x 8 matrix lie in different banks.
template <int DP>
constexpr int pitch() { return DP + 8; }
template <int DP>
constexpr int tile_elems() { return kT * pitch<DP>(); }
template <bool B32>
constexpr int bias_pitch() { return B32 ? kT + 4 : kT + 8; }  // elements of the bias type

template <typename T>
__device__ __forceinline__ T* row_of(const oops_ta_pair& t, int b, int r, int h, int64_t c) {
  return reinterpret_cast<T*>(t.ptr) + b * t.sb + int64_t(r) * t.sr + int64_t(h) * t.sh + c * t.sc;
}

// dst[i][0 .. DP) = columns first .. first + 63 of one head of one pair row; zeros outside the axis and the head, and for
// columns that `keep` drops (their rows may hold anything).
template <typename T, int DP>
__device__ __forceinline__ void load_tile(T* dst, const oops_ta_pair& t, const MmaProblem& p, int b, int r, int h, int first,
                                          const uint8_t* keep) {
  const T* head = row_of<T>(t, b, r, h, 0);
#pragma unroll
  for (int i = threadIdx.x; i < kT * (DP / 8); i += kThreads) {
    const int row = i / (DP / 8), c = (i % (DP / 8)) * 8, col = first + row;
    const bool take = col < p.cols && (!keep || keep[int64_t(col) * p.m_sc] != 0);
    const T* src = head + int64_t(col) * t.sc + c;
    T* to = dst + row * pitch<DP>() + c;
    if (p.vec) {
      const bool on = take && c < p.dim;
      copy16(to, on ? src : head, on ? 16 : 0);
    } else {
      uint16_t word[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) word[e] = take && c + e < p.dim ? reinterpret_cast<const uint16_t*>(src)[e] : uint16_t(0);
      *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(word);
    }
  }
}

template <typename B, int PITCH>
__device__ __forceinline__ void load_bias(B* dst, const B* plane, const MmaProblem& p, int q0, int k0) {
  constexpr int kWord = 16 / int(sizeof(B));
  if (p.bias_vec) {
#pragma unroll
    for (int i = threadIdx.x; i < kT * kT / kWord; i += kThreads) {
      const int row = i / (kT / kWord), c = (i % (kT / kWord)) * kWord;
      const int width = q0 + row < p.cols ? min(kWord, p.cols - k0 - c) : 0;
      copy16(dst + row * PITCH + c, width > 0 ? plane + int64_t(q0 + row) * p.b_sq + k0 + c : plane, width > 0 ? width * int(sizeof(B)) : 0);
    }
  } else {
#pragma unroll 4
    for (int i = threadIdx.x; i < kT * kT; i += kThreads) {
      const int q = q0 + i / kT, k = k0 + i % kT;
      B v = B(0.f);
      if (q < p.cols && k < p.cols) v = plane[int64_t(q) * p.b_sq + int64_t(k) * p.b_sk];
      dst[(i / kT) * PITCH + i % kT] = v;
    }
  }
}

// Bit i: column first + i exists and is kept.  Every warp works it out for itself.
__device__ __forceinline__ uint64_t keep_bits(const MmaProblem& p, const uint8_t* keep, int first) {
  const int lane = threadIdx.x & 31;
  uint32_t half[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int col = first + 32 * i + lane;
    half[i] = __ballot_sync(0xffffffffu, col < p.cols && (!keep || keep[int64_t(col) * p.m_sc] != 0));
  }
  return uint64_t(half[1]) << 32 | half[0];
}

// A operands of the warp's 16 tile rows, all channels.
template <typename T, int DP>
__device__ __forceinline__ void load_rows(uint32_t (&a)[DP / 16][4], const T* tile, int row0) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kc = 0; kc < DP / 16; ++kc) ldmatrix4(a[kc], tile + (row0 + (lane & 15)) * pitch<DP>() + kc * 16 + (lane >> 4) * 8);
}

template <typename T, int NT>
__device__ __forceinline__ void score_step(float (&s)[NT][4], const uint32_t (&a)[4], const T* columns, int pitch, bool first) {
#pragma unroll
  for (int np = 0; np < NT / 2; ++np) {
    uint32_t b[4];
    ldmatrix4(b, columns + np * 16 * pitch);
    if (first) {
      Pair16<T>::mma_first(s[2 * np], a, b[0], b[1]);
      Pair16<T>::mma_first(s[2 * np + 1], a, b[2], b[3]);
    } else {
      Pair16<T>::mma(s[2 * np], a, b[0], b[1]);
      Pair16<T>::mma(s[2 * np + 1], a, b[2], b[3]);
    }
  }
}

// s[nt] = rows x (columns col0 + 8 nt ...)^T over the channels: NT tiles of 8 columns.
template <typename T, int DP, int NT>
__device__ __forceinline__ void scores(float (&s)[NT][4], const uint32_t (&a)[DP / 16][4], const T* tile, int col0) {
  const int lane = threadIdx.x & 31;
  const T* columns = tile + (col0 + (lane & 7) + (lane >> 4) * 8) * pitch<DP>() + ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int kc = 0; kc < DP / 16; ++kc) score_step<T, NT>(s, a[kc], columns + kc * 16, pitch<DP>(), kc == 0);
}

// The same with the rows fetched from their tile (row0 ...) as they are needed: registers for shared-memory reads.
template <typename T, int DP, int NT>
__device__ __forceinline__ void scores(float (&s)[NT][4], const T* rows, int row0, const T* tile, int col0) {
  const int lane = threadIdx.x & 31;
  const T* columns = tile + (col0 + (lane & 7) + (lane >> 4) * 8) * pitch<DP>() + ((lane >> 3) & 1) * 8;
  const T* row = rows + (row0 + (lane & 15)) * pitch<DP>() + (lane >> 4) * 8;
#pragma unroll
  for (int kc = 0; kc < DP / 16; ++kc) {
    uint32_t a[4];
    ldmatrix4(a, row + kc * 16);
    score_step<T, NT>(s, a, columns + kc * 16, pitch<DP>(), kc == 0);
  }
}

// acc += w (16 rows x 8 NT columns, f32, as a 16-bit value and its remainder) x tile rows col0 ... (channels as columns)
template <typename T, int DP, int NT>
__device__ __forceinline__ void accumulate(float (&acc)[DP / 8][4], const float (&w)[NT][4], const T* tile, int col0) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kc = 0; kc < NT / 2; ++kc) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x = w[2 * kc + (i >> 1)][(i & 1) * 2], y = w[2 * kc + (i >> 1)][(i & 1) * 2 + 1];
      hi[i] = Pair16<T>::pack(x, y);
      const float2 rest = __ffma2_rn(Pair16<T>::widen(hi[i]), make_float2(-1.f, -1.f), make_float2(x, y));
      lo[i] = Pair16<T>::pack(rest.x, rest.y);
    }
#pragma unroll
    for (int np = 0; np < DP / 16; ++np) {
      uint32_t b[4];
      ldmatrix4_trans(b, tile + (col0 + kc * 16 + (lane & 15)) * pitch<DP>() + np * 16 + (lane >> 4) * 8);
      Pair16<T>::mma(acc[2 * np], hi, b[0], b[1]);
      Pair16<T>::mma(acc[2 * np], lo, b[0], b[1]);
      Pair16<T>::mma(acc[2 * np + 1], hi, b[2], b[3]);
      Pair16<T>::mma(acc[2 * np + 1], lo, b[2], b[3]);
    }
  }
}

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 pair_of(const float (&s)[4], int half) { return make_float2(s[2 * half], s[2 * half + 1]); }
__device__ __forceinline__ void set_pair(float (&s)[4], int half, float2 v) {
  s[2 * half] = v.x;
  s[2 * half + 1] = v.y;
}
// exp(x) 2^kUp
template <typename T>
__device__ __forceinline__ float2 ex2_above(float2 x) {
  x = Pair16<T>::kWide ? __fmul2_rn(x, both(kLog2e)) : __ffma2_rn(x, both(kLog2e), both(Pair16<T>::kUp));
  return make_float2(ex2(x.x), ex2(x.y));
}
// exp(score * scale + bias - lse) 2^kUp, `norm` = -lse.  The logit is made as the forward pass makes it and the norm comes off before
// the change of base: with log2(e) multiplied into either of them, a row whose logits are all far from zero (a bias of -1e9,
// or the lowest value of the type) would see the two round apart, or overflow, instead of cancelling.
template <typename T>
__device__ __forceinline__ float2 probability(float2 score, float scale, float2 bias, float2 norm) {
  return ex2_above<T>(__fadd2_rn(__ffma2_rn(score, both(scale), bias), norm));
}

// Power of two that a row of dS is multiplied by before its split into 16-bit numbers, and its accumulator with it.  f16 has
// neither the exponents that dS reaches under a scaled loss (infinite above 65504) nor those of small gradients (nothing
// below 2^-25), both of which K or Q can bring back into its range.  The scale starts high and only falls: a step whose largest
// value would pass 2^15 brings that value to 2^14, and the accumulator along.  What is small against an earlier step loses no
// more than an f32 sum would: its digits end 2^-38 below that step's largest value.  (bf16 needs none of this.)
template <typename T>
struct RowScale {
  int up[2] = {110, 110};  // exponents, of rows g and g + 8

  template <int DP, int NT>
  __device__ __forceinline__ void apply(float (&w)[NT][4], float (&acc)[DP / 8][4]) {
    if constexpr (!Pair16<T>::kWide) {
      float peak[2] = {0.f, 0.f};
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) peak[i >> 1] = fmaxf(peak[i >> 1], fabsf(w[nt][i]));
      float factor[2] = {power(up[0]), power(up[1])};
      if (__any_sync(0xffffffffu, fmaxf(peak[0] * factor[0], peak[1] * factor[1]) > 32768.f)) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          peak[half] = fmaxf(peak[half], __shfl_xor_sync(0xffffffffu, peak[half], 1));
          peak[half] = fmaxf(peak[half], __shfl_xor_sync(0xffffffffu, peak[half], 2));
          // exponent of the largest value to 14
          const int wanted = min(up[half], 14 - (int(__float_as_uint(peak[half]) >> 23) - 127));
          const float shrink = ex2(float(wanted - up[half]));
          up[half] = wanted;
          factor[half] = power(wanted);
#pragma unroll
          for (int i = 0; i < DP / 8; ++i) set_pair(acc[i], half, __fmul2_rn(pair_of(acc[i], half), both(shrink)));
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) set_pair(w[nt], half, __fmul2_rn(pair_of(w[nt], half), both(factor[half])));
    }
  }
  // What the accumulator's rows are to be multiplied by.
  __device__ __forceinline__ float undo(int half) const { return Pair16<T>::kWide ? 1.f : power(-up[half]); }
  static __device__ __forceinline__ float power(int exponent) { return __uint_as_float(uint32_t(exponent + 127) << 23); }
};
// Columns 8 nt + 2 t, + 1 of an accumulator become `value` where their bit is not set.
template <int NT>
__device__ __forceinline__ void drop_columns(float (&s)[NT][4], uint64_t bits, int t, float value) {
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const uint32_t kept = uint32_t(bits >> (nt * 8 + 2 * t));
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (((kept >> (i & 1)) & 1) == 0) s[nt][i] = value;
  }
}

// Two neighbouring bias values of a tile row.
template <typename T, bool B32>
__device__ __forceinline__ float2 bias_pair(const void* tile, int row, int col) {
  if constexpr (B32) {
    return *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(tile) + row * bias_pitch<true>() + col);
  } else {
    return Pair16<T>::widen(*reinterpret_cast<const uint32_t*>(reinterpret_cast<const T*>(tile) + row * bias_pitch<false>() + col));
  }
}

template <typename T>
__device__ __forceinline__ void store_pair(T* row, int c, const MmaProblem& p, float x, float y, bool whole) {
  if (whole) {
    *reinterpret_cast<uint32_t*>(row + c) = Pair16<T>::pack(x, y);
  } else {
    if (c < p.dim) row[c] = T(x);
    if (c + 1 < p.dim) row[c + 1] = T(y);
  }
}

// Rows `row0 + lane / 4` and eight further of an accumulator, times f0 and f1.
template <typename T, int DP>
__device__ __forceinline__ void store_rows(const oops_ta_pair& to, const MmaProblem& p, int b, int r, int h, int col, const float (&acc)[DP / 8][4],
                                           float f0, float f1) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int at = col + (lane >> 2) + 8 * half;
    if (at >= p.cols) continue;
    T* row = row_of<T>(to, b, r, h, at);
    const float f = half ? f1 : f0;
#pragma unroll
    for (int nt = 0; nt < DP / 8; ++nt) {
      const int c = nt * 8 + (lane & 3) * 2;
      if (c < p.dim) store_pair(row, c, p, acc[nt][2 * half] * f, acc[nt][2 * half + 1] * f, p.vec != 0);
    }
  }
}

template <typename T, bool B32>
using BiasType = typename std::conditional<B32, float, T>::type;

template <typename T, bool B32>
__device__ __forceinline__ const BiasType<T, B32>* bias_plane(const MmaProblem& p, int b, int r, int h) {
  if (!p.bias) return nullptr;
  return reinterpret_cast<const BiasType<T, B32>*>(p.bias) + b * p.b_sb + int64_t(p.bias_groups == 1 ? 0 : r) * p.b_sg + h * p.b_sh;
}

template <bool B32>
constexpr int bias_bytes() { return kT * bias_pitch<B32>() * (B32 ? 4 : 2); }

// Q passes through the second stage's memory into registers: four CTAs then fit an SM, 592 at once, where three left the
// 512 CTAs of a 4-sample, 16-head, 512-token call a second wave of 68.
template <typename T, int DP, bool B32>
__global__ void __launch_bounds__(kThreads, 4) mma_forward_kernel(const MmaProblem p) {
  extern __shared__ __align__(16) uint8_t mma_smem[];
  constexpr int kStage = 2 * tile_elems<DP>() * 2 + bias_bytes<B32>();  // K | V | bias
  uint8_t* stages = mma_smem;
  T* Q = reinterpret_cast<T*>(stages + kStage);
  int idx = blockIdx.x;
  const int tiles = (p.cols + kT - 1) / kT, qt = idx % tiles;
  idx /= tiles;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int r = idx % p.rows, b = idx / p.rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;
  const auto* plane = bias_plane<T, B32>(p, b, r, h);

  auto request = [&](int kt) {
    uint8_t* at = stages + (kt & 1) * kStage;
    load_tile<T, DP>(reinterpret_cast<T*>(at), p.k, p, b, r, h, kt * kT, keep);
    load_tile<T, DP>(reinterpret_cast<T*>(at) + tile_elems<DP>(), p.v, p, b, r, h, kt * kT, keep);
    if (plane)
      load_bias<BiasType<T, B32>, bias_pitch<B32>()>(reinterpret_cast<BiasType<T, B32>*>(at + 2 * tile_elems<DP>() * 2), plane, p, qt * kT, kt * kT);
  };
  load_tile<T, DP>(Q, p.q, p, b, r, h, qt * kT, nullptr);
  copies_commit();
  request(0);
  copies_commit();
  uint32_t q[DP / 16][4];
  float o[DP / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  copies_wait<1>();
  __syncthreads();
  load_rows<T, DP>(q, Q, warp * 16);
  __syncthreads();

  for (int kt = 0; kt < tiles; ++kt) {
    if (kt + 1 < tiles) request(kt + 1);
    copies_commit();
    copies_wait<1>();
    __syncthreads();
    const uint64_t bits = keep_bits(p, keep, kt * kT);
    const uint8_t* at = stages + (kt & 1) * kStage;
    if (bits) {  // the same for every warp
      const T* K = reinterpret_cast<const T*>(at);
      const void* bias = at + 2 * tile_elems<DP>() * 2;
      float s[8][4];
      scores<T, DP, 8>(s, q, K, 0);
      // logits, then the online softmax of rows g and g + 8 (a quad of lanes holds a row)
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float2 add = both(0.f);
          if (plane) add = bias_pair<T, B32>(bias, warp * 16 + g + 8 * half, nt * 8 + 2 * t);
          set_pair(s[nt], half, __ffma2_rn(pair_of(s[nt], half), both(p.scale), add));
        }
      if (bits != ~0ull) drop_columns(s, bits, t, -INFINITY);
      float peak[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) peak[i >> 1] = fmaxf(peak[i >> 1], s[nt][i]);
      float shrink[2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        peak[half] = fmaxf(peak[half], __shfl_xor_sync(0xffffffffu, peak[half], 1));
        peak[half] = fmaxf(peak[half], __shfl_xor_sync(0xffffffffu, peak[half], 2));
        const float before = m[half];
        m[half] = fmaxf(before, peak[half]);
        const float base = m[half] == -INFINITY ? 0.f : m[half];
        shrink[half] = ex2((before - base) * kLog2e);
        peak[half] = base;
        l[half] *= shrink[half];
      }
      float2 sum[2] = {both(0.f), both(0.f)};
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const float2 e = ex2_above<T>(__fadd2_rn(pair_of(s[nt], half), both(-peak[half])));
          set_pair(s[nt], half, e);
          sum[half] = __fadd2_rn(sum[half], e);
        }
#pragma unroll
      for (int half = 0; half < 2; ++half) l[half] += sum[half].x + sum[half].y;
#pragma unroll
      for (int i = 0; i < DP / 8; ++i) {
        o[i][0] *= shrink[0];
        o[i][1] *= shrink[0];
        o[i][2] *= shrink[1];
        o[i][3] *= shrink[1];
      }
      accumulate<T, DP, 8>(o, s, K + tile_elems<DP>(), 0);
    }
    __syncthreads();  // the stage may be overwritten
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    l[half] += __shfl_xor_sync(0xffffffffu, l[half], 1);
    l[half] += __shfl_xor_sync(0xffffffffu, l[half], 2);
    const int at = qt * kT + warp * 16 + g + 8 * half;
    const bool some = l[half] > 0.f || l[half] != l[half];
    if (p.lse && t == 0 && at < p.cols)
      p.lse[((int64_t(b) * p.rows + r) * p.heads + h) * p.cols + at] = some ? m[half] + (__log2f(l[half]) - Pair16<T>::kUp) * 0.6931471805599453f : 0.f;
    l[half] = some ? 1.f / l[half] : 0.f;
  }
  store_rows<T, DP>(p.out, p, b, r, h, qt * kT + warp * 16, o, l[0], l[1]);
}

// delta[q] = sum_d out * dout, eight lanes per (row, head, query).
template <typename T>
__global__ void __launch_bounds__(256) mma_delta_kernel(const MmaProblem p, int64_t total) {
  const int64_t i = (int64_t(blockIdx.x) * 256 + threadIdx.x) >> 3;
  const int part = threadIdx.x & 7;
  float sum = 0.f;
  if (i < total) {
    const int64_t q = i % p.cols, z = i / p.cols;
    const int h = int(z % p.heads), r = int(z / p.heads % p.rows), b = int(z / p.heads / p.rows);
    const T* o = row_of<T>(p.out, b, r, h, q);
    const T* d = row_of<T>(p.dout, b, r, h, q);
    if (p.vec) {
      const int c = part * 8;
      if (c < p.dim) {
        const uint4 x = *reinterpret_cast<const uint4*>(o + c), y = *reinterpret_cast<const uint4*>(d + c);
        const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 a = Pair16<T>::widen(xw[e]), g = Pair16<T>::widen(yw[e]);
          sum += a.x * g.x + a.y * g.y;
        }
      }
    } else {
      for (int c = part; c < p.dim; c += 8) sum += float(o[c]) * float(d[c]);
    }
  }
#pragma unroll
  for (int x = 4; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
  if (i < total && part == 0) p.delta[i] = sum;
}

// dQ of 64 queries: S = Q K^T, dP = dO V^T, dQ += dS K; the per-row bias gradient is dS itself.
template <typename T, int DP, bool B32>
__device__ __forceinline__ void query_gradient(const MmaProblem& p, uint8_t* smem, int idx) {
  constexpr float kDown = Pair16<T>::kWide ? 1.f : 1.f / 16384.f;  // takes 2^kUp back
  constexpr int kStage = 2 * tile_elems<DP>() * 2 + bias_bytes<B32>();
  T* Q = reinterpret_cast<T*>(smem);
  uint8_t* stages = smem + 2 * tile_elems<DP>() * 2;
  const int tiles = (p.cols + kT - 1) / kT, qt = idx % tiles;
  idx /= tiles;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int r = idx % p.rows, b = idx / p.rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;
  const auto* plane = bias_plane<T, B32>(p, b, r, h);
  auto request = [&](int kt) {
    uint8_t* at = stages + (kt & 1) * kStage;
    load_tile<T, DP>(reinterpret_cast<T*>(at), p.k, p, b, r, h, kt * kT, keep);
    load_tile<T, DP>(reinterpret_cast<T*>(at) + tile_elems<DP>(), p.v, p, b, r, h, kt * kT, keep);
    if (plane)
      load_bias<BiasType<T, B32>, bias_pitch<B32>()>(reinterpret_cast<BiasType<T, B32>*>(at + 2 * tile_elems<DP>() * 2), plane, p, qt * kT, kt * kT);
  };
  load_tile<T, DP>(Q, p.q, p, b, r, h, qt * kT, nullptr);
  load_tile<T, DP>(Q + tile_elems<DP>(), p.dout, p, b, r, h, qt * kT, nullptr);
  request(0);
  copies_commit();
  float norm[2], delta[2];
  const int row0 = qt * kT + warp * 16 + g;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int at = row0 + 8 * half;
    const int64_t stat = ((int64_t(b) * p.rows + r) * p.heads + h) * p.cols + at;
    norm[half] = at < p.cols ? -p.lse[stat] : -INFINITY;
    delta[half] = at < p.cols ? p.delta[stat] : 0.f;
  }
  float dq[DP / 8][4];
#pragma unroll
  for (int i = 0; i < DP / 8; ++i) dq[i][0] = dq[i][1] = dq[i][2] = dq[i][3] = 0.f;
  RowScale<T> rows;
  for (int kt = 0; kt < tiles; ++kt) {
    if (kt + 1 < tiles) request(kt + 1);
    copies_commit();
    copies_wait<1>();
    __syncthreads();
    const uint64_t all = keep_bits(p, keep, kt * kT);
    const uint8_t* at = stages + (kt & 1) * kStage;
    const T* K = reinterpret_cast<const T*>(at);
    const void* bias = at + 2 * tile_elems<DP>() * 2;
#pragma unroll 1
    for (int col0 = 0; col0 < kT; col0 += 32) {  // 32 keys at a time keep the registers of three CTAs per SM
      const uint32_t bits = uint32_t(all >> col0);
      float s[4][4], dp[4][4];
      scores<T, DP, 4>(s, Q, warp * 16, K, col0);
      scores<T, DP, 4>(dp, Q + tile_elems<DP>(), warp * 16, K + tile_elems<DP>(), col0);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float2 add = both(0.f);
          if (plane) add = bias_pair<T, B32>(bias, warp * 16 + g + 8 * half, col0 + nt * 8 + 2 * t);
          const float2 e = probability<T>(pair_of(s[nt], half), p.scale, add, both(norm[half]));
          set_pair(s[nt], half, __fmul2_rn(e, __fadd2_rn(pair_of(dp[nt], half), both(-delta[half]))));
        }
      if (bits != 0xffffffffu) drop_columns(s, bits, t, 0.f);
      if (p.dbias && p.bias_groups > 1) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int query = row0 + 8 * (i >> 1), key = kt * kT + col0 + nt * 8 + 2 * t + (i & 1);
            if (query < p.cols && key < p.cols)
              reinterpret_cast<BiasType<T, B32>*>(p.dbias)[b * p.db_sb + int64_t(r) * p.db_sg + h * p.db_sh + int64_t(query) * p.db_sq +
                                                          int64_t(key) * p.db_sk] = BiasType<T, B32>(s[nt][i] * kDown);
          }
      }
      if (p.dq.ptr) {
        rows.template apply<DP, 4>(s, dq);
        accumulate<T, DP, 4>(dq, s, K, col0);
      }
    }
    __syncthreads();
  }
  if (p.dq.ptr)
    store_rows<T, DP>(p.dq, p, b, r, h, qt * kT + warp * 16, dq, rows.undo(0) * (p.scale * kDown), rows.undo(1) * (p.scale * kDown));
}

// dK and dV of 64 keys: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q.
template <typename T, int DP, bool B32>
__device__ __forceinline__ void key_gradient(const MmaProblem& p, uint8_t* smem, int idx) {
  constexpr float kDown = Pair16<T>::kWide ? 1.f : 1.f / 16384.f;  // takes 2^kUp back
  constexpr int kStage = 2 * tile_elems<DP>() * 2 + bias_bytes<B32>() + 2 * kT * 4;  // Q | dO | bias | -lse | delta
  T* K = reinterpret_cast<T*>(smem);
  uint8_t* stages = smem + 2 * tile_elems<DP>() * 2;
  const int tiles = (p.cols + kT - 1) / kT, kt = idx % tiles;
  idx /= tiles;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int r = idx % p.rows, b = idx / p.rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;
  const auto* plane = bias_plane<T, B32>(p, b, r, h);
  const int64_t stat0 = ((int64_t(b) * p.rows + r) * p.heads + h) * p.cols;
  auto request = [&](int qt) {
    uint8_t* at = stages + (qt & 1) * kStage;
    load_tile<T, DP>(reinterpret_cast<T*>(at), p.q, p, b, r, h, qt * kT, nullptr);
    load_tile<T, DP>(reinterpret_cast<T*>(at) + tile_elems<DP>(), p.dout, p, b, r, h, qt * kT, nullptr);
    at += 2 * tile_elems<DP>() * 2;
    if (plane)
      load_bias<BiasType<T, B32>, bias_pitch<B32>()>(reinterpret_cast<BiasType<T, B32>*>(at), plane, p, qt * kT, kt * kT);
    float* stats = reinterpret_cast<float*>(at + bias_bytes<B32>());
    const int q = qt * kT + (threadIdx.x & 63);
    if (threadIdx.x < kT) stats[threadIdx.x] = q < p.cols ? -p.lse[stat0 + q] : -INFINITY;
    else stats[threadIdx.x] = q < p.cols ? p.delta[stat0 + q] : 0.f;
  };
  load_tile<T, DP>(K, p.k, p, b, r, h, kt * kT, keep);
  load_tile<T, DP>(K + tile_elems<DP>(), p.v, p, b, r, h, kt * kT, keep);
  request(0);
  copies_commit();
  const uint64_t all = keep_bits(p, keep, kt * kT), bits = all >> (warp * 16 + g);
  const bool all_kept = all == ~0ull;
  const bool kept[2] = {(bits & 1) != 0, ((bits >> 8) & 1) != 0};
  float dk[DP / 8][4], dv[DP / 8][4];
#pragma unroll
  for (int i = 0; i < DP / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) dk[i][e] = dv[i][e] = 0.f;
  RowScale<T> rows;
  for (int qt = 0; qt < tiles; ++qt) {
    if (qt + 1 < tiles) request(qt + 1);
    copies_commit();
    copies_wait<1>();
    __syncthreads();
    const uint8_t* at = stages + (qt & 1) * kStage;
    const T* Q = reinterpret_cast<const T*>(at);
    const uint8_t* bias = at + 2 * tile_elems<DP>() * 2;
    const float* stats = reinterpret_cast<const float*>(bias + bias_bytes<B32>());
#pragma unroll 1
    for (int col0 = 0; col0 < kT; col0 += 32) {
      float s[4][4], dp[4][4];
      scores<T, DP, 4>(s, K, warp * 16, Q, col0);
      scores<T, DP, 4>(dp, K + tile_elems<DP>(), warp * 16, Q + tile_elems<DP>(), col0);
      // the bias tile has queries as rows: its 8 x 8 blocks are read transposed
      float2 add[4][2];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) add[nt][0] = add[nt][1] = make_float2(0.f, 0.f);
      if (plane) {
        if constexpr (B32) {
          const float* tile = reinterpret_cast<const float*>(bias);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const float* from = tile + (col0 + nt * 8 + 2 * t) * bias_pitch<true>() + warp * 16 + g + 8 * half;
              add[nt][half] = make_float2(from[0], from[bias_pitch<true>()]);
            }
        } else {
          const T* tile = reinterpret_cast<const T*>(bias);
#pragma unroll
          for (int np = 0; np < 2; ++np) {
            uint32_t w[4];  // blocks (queries 16 np, keys 0), (0, 8), (8, 0), (8, 8)
            ldmatrix4_trans(w, tile + (col0 + np * 16 + (lane & 7) + (lane >> 4) * 8) * bias_pitch<false>() + warp * 16 + ((lane >> 3) & 1) * 8);
            add[2 * np][0] = Pair16<T>::widen(w[0]);
            add[2 * np][1] = Pair16<T>::widen(w[1]);
            add[2 * np + 1][0] = Pair16<T>::widen(w[2]);
            add[2 * np + 1][1] = Pair16<T>::widen(w[3]);
          }
        }
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const float2 norm = *reinterpret_cast<const float2*>(stats + col0 + nt * 8 + 2 * t);
        const float2 delta = *reinterpret_cast<const float2*>(stats + kT + col0 + nt * 8 + 2 * t);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const float2 e = probability<T>(pair_of(s[nt], half), p.scale, add[nt][half], norm);
          set_pair(s[nt], half, e);
          set_pair(dp[nt], half, __fmul2_rn(e, __fadd2_rn(pair_of(dp[nt], half), make_float2(-delta.x, -delta.y))));
        }
      }
      if (!all_kept) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (!kept[i >> 1]) s[nt][i] = dp[nt][i] = 0.f;
      }
      if (p.dv.ptr) accumulate<T, DP, 4>(dv, s, Q + tile_elems<DP>(), col0);
      if (p.dk.ptr) {
        rows.template apply<DP, 4>(dp, dk);
        accumulate<T, DP, 4>(dk, dp, Q, col0);
      }
    }
    __syncthreads();
  }
  // a dropped key gets exact zeros, whatever the upstream gradient holds
#pragma unroll
  for (int i = 0; i < DP / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (!kept[e >> 1]) dk[i][e] = dv[i][e] = 0.f;
  if (p.dk.ptr)
    store_rows<T, DP>(p.dk, p, b, r, h, kt * kT + warp * 16, dk, rows.undo(0) * (p.scale * kDown), rows.undo(1) * (p.scale * kDown));
  if (p.dv.ptr) store_rows<T, DP>(p.dv, p, b, r, h, kt * kT + warp * 16, dv, kDown, kDown);
}

// A 64 x 64 tile of the row-shared bias gradient: the sum of dS over the part's rows.
template <typename T, int DP, bool B32>
__device__ __forceinline__ void bias_gradient(const MmaProblem& p, uint8_t* smem, int idx) {
  constexpr float kDown = Pair16<T>::kWide ? 1.f : 1.f / 16384.f;
  constexpr int kStage = 4 * tile_elems<DP>() * 2;  // Q | dO | K | V of a row
  const int tiles = (p.cols + kT - 1) / kT, kt = idx % tiles;
  idx /= tiles;
  const int qt = idx % tiles;
  idx /= tiles;
  const int h = idx % p.heads;
  idx /= p.heads;
  const int b = idx % p.batch, part = idx / p.batch;
  const int first = part * p.rows_per_part, last = min(p.rows, first + p.rows_per_part);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  // the thread's bias values stay in registers: [8 columns][row g, row g + 8][two neighbours]
  using Bias = BiasType<T, B32>;
  const Bias* plane = bias_plane<T, B32>(p, b, 0, h);
  Bias add[8][2][2];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int query = qt * kT + warp * 16 + g + 8 * half, key = kt * kT + nt * 8 + 2 * t;
      const Bias* from = plane + int64_t(query) * p.b_sq + int64_t(key) * p.b_sk;
      add[nt][half][0] = query < p.cols && key < p.cols ? from[0] : Bias(0.f);
      add[nt][half][1] = query < p.cols && key + 1 < p.cols ? from[p.b_sk] : Bias(0.f);
    }
  auto request = [&](int r) {
    T* at = reinterpret_cast<T*>(smem + ((r - first) & 1) * kStage);
    const uint8_t* keep = p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr;
    load_tile<T, DP>(at, p.q, p, b, r, h, qt * kT, nullptr);
    load_tile<T, DP>(at + tile_elems<DP>(), p.dout, p, b, r, h, qt * kT, nullptr);
    load_tile<T, DP>(at + 2 * tile_elems<DP>(), p.k, p, b, r, h, kt * kT, keep);
    load_tile<T, DP>(at + 3 * tile_elems<DP>(), p.v, p, b, r, h, kt * kT, keep);
  };
  float acc[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  const int row0 = qt * kT + warp * 16 + g;
  if (first < last) request(first);
  copies_commit();
  for (int r = first; r < last; ++r) {
    if (r + 1 < last) request(r + 1);
    copies_commit();
    float norm[2], delta[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int at = row0 + 8 * half;
      const int64_t stat = ((int64_t(b) * p.rows + r) * p.heads + h) * p.cols + at;
      norm[half] = at < p.cols ? -p.lse[stat] : -INFINITY;
      delta[half] = at < p.cols ? p.delta[stat] : 0.f;
    }
    const uint64_t all = keep_bits(p, p.mask ? p.mask + b * p.m_sb + int64_t(r) * p.m_sr : nullptr, kt * kT);
    copies_wait<1>();
    __syncthreads();
    const T* Q = reinterpret_cast<const T*>(smem + ((r - first) & 1) * kStage);
    if (all) {
#pragma unroll
      for (int col0 = 0; col0 < kT; col0 += 32) {
        const uint32_t bits = uint32_t(all >> col0);
        float s[4][4], dp[4][4];
        scores<T, DP, 4>(s, Q, warp * 16, Q + 2 * tile_elems<DP>(), col0);
        scores<T, DP, 4>(dp, Q + tile_elems<DP>(), warp * 16, Q + 3 * tile_elems<DP>(), col0);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const Bias* two = add[col0 / 8 + nt][half];
            set_pair(s[nt], half, probability<T>(pair_of(s[nt], half), p.scale, make_float2(float(two[0]), float(two[1])), both(norm[half])));
            set_pair(dp[nt], half, __fadd2_rn(pair_of(dp[nt], half), both(-delta[half])));
          }
        if (bits != 0xffffffffu) {
          drop_columns(s, bits, t, 0.f);
          drop_columns(dp, bits, t, 0.f);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            float (&to)[4] = acc[col0 / 8 + nt];
            set_pair(to, half, __ffma2_rn(pair_of(s[nt], half), pair_of(dp[nt], half), pair_of(to, half)));
          }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int query = row0 + 8 * (i >> 1), key = kt * kT + nt * 8 + 2 * t + (i & 1);
      if (query >= p.cols || key >= p.cols) continue;
      if (p.num_parts > 1) {
        p.parts[(((int64_t(part) * p.batch + b) * p.heads + h) * p.cols + query) * p.cols + key] = acc[nt][i] * kDown;
      } else {
        const int64_t at = b * p.db_sb + h * p.db_sh + int64_t(query) * p.db_sq + int64_t(key) * p.db_sk;
        if (p.dbias_f32) reinterpret_cast<float*>(p.dbias)[at] = acc[nt][i] * kDown;
        else reinterpret_cast<T*>(p.dbias)[at] = T(acc[nt][i] * kDown);
      }
    }
}

template <typename T, int DP, bool B32>
__global__ void __launch_bounds__(kThreads, DP <= 32 ? 4 : 3) mma_backward_kernel(const MmaProblem p) {
  extern __shared__ __align__(16) uint8_t mma_smem[];
  const int idx = blockIdx.x;
  if (idx < p.dkv_ctas) key_gradient<T, DP, B32>(p, mma_smem, idx);
  else if (idx < p.dkv_ctas + p.dq_ctas) query_gradient<T, DP, B32>(p, mma_smem, idx - p.dkv_ctas);
  else bias_gradient<T, DP, B32>(p, mma_smem, idx - p.dkv_ctas - p.dq_ctas);
}

template <typename T>
__global__ void __launch_bounds__(256) mma_bias_sum_kernel(const float* __restrict__ parts, int num_parts, void* dbias, int f32, int64_t sb,
                                                           int64_t sh, int64_t sq, int64_t sk, int heads, int cols, int64_t plane) {
  const int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x;
  if (i >= plane) return;
  float sum = 0.f;
#pragma unroll 4
  for (int part = 0; part < num_parts; ++part) sum += parts[int64_t(part) * plane + i];
  const int64_t k = i % cols, q = i / cols % cols, z = i / (int64_t(cols) * cols);
  const int64_t at = z / heads * sb + z % heads * sh + q * sq + k * sk;
  if (f32) reinterpret_cast<float*>(dbias)[at] = sum;
  else reinterpret_cast<T*>(dbias)[at] = T(sum);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------

bool words_ok(const oops_ta_pair& t) {
  return !t.ptr || ((reinterpret_cast<uintptr_t>(t.ptr) & 15) == 0 && t.sb % 8 == 0 && t.sr % 8 == 0 && t.sc % 8 == 0 && t.sh % 8 == 0);
}

uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }
int64_t row_tiles(const oops_ta_problem& p) { return int64_t(p.batch) * p.rows * p.heads * ceil_div(p.cols, kT); }
bool shared_gradient(const oops_ta_problem& p, const oops_ta_grads& g) { return g.dbias && p.bias_groups == 1; }

// Rows are split until the bias tiles alone could fill the SMs twice; more parts only add planes to sum.
int bias_parts(const oops_ta_problem& p) {
  const int64_t tiles = int64_t(p.batch) * p.heads * ceil_div(p.cols, kT) * ceil_div(p.cols, kT);
  return (int)std::min<int64_t>(std::max<int64_t>(1, ceil_div(2 * 148, tiles)), std::min(p.rows, 16));
}

MmaProblem describe(const oops_ta_problem& p) {
  MmaProblem m{};
  m.q = p.q;
  m.k = p.k;
  m.v = p.v;
  m.mask = p.mask;
  m.m_sb = p.mask_sb;
  m.m_sr = p.mask_sr;
  m.m_sc = p.mask_sc;
  if (p.bias_groups) {
    const int word = 16 / int(dtype_size(p.bias_dtype));
    m.bias = p.bias;
    m.b_sb = p.bias_sb;
    m.b_sg = p.bias_sg;
    m.b_sh = p.bias_sh;
    m.b_sq = p.bias_sq;
    m.b_sk = p.bias_sk;
    m.bias_vec = p.bias_sk == 1 && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0 && p.bias_sb % word == 0 && p.bias_sg % word == 0 &&
                 p.bias_sh % word == 0 && p.bias_sq % word == 0;
  }
  m.batch = p.batch;
  m.rows = p.rows;
  m.cols = p.cols;
  m.heads = p.heads;
  m.dim = p.head_dim;
  m.bias_groups = p.bias_groups;
  m.scale = p.scale;
  return m;
}

template <typename Kernel>
int launch(Kernel kernel, const MmaProblem& m, int64_t grid, int smem, cudaStream_t stream, const char* what) {
  const int status = reserve_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (status) return status;
  kernel<<<(unsigned)grid, kThreads, smem, stream>>>(m);
  count_launch();
  return check_launch(what);
}

// Calls run(type, padded head size, f32 bias).
template <typename F>
int by_kind(const oops_ta_problem& p, F&& run) {
  auto sized = [&](auto type, auto b32) -> int {
    if (p.head_dim <= 16) return run(type, std::integral_constant<int, 16>{}, b32);
    if (p.head_dim <= 32) return run(type, std::integral_constant<int, 32>{}, b32);
    if (p.head_dim <= 48) return run(type, std::integral_constant<int, 48>{}, b32);
    return run(type, std::integral_constant<int, 64>{}, b32);
  };
  auto typed = [&](auto type) -> int {
    return p.bias_groups && p.bias_dtype == OOPS_TA_F32 ? sized(type, std::true_type{}) : sized(type, std::false_type{});
  };
  return p.dtype == OOPS_TA_BF16 ? typed(__nv_bfloat16{}) : typed(__half{});
}

}  // namespace

// Head sizes above 64 would need more accumulators in the dK/dV part than there are registers (up to 64 every instance of the
// reverse spills 8 to 24 bytes already); they stay with the kernels that keep logits in memory.
bool mma_applies(const oops_ta_problem& p) {
  if (p.dtype != OOPS_TA_F16 && p.dtype != OOPS_TA_BF16) return false;
  if (p.head_dim > 64) return false;
  const int64_t tiles = ceil_div(p.cols, kT);
  return 2 * row_tiles(p) + 16 * int64_t(p.batch) * p.heads * tiles * tiles <= 0x7fffffffll;
}

uint64_t mma_backward_workspace(const oops_ta_problem& p, const oops_ta_grads& g) {
  uint64_t total = align256(uint64_t(p.batch) * p.rows * p.heads * p.cols * sizeof(float));
  if (shared_gradient(p, g) && bias_parts(p) > 1)
    total += align256(uint64_t(bias_parts(p)) * p.batch * p.heads * p.cols * p.cols * sizeof(float));
  return total;
}

int mma_forward(const oops_ta_problem& p, const oops_ta_pair& out, float* lse, cudaStream_t stream) {
  if (wide_forward_applies(p, out)) return wide_forward(p, out, lse, stream);
  MmaProblem m = describe(p);
  m.out = out;
  m.lse = lse;
  m.vec = p.head_dim % 8 == 0 && words_ok(p.q) && words_ok(p.k) && words_ok(p.v) && words_ok(out);
  return by_kind(p, [&](auto type, auto width, auto b32) -> int {
    using T = decltype(type);
    constexpr int DP = decltype(width)::value;
    constexpr bool B32 = decltype(b32)::value;
    return launch(mma_forward_kernel<T, DP, B32>, m, row_tiles(p), 4 * tile_elems<DP>() * 2 + 2 * bias_bytes<B32>(), stream, "mma forward");
  });
}

int mma_backward(const oops_ta_problem& p, const oops_ta_pair& out, const oops_ta_pair& dout, const float* lse, const oops_ta_grads& g,
                 cudaStream_t stream) {
  const uint64_t need = mma_backward_workspace(p, g);
  if (p.workspace_bytes < need || !p.workspace)
    return fail(OOPS_TA_WORKSPACE_TOO_SMALL, "backward needs %llu scratch bytes, got %llu", (unsigned long long)need,
                (unsigned long long)p.workspace_bytes);
  MmaProblem m = describe(p);
  m.out = out;
  m.dout = dout;
  m.dq = g.dq;
  m.dk = g.dk;
  m.dv = g.dv;
  m.lse = const_cast<float*>(lse);
  m.vec = p.head_dim % 8 == 0;
  for (const oops_ta_pair* t : {&p.q, &p.k, &p.v, &out, &dout, &g.dq, &g.dk, &g.dv}) m.vec = m.vec && words_ok(*t);
  m.delta = reinterpret_cast<float*>(p.workspace);
  const int64_t stats = int64_t(p.batch) * p.rows * p.heads * p.cols;
  m.num_parts = 1;
  if (g.dbias) {
    m.dbias = g.dbias;
    m.db_sb = g.dbias_sb;
    m.db_sg = g.dbias_sg;
    m.db_sh = g.dbias_sh;
    m.db_sq = g.dbias_sq;
    m.db_sk = g.dbias_sk;
    m.dbias_f32 = p.bias_dtype == OOPS_TA_F32 || (p.flags & OOPS_TA_FLAG_DBIAS_F32) != 0;
    if (shared_gradient(p, g)) {
      m.num_parts = bias_parts(p);
      m.rows_per_part = (int)ceil_div(p.rows, m.num_parts);
      m.parts = reinterpret_cast<float*>(reinterpret_cast<char*>(p.workspace) + align256(uint64_t(stats) * sizeof(float)));
    }
  }
  if ((p.flags & OOPS_TA_FLAG_REUSE_DELTA) == 0) {
    const unsigned blocks = (unsigned)ceil_div(stats * 8, 256);
    if (p.dtype == OOPS_TA_BF16) mma_delta_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(m, stats);
    else mma_delta_kernel<__half><<<blocks, 256, 0, stream>>>(m, stats);
    count_launch();
    const int status = check_launch("mma delta");
    if (status) return status;
  }
  const int64_t tiles = ceil_div(p.cols, kT);
  m.dkv_ctas = g.dk.ptr || g.dv.ptr ? (int)row_tiles(p) : 0;
  m.dq_ctas = g.dq.ptr || (g.dbias && p.bias_groups > 1) ? (int)row_tiles(p) : 0;
  const int64_t grid = int64_t(m.dkv_ctas) + m.dq_ctas +
                       (shared_gradient(p, g) ? int64_t(m.num_parts) * p.batch * p.heads * tiles * tiles : 0);
  if (grid == 0) return OOPS_TA_OK;
  const bool wide = wide_backward_applies(p, dout, g);
  int status = wide ? wide_backward(p, dout, lse, m.delta, g, m.num_parts, m.parts, stream) : by_kind(p, [&](auto type, auto width, auto b32) -> int {
    using T = decltype(type);
    constexpr int DP = decltype(width)::value;
    constexpr bool B32 = decltype(b32)::value;
    constexpr int rows_smem = 6 * tile_elems<DP>() * 2 + 2 * (bias_bytes<B32>() + 2 * kT * 4);
    constexpr int bias_smem = 8 * tile_elems<DP>() * 2;
    return launch(mma_backward_kernel<T, DP, B32>, m, grid, shared_gradient(p, g) ? std::max(rows_smem, bias_smem) : rows_smem, stream,
                  "mma backward");
  });
  if (status || m.num_parts == 1) return status;
  const int64_t plane = int64_t(p.batch) * p.heads * p.cols * p.cols;
  const unsigned blocks = (unsigned)ceil_div(plane, 256);
  if (p.dtype == OOPS_TA_BF16)
    mma_bias_sum_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(m.parts, m.num_parts, m.dbias, m.dbias_f32, m.db_sb, m.db_sh, m.db_sq, m.db_sk,
                                                                   p.heads, p.cols, plane);
  else
    mma_bias_sum_kernel<__half><<<blocks, 256, 0, stream>>>(m.parts, m.num_parts, m.dbias, m.dbias_f32, m.db_sb, m.db_sh, m.db_sq, m.db_sk, p.heads,
                                                            p.cols, plane);
  count_launch();
  return check_launch("mma shared-bias sum");
}

}  // namespace oops_ta
