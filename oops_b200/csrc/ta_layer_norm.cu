// Layer normalisation over the last axis of (rows, width) activations, forward and reverse: the step before the q/k/v
// and bias projections of a pair block (reference: oops/normalization/layer_norm/layer_norm.py:37-110 and its Triton
// kernels).  Byte work bound by HBM: one warp owns a row, 16-byte accesses, every statistic in f32.
//   forward:  y = (x - mean) * rstd * weight + bias,  mean and rstd (f32 per row) kept for the reverse pass
//   reverse:  g = dy * weight, xhat = (x - mean) * rstd,
//             dx = rstd * (g - mean_c(g) - xhat * mean_c(g * xhat)),  dweight = sum_rows dy * xhat,  dbias = sum_rows dy
// Rows of up to 1024 elements live in registers between the passes over them (one read of x per kernel); wider rows
// (up to 8192) are read again from L2.  dweight and dbias are summed per warp in registers over the rows the warp
// walks, then per CTA in shared memory, written as f32 partial rows and added in a fixed order by a second small
// kernel: bitwise reproducible, no atomics.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <initializer_list>
#include <type_traits>

#include "ta_internal.h"

namespace oops_ta {
namespace {

constexpr int kLnWarps = 8;             // warps (= rows in flight) per CTA
constexpr int kLnCached = 1024;         // widest row kept in registers
constexpr int kLnPerLane = kLnCached / 32;
constexpr int kLnCtasPerSm = 4;         // most CTAs that a launch has per SM

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// V consecutive elements of a row: one element (any alignment), or 16 bytes (V = 4 for f32, 8 for 16-bit types).
template <typename T, int V>
struct LnVec {
  static __device__ __forceinline__ void load(const T* p, float (&out)[V]) {
    if constexpr (V == 1) {
      out[0] = float(*p);
    } else if constexpr (sizeof(T) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(p);
      out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    } else {
      const uint4 v = *reinterpret_cast<const uint4*>(p);
      const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = float(e[i]);
    }
  }
  static __device__ __forceinline__ void store(T* p, const float (&in)[V]) {
    if constexpr (V == 1) {
      *p = T(in[0]);
    } else if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(p) = make_float4(in[0], in[1], in[2], in[3]);
    } else {
      uint4 v;
      T* e = reinterpret_cast<T*>(&v);
#pragma unroll
      for (int i = 0; i < 8; ++i) e[i] = T(in[i]);
      *reinterpret_cast<uint4*>(p) = v;
    }
  }
};

// First element of group g of lane `lane`: a warp's accesses are 32 * V contiguous elements.
template <int V>
__device__ __forceinline__ int ln_first(int lane, int g) { return (g * 32 + lane) * V; }

struct LnShape {
  int64_t rows;
  int width;
  int64_t x_stride, y_stride, dy_stride, dx_stride;  // row strides in elements
  int share = 0;  // row blocks of a warp where a turn of every warp is more than there are (the kernels that share rows)
};

// affine parameters may be of the activation type or f32 ("master" parameters of 16-bit activations)
template <typename A>
__device__ __forceinline__ float affine_at(const void* p, int i, float missing) {
  return p ? float(reinterpret_cast<const A*>(p)[i]) : missing;
}

template <typename T, typename A, int V, bool CACHED>
__global__ void __launch_bounds__(kLnWarps * 32) layer_norm_forward_kernel(LnShape s, const T* __restrict__ x,
                                                                           const void* __restrict__ weight,
                                                                           const void* __restrict__ bias, float eps,
                                                                           T* __restrict__ y, float* __restrict__ mean_out,
                                                                           float* __restrict__ rstd_out) {
  constexpr int kGroups = kLnPerLane / V;  // groups of V elements a lane holds of a cached row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float inv_width = 1.f / float(s.width);
  for (int64_t row = int64_t(blockIdx.x) * kLnWarps + warp; row < s.rows; row += int64_t(gridDim.x) * kLnWarps) {
    const T* xr = x + row * s.x_stride;
    T* yr = y + row * s.y_stride;
    float vals[CACHED ? kGroups : 1][V];
    float sum = 0.f;
    if (CACHED) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int i = ln_first<V>(lane, g);
#pragma unroll
        for (int e = 0; e < V; ++e) vals[g][e] = 0.f;
        if (i < s.width) LnVec<T, V>::load(xr + i, vals[g]);
#pragma unroll
        for (int e = 0; e < V; ++e) sum += vals[g][e];
      }
    } else {
      for (int i = lane; i < s.width; i += 32) sum += float(xr[i]);
    }
    const float mean = warp_sum(sum) * inv_width;
    float sq = 0.f;
    if (CACHED) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        if (ln_first<V>(lane, g) < s.width) {
#pragma unroll
          for (int e = 0; e < V; ++e) {
            const float d = vals[g][e] - mean;
            sq += d * d;
          }
        }
      }
    } else {
      for (int i = lane; i < s.width; i += 32) {
        const float d = float(xr[i]) - mean;
        sq += d * d;
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) * inv_width + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    if (CACHED) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int i = ln_first<V>(lane, g);
        if (i < s.width) {
          float out[V];
#pragma unroll
          for (int e = 0; e < V; ++e)
            out[e] = (vals[g][e] - mean) * rstd * affine_at<A>(weight, i + e, 1.f) + affine_at<A>(bias, i + e, 0.f);
          LnVec<T, V>::store(yr + i, out);
        }
      }
    } else {
      for (int i = lane; i < s.width; i += 32)
        yr[i] = T((float(xr[i]) - mean) * rstd * affine_at<A>(weight, i, 1.f) + affine_at<A>(bias, i, 0.f));
    }
  }
}

// Reverse pass.  dweight/dbias: every lane sums its columns over the rows its warp walks (cached rows only), the
// eight warps of a CTA are added through shared memory, and the CTA writes one f32 partial row per tensor.
template <typename T, typename A, int V, bool CACHED>
__global__ void __launch_bounds__(kLnWarps * 32) layer_norm_backward_kernel(LnShape s, const T* __restrict__ dy,
                                                                            const T* __restrict__ x,
                                                                            const void* __restrict__ weight,
                                                                            const float* __restrict__ mean_in,
                                                                            const float* __restrict__ rstd_in,
                                                                            T* __restrict__ dx, float* __restrict__ dw_parts,
                                                                            float* __restrict__ db_parts) {
  constexpr int kGroups = kLnPerLane / V;
  extern __shared__ float ln_smem[];  // [kLnWarps][width] when partials are wanted
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float inv_width = 1.f / float(s.width);
  const bool want_parts = CACHED && (dw_parts != nullptr || db_parts != nullptr);
  float dw[CACHED ? kGroups : 1][V], db[CACHED ? kGroups : 1][V];
#pragma unroll
  for (int g = 0; g < (CACHED ? kGroups : 1); ++g)
#pragma unroll
    for (int e = 0; e < V; ++e) dw[g][e] = db[g][e] = 0.f;

  for (int64_t row = int64_t(blockIdx.x) * kLnWarps + warp; row < s.rows; row += int64_t(gridDim.x) * kLnWarps) {
    const T* xr = x + row * s.x_stride;
    const T* gr = dy + row * s.dy_stride;
    const float mean = mean_in[row], rstd = rstd_in[row];
    if (CACHED) {
      float xh[kGroups][V], gw[kGroups][V];
      float c1 = 0.f, c2 = 0.f;
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int i = ln_first<V>(lane, g);
#pragma unroll
        for (int e = 0; e < V; ++e) xh[g][e] = gw[g][e] = 0.f;
        if (i < s.width) {
          float xv[V], gv[V];
          LnVec<T, V>::load(xr + i, xv);
          LnVec<T, V>::load(gr + i, gv);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            xh[g][e] = (xv[e] - mean) * rstd;
            dw[g][e] += gv[e] * xh[g][e];
            db[g][e] += gv[e];
            gw[g][e] = gv[e] * affine_at<A>(weight, i + e, 1.f);
            c1 += gw[g][e] * xh[g][e];
            c2 += gw[g][e];
          }
        }
      }
      c1 = warp_sum(c1) * inv_width;
      c2 = warp_sum(c2) * inv_width;
      if (dx) {
        T* dr = dx + row * s.dx_stride;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          const int i = ln_first<V>(lane, g);
          if (i < s.width) {
            float out[V];
#pragma unroll
            for (int e = 0; e < V; ++e) out[e] = rstd * (gw[g][e] - c2 - xh[g][e] * c1);
            LnVec<T, V>::store(dr + i, out);
          }
        }
      }
    } else {
      float c1 = 0.f, c2 = 0.f;
      for (int i = lane; i < s.width; i += 32) {
        const float xhat = (float(xr[i]) - mean) * rstd, g = float(gr[i]) * affine_at<A>(weight, i, 1.f);
        c1 += g * xhat;
        c2 += g;
      }
      c1 = warp_sum(c1) * inv_width;
      c2 = warp_sum(c2) * inv_width;
      if (dx) {
        T* dr = dx + row * s.dx_stride;
        for (int i = lane; i < s.width; i += 32) {
          const float xhat = (float(xr[i]) - mean) * rstd, g = float(gr[i]) * affine_at<A>(weight, i, 1.f);
          dr[i] = T(rstd * (g - c2 - xhat * c1));
        }
      }
    }
  }
  if (want_parts) {
    for (int pass = 0; pass < 2; ++pass) {
      float* parts = pass == 0 ? dw_parts : db_parts;
      if (!parts) continue;
      __syncthreads();
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int i = ln_first<V>(lane, g);
        if (i < s.width) {
#pragma unroll
          for (int e = 0; e < V; ++e) ln_smem[warp * s.width + i + e] = pass == 0 ? dw[g][e] : db[g][e];
        }
      }
      __syncthreads();
      for (int i = threadIdx.x; i < s.width; i += kLnWarps * 32) {
        float total = 0.f;
#pragma unroll
        for (int w = 0; w < kLnWarps; ++w) total += ln_smem[w * s.width + i];
        parts[int64_t(blockIdx.x) * s.width + i] = total;
      }
    }
  }
}

// ---- rows of up to 1024 elements with 16-byte accesses: LPR lanes share a row, each holding GROUPS groups of V
// elements; a warp works on 32 / LPR rows at once and on kLnUnroll such row blocks per loop turn, so that enough
// loads are in flight to cover the memory latency (a 128-channel bf16 row is only 256 bytes).
constexpr int kLnUnroll = 4;

template <int LPR>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Packed arithmetic: a group of V elements is V / 2 pairs of f32, and every add / multiply-add below works on a pair
// (fma.rn.f32x2 and friends), which halves the instructions per byte; 16-bit rows were bound by instruction issue.
typedef float2 ln2;
__device__ __forceinline__ ln2 ln_fma2(ln2 a, ln2 b, ln2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ ln2 ln_add2(ln2 a, ln2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ ln2 ln_mul2(ln2 a, ln2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ ln2 ln_both(float v) { return make_float2(v, v); }

template <typename T, int V>
__device__ __forceinline__ void ln_unpack2(const uint4& raw, ln2 (&out)[V / 2]) {
  static_assert(V * sizeof(T) == 16, "a raw group is 16 bytes");
  if constexpr (sizeof(T) == 4) {
    out[0] = make_float2(__uint_as_float(raw.x), __uint_as_float(raw.y));
    out[1] = make_float2(__uint_as_float(raw.z), __uint_as_float(raw.w));
  } else {
    const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        out[i] = make_float2(__uint_as_float(words[i] << 16), __uint_as_float(words[i] & 0xffff0000u));
      } else {
        out[i] = __half22float2(*reinterpret_cast<const __half2*>(&words[i]));
      }
    }
  }
}

template <typename T, int V>
__device__ __forceinline__ uint4 ln_pack2(const ln2 (&in)[V / 2]) {
  if constexpr (sizeof(T) == 4) {
    return make_uint4(__float_as_uint(in[0].x), __float_as_uint(in[0].y), __float_as_uint(in[1].x), __float_as_uint(in[1].y));
  } else {
    uint32_t words[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        const __nv_bfloat162 h = __float22bfloat162_rn(in[i]);
        words[i] = *reinterpret_cast<const uint32_t*>(&h);
      } else {
        const __half2 h = __float22half2_rn(in[i]);
        words[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    return make_uint4(words[0], words[1], words[2], words[3]);
  }
}

// Row blocks that a lane has asked for stand in shared memory, 16 bytes of its own each, which no other lane touches: the blocks of the
// next turn travel under the arithmetic of this one, and cost no registers (held in registers they spill).  A warp's blocks of a turn
// are neighbours, 2 KB in a row.  768 x 768 rows of 128 channels, bf16: forward 64.9 -> 50.8 us (5.9 TB/s; the copy reaches 6.56),
// reverse 86.9 -> 75.0 (6.0 TB/s); 200000 rows of 256: 39.6 -> 30.5 and 68.1 -> 53.9; f32 rows of 512 bytes that fill the L2 several times over
// were at 6.2 TB/s and stay there.
constexpr int ln_turn(int groups, int tensors, bool staged) { return staged ? kLnUnroll / (groups * tensors) : kLnUnroll / tensors; }  // row blocks
// Resident CTAs per SM: with a turn ahead, two keep HBM busy and have the registers for four blocks' arithmetic side by side; f32 forward
// rows need fewer registers (700000 x 128: 120 us with two, 116 with three, 131 with four).
constexpr int ln_ctas(int tensors, int size, bool staged) { return !staged ? kLnCtasPerSm : size == 4 && tensors == 1 ? 3 : 2; }
constexpr int kLnStage = kLnUnroll * kLnWarps * 32 * 16;  // bytes of a turn of a CTA, whatever the groups and tensors
__device__ __forceinline__ void ln_copy16(uint32_t to, const void* from, bool take) {  // zeros where it is not taken
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(take ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ln_copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ln_copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 ln_take16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

template <typename T, typename A, int V, int GROUPS, int LPR, bool STAGED>
__global__ void __launch_bounds__(kLnWarps * 32, STAGED || GROUPS == 1 ? ln_ctas(1, sizeof(T), STAGED) : 1) layer_norm_forward_rows_kernel(LnShape s, const T* __restrict__ x,
                                                                                const void* __restrict__ weight,
                                                                                const void* __restrict__ bias, float eps,
                                                                                T* __restrict__ y, float* __restrict__ mean_out,
                                                                                float* __restrict__ rstd_out) {
  constexpr int kRowsPerWarp = 32 / LPR, P = V / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / LPR, l = lane % LPR;
  const float inv_width = 1.f / float(s.width);
  // this lane's affine parameters, fetched once (zero outside the row)
  ln2 w[GROUPS][P], b[GROUPS][P];
#pragma unroll
  for (int g = 0; g < GROUPS; ++g)
#pragma unroll
    for (int e = 0; e < P; ++e) {
      const int i = (g * LPR + l) * V + 2 * e;
      const bool in = i < s.width;
      w[g][e] = make_float2(in ? affine_at<A>(weight, i, 1.f) : 0.f, in ? affine_at<A>(weight, i + 1, 1.f) : 0.f);
      b[g][e] = make_float2(in ? affine_at<A>(bias, i, 0.f) : 0.f, in ? affine_at<A>(bias, i + 1, 0.f) : 0.f);
    }
  const int64_t blocks = (s.rows + kRowsPerWarp - 1) / kRowsPerWarp;  // row blocks of one warp
  const int64_t stride = int64_t(gridDim.x) * kLnWarps;
  constexpr int kTurn = ln_turn(GROUPS, 1, STAGED);
  extern __shared__ __align__(16) float ln_smem[];
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(ln_smem) + threadIdx.x * 16;
  constexpr uint32_t kPiece = kLnWarps * 32 * 16;  // 16 bytes of every lane
  // A warp's blocks of a turn are neighbours.  `left` rows are there from the turn's first one on; a turn later they are `ahead` fewer.
  constexpr int64_t apart = kRowsPerWarp;
  const int64_t ahead = stride * kTurn * kRowsPerWarp, x_apart = apart * s.x_stride, y_apart = apart * s.y_stride;
  const int64_t first = (int64_t(blockIdx.x) * kLnWarps + warp) * s.share;
  int64_t row = first * kRowsPerWarp + sub, left = s.rows - row;
  if (s.share < kTurn) left = min(left, s.share * apart);
  const T* from = x + row * s.x_stride + l * V;
  T* to = y + row * s.y_stride + l * V;
  auto request = [&](int64_t left, uint32_t at) {  // `from` is the turn's first row
#pragma unroll
    for (int u = 0; u < kTurn; ++u) {
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        const bool take = u * apart < left && (g * LPR + l) * V < s.width;
        ln_copy16(at + (u * GROUPS + g) * kPiece, take ? from + u * x_apart + g * LPR * V : x, take);
      }
    }
    from += ahead * s.x_stride;
  };
  if constexpr (STAGED) {
    request(left, mine);
    ln_copies_commit();
  }
  uint32_t stage = 0;
  for (int64_t blk0 = first; blk0 < blocks; blk0 += stride * kTurn, row += ahead, left -= ahead, to += ahead * s.y_stride) {
    uint4 raw[kTurn][GROUPS];
    if constexpr (STAGED) {
      if (blk0 + stride * kTurn < blocks) request(left - ahead, mine + (stage ^ kLnStage));
      ln_copies_commit();
      ln_copies_wait<1>();
#pragma unroll
      for (int u = 0; u < kTurn; ++u)
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) raw[u][g] = ln_take16(mine + stage + (u * GROUPS + g) * kPiece);
      stage ^= kLnStage;
    } else {
#pragma unroll
      for (int u = 0; u < kTurn; ++u) {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          raw[u][g] = make_uint4(0, 0, 0, 0);  // zero bits are 0.0 in every served type
          if (u * apart < left && (g * LPR + l) * V < s.width)
            raw[u][g] = *reinterpret_cast<const uint4*>(from + u * x_apart + g * LPR * V);
        }
      }
      from += ahead * s.x_stride;
    }
#pragma unroll
    for (int u = 0; u < kTurn; ++u) {
      const bool live = u * apart < left;
      ln2 v[GROUPS][P];
      ln2 sum2 = ln_both(0.f);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        ln_unpack2<T, V>(raw[u][g], v[g]);
#pragma unroll
        for (int e = 0; e < P; ++e) sum2 = ln_add2(sum2, v[g][e]);
      }
      const float mean = row_sum<LPR>(sum2.x + sum2.y) * inv_width;
      const ln2 neg_mean = ln_both(-mean);
      ln2 sq2 = ln_both(0.f);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g)
        if ((g * LPR + l) * V < s.width) {
#pragma unroll
          for (int e = 0; e < P; ++e) {
            v[g][e] = ln_add2(v[g][e], neg_mean);  // centred from here on
            sq2 = ln_fma2(v[g][e], v[g][e], sq2);
          }
        }
      const float rstd = rsqrtf(row_sum<LPR>(sq2.x + sq2.y) * inv_width + eps);
      if (!live) continue;
      if (l == 0) {
        if (mean_out) mean_out[row + u * apart] = mean;
        if (rstd_out) rstd_out[row + u * apart] = rstd;
      }
      const ln2 rstd2 = ln_both(rstd);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        const int i = (g * LPR + l) * V;
        if (i < s.width) {
          ln2 out[P];
#pragma unroll
          for (int e = 0; e < P; ++e) out[e] = ln_fma2(ln_mul2(v[g][e], rstd2), w[g][e], b[g][e]);
          *reinterpret_cast<uint4*>(to + u * y_apart + g * LPR * V) = ln_pack2<T, V>(out);
        }
      }
    }
  }
  if constexpr (STAGED) ln_copies_wait<0>();  // (the request for a turn that does not come)
}

template <typename T, typename A, int V, int GROUPS, int LPR, bool STAGED>
__global__ void __launch_bounds__(kLnWarps * 32, STAGED || GROUPS == 1 ? ln_ctas(2, sizeof(T), STAGED) : 1) layer_norm_backward_rows_kernel(LnShape s, const T* __restrict__ dy,
                                                                                 const T* __restrict__ x,
                                                                                 const void* __restrict__ weight,
                                                                                 const float* __restrict__ mean_in,
                                                                                 const float* __restrict__ rstd_in,
                                                                                 T* __restrict__ dx, float* __restrict__ dw_parts,
                                                                                 float* __restrict__ db_parts) {
  constexpr int kRowsPerWarp = 32 / LPR, P = V / 2;
  constexpr int kU = ln_turn(GROUPS, 2, STAGED);  // two tensors are read per row
  extern __shared__ __align__(16) float ln_smem[];  // two turns' row blocks; then [kLnWarps * kRowsPerWarp][width] when partials are wanted
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / LPR, l = lane % LPR;
  const float inv_width = 1.f / float(s.width);
  ln2 w[GROUPS][P], dw[GROUPS][P], db[GROUPS][P];
#pragma unroll
  for (int g = 0; g < GROUPS; ++g)
#pragma unroll
    for (int e = 0; e < P; ++e) {
      const int i = (g * LPR + l) * V + 2 * e;
      const bool in = i < s.width;
      w[g][e] = make_float2(in ? affine_at<A>(weight, i, 1.f) : 0.f, in ? affine_at<A>(weight, i + 1, 1.f) : 0.f);
      dw[g][e] = db[g][e] = ln_both(0.f);
    }
  const int64_t blocks = (s.rows + kRowsPerWarp - 1) / kRowsPerWarp;
  const int64_t stride = int64_t(gridDim.x) * kLnWarps;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(ln_smem) + threadIdx.x * 16;
  constexpr uint32_t kPiece = kLnWarps * 32 * 16;  // 16 bytes of every lane
  // A warp's blocks of a turn are neighbours.  `left` rows are there from the turn's first one on; a turn later they are `ahead` fewer.
  constexpr int64_t apart = kRowsPerWarp;
  const int64_t ahead = stride * kU * kRowsPerWarp, x_apart = apart * s.x_stride, g_apart = apart * s.dy_stride, d_apart = apart * s.dx_stride;
  const int64_t first = (int64_t(blockIdx.x) * kLnWarps + warp) * s.share, row0 = first * kRowsPerWarp + sub;
  int64_t left = s.rows - row0;
  if (s.share < kU) left = min(left, s.share * apart);
  const T* from_x = x + row0 * s.x_stride + l * V;
  const T* from_g = dy + row0 * s.dy_stride + l * V;
  T* to = dx + row0 * s.dx_stride + l * V;
  const float* mean_at = mean_in + row0;
  const float* rstd_at = rstd_in + row0;
  float mean_next[kU], rstd_next[kU];
  auto request = [&](int64_t left, uint32_t at) {  // the pointers are at the turn's first row
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const bool there = u * apart < left;
      mean_next[u] = there ? mean_at[u * apart] : 0.f;
      rstd_next[u] = there ? rstd_at[u * apart] : 0.f;
      if constexpr (STAGED) {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          const bool take = there && (g * LPR + l) * V < s.width;
          ln_copy16(at + (2 * (u * GROUPS + g)) * kPiece, take ? from_x + u * x_apart + g * LPR * V : x, take);
          ln_copy16(at + (2 * (u * GROUPS + g) + 1) * kPiece, take ? from_g + u * g_apart + g * LPR * V : dy, take);
        }
      }
    }
    mean_at += ahead;
    rstd_at += ahead;
    if constexpr (STAGED) {
      from_x += ahead * s.x_stride;
      from_g += ahead * s.dy_stride;
      ln_copies_commit();
    }
  };
  request(left, mine);
  uint32_t stage = 0;
  for (int64_t blk0 = first; blk0 < blocks; blk0 += stride * kU, left -= ahead, to += ahead * s.dx_stride) {
    uint4 xraw[kU][GROUPS], graw[kU][GROUPS];
    float mean[kU], rstd[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      mean[u] = mean_next[u];
      rstd[u] = rstd_next[u];
    }
    request(left - ahead, mine + (stage ^ kLnStage));
    if constexpr (STAGED) {
      ln_copies_wait<1>();
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          xraw[u][g] = ln_take16(mine + stage + (2 * (u * GROUPS + g)) * kPiece);
          graw[u][g] = ln_take16(mine + stage + (2 * (u * GROUPS + g) + 1) * kPiece);
        }
      stage ^= kLnStage;
    } else {
#pragma unroll
      for (int u = 0; u < kU; ++u) {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          xraw[u][g] = graw[u][g] = make_uint4(0, 0, 0, 0);
          if (u * apart < left && (g * LPR + l) * V < s.width) {
            xraw[u][g] = *reinterpret_cast<const uint4*>(from_x + u * x_apart + g * LPR * V);
            graw[u][g] = *reinterpret_cast<const uint4*>(from_g + u * g_apart + g * LPR * V);
          }
        }
      }
      from_x += ahead * s.x_stride;
      from_g += ahead * s.dy_stride;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const bool live = u * apart < left;
      const ln2 rstd2 = ln_both(rstd[u]), neg_mean2 = ln_both(-mean[u]);
      ln2 xh[GROUPS][P], gw[GROUPS][P];
      ln2 c1 = ln_both(0.f), c2 = ln_both(0.f);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        ln2 gv[P];
        ln_unpack2<T, V>(xraw[u][g], xh[g]);
        ln_unpack2<T, V>(graw[u][g], gv);
        const bool inside = live && (g * LPR + l) * V < s.width;
#pragma unroll
        for (int e = 0; e < P; ++e) {
          xh[g][e] = inside ? ln_mul2(ln_add2(xh[g][e], neg_mean2), rstd2) : ln_both(0.f);
          dw[g][e] = ln_fma2(gv[e], xh[g][e], dw[g][e]);
          db[g][e] = ln_add2(db[g][e], gv[e]);
          gw[g][e] = ln_mul2(gv[e], w[g][e]);
          c1 = ln_fma2(gw[g][e], xh[g][e], c1);
          c2 = ln_add2(c2, gw[g][e]);
        }
      }
      const float m1 = row_sum<LPR>(c1.x + c1.y) * inv_width, m2 = row_sum<LPR>(c2.x + c2.y) * inv_width;
      if (!live || !dx) continue;
      const ln2 neg_m1 = ln_both(-m1), neg_m2 = ln_both(-m2);
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        const int i = (g * LPR + l) * V;
        if (i < s.width) {
          ln2 out[P];
#pragma unroll
          for (int e = 0; e < P; ++e) out[e] = ln_mul2(ln_fma2(xh[g][e], neg_m1, ln_add2(gw[g][e], neg_m2)), rstd2);
          *reinterpret_cast<uint4*>(to + u * d_apart + g * LPR * V) = ln_pack2<T, V>(out);
        }
      }
    }
  }
  // The request for a turn that does not come is still under way, as zeros; the sums below take the memory that it writes.
  if constexpr (STAGED) ln_copies_wait<0>();
  if (dw_parts != nullptr || db_parts != nullptr) {
    constexpr int kSubs = kLnWarps * kRowsPerWarp;
    for (int pass = 0; pass < 2; ++pass) {
      float* parts = pass == 0 ? dw_parts : db_parts;
      if (!parts) continue;
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GROUPS; ++g)
#pragma unroll
        for (int e = 0; e < P; ++e) {
          const int i = (g * LPR + l) * V + 2 * e;
          if (i < s.width) {
            const ln2 v = pass == 0 ? dw[g][e] : db[g][e];
            ln_smem[(warp * kRowsPerWarp + sub) * s.width + i] = v.x;
            ln_smem[(warp * kRowsPerWarp + sub) * s.width + i + 1] = v.y;
          }
        }
      __syncthreads();
      for (int i = threadIdx.x; i < s.width; i += kLnWarps * 32) {
        float total = 0.f;
        for (int k = 0; k < kSubs; ++k) total += ln_smem[k * s.width + i];
        parts[int64_t(blockIdx.x) * s.width + i] = total;
      }
    }
  }
}

// Column sums for rows too wide to keep per-lane sums in registers: CTA (column block, row part), one column per thread.
template <typename T>
__global__ void layer_norm_wide_parts_kernel(LnShape s, const T* __restrict__ dy, const T* __restrict__ x,
                                             const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                                             int64_t rows_per_part, float* __restrict__ dw_parts, float* __restrict__ db_parts) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= s.width) return;
  const int64_t first = int64_t(blockIdx.y) * rows_per_part, last = min(first + rows_per_part, s.rows);
  float dw = 0.f, db = 0.f;
  for (int64_t row = first; row < last; ++row) {
    const float g = float(dy[row * s.dy_stride + col]);
    dw += g * (float(x[row * s.x_stride + col]) - mean_in[row]) * rstd_in[row];
    db += g;
  }
  if (dw_parts) dw_parts[int64_t(blockIdx.y) * s.width + col] = dw;
  if (db_parts) db_parts[int64_t(blockIdx.y) * s.width + col] = db;
}

// out[col] = sum over parts of parts[part][col], stored in the parameter's type, for dweight (blockIdx.y = 0) and
// dbias (1) in one launch.  A block owns 32 columns; its eight warps each add every eighth partial row (coalesced
// 128-byte reads), and the eight sums are added in warp order: the order is fixed, so the result is reproducible.
template <typename A>
__global__ void __launch_bounds__(256) layer_norm_reduce_parts_kernel(const float* __restrict__ dw_parts,
                                                                      const float* __restrict__ db_parts, int num_parts, int width,
                                                                      A* __restrict__ dweight, A* __restrict__ dbias) {
  __shared__ float sums[8][32];
  const float* parts = blockIdx.y == 0 ? dw_parts : db_parts;
  A* out = blockIdx.y == 0 ? dweight : dbias;
  if (!parts || !out) return;  // the whole block takes the same branch
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.x * 32 + lane;
  float total = 0.f;
  if (col < width)
    for (int p = warp; p < num_parts; p += 8) total += parts[int64_t(p) * width + col];
  sums[warp][lane] = total;
  __syncthreads();
  if (warp == 0 && col < width) {
    float all = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) all += sums[w][lane];
    out[col] = A(all);
  }
}

constexpr int kLnMaxWidth = 8192;
constexpr int kLnWideParts = 64;

int sm_total() {
  int device = 0, sms = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

// The launch of a kernel that shares rows: `share` row blocks of a warp in a turn, and as many CTAs as then have rows.  A turn is all of its
// blocks except where they would leave SMs without any: a warp works through its blocks in turn (64 f32 rows of 384: 3.6 us with four a
// warp, 3.1 with one), but more warps than one CTA per SM has gain nothing (4096 of them: 5.7 us with four, 9.5 with one).
struct LnLaunch {
  int grid, share;
};
LnLaunch ln_launch(int64_t rows, int lanes, int turn, int ctas_per_sm) {
  const int64_t blocks = (rows + 32 / lanes - 1) / (32 / lanes), warps = int64_t(sm_total()) * kLnWarps;
  const int64_t share = std::min<int64_t>(turn, (blocks + warps - 1) / warps);
  return {int(std::min<int64_t>(int64_t(sm_total()) * ctas_per_sm, (blocks + share * kLnWarps - 1) / (share * kLnWarps))), int(share)};
}

int ln_grid(int64_t rows) { return int(std::min<int64_t>((rows + kLnWarps - 1) / kLnWarps, int64_t(sm_total()) * kLnCtasPerSm)); }

bool ln_vector_ok(int vec, int width, std::initializer_list<const void*> pointers, std::initializer_list<int64_t> strides) {
  if (width % vec) return false;
  for (const void* p : pointers)
    if (p && (reinterpret_cast<uintptr_t>(p) & 15)) return false;
  for (int64_t st : strides)
    if (st % vec) return false;
  return true;
}

template <typename T, typename A>
int forward_typed(const LnShape& s, const void* x, const void* weight, const void* bias, float eps, void* y, float* mean,
                  float* rstd, cudaStream_t stream) {
  constexpr int kVec = 16 / int(sizeof(T));
  const bool vec = ln_vector_ok(kVec, s.width, {x, y}, {s.x_stride, s.y_stride});
  const bool cached = s.width <= kLnCached;
  const int grid = ln_grid(s.rows), threads = kLnWarps * 32;
  const T* xp = reinterpret_cast<const T*>(x);
  T* yp = reinterpret_cast<T*>(y);
  const int units = (s.width + kVec - 1) / kVec;  // 16-byte groups of a row
  if (vec && units <= 128) {
    auto rows = [&](auto groups, auto lanes, auto staged) {
      constexpr int GROUPS = decltype(groups)::value, LPR = decltype(lanes)::value;
      constexpr bool STAGED = decltype(staged)::value;
      const LnLaunch launch = ln_launch(s.rows, LPR, ln_turn(GROUPS, 1, STAGED), ln_ctas(1, sizeof(T), STAGED));
      LnShape shared = s;
      shared.share = launch.share;
      layer_norm_forward_rows_kernel<T, A, kVec, GROUPS, LPR, STAGED>
          <<<launch.grid, threads, STAGED ? 2 * kLnStage : 0, stream>>>(shared, xp, weight, bias, eps, yp, mean, rstd);
    };
    using std::integral_constant;
    if (units <= 8) rows(integral_constant<int, 1>{}, integral_constant<int, 8>{}, std::true_type{});
    else if (units <= 16) rows(integral_constant<int, 1>{}, integral_constant<int, 16>{}, std::true_type{});
    else if (units <= 32) rows(integral_constant<int, 2>{}, integral_constant<int, 16>{}, std::true_type{});
    else if (units <= 64) rows(integral_constant<int, 2>{}, integral_constant<int, 32>{}, std::true_type{});
    else rows(integral_constant<int, 4>{}, integral_constant<int, 32>{}, std::false_type{});
  } else if (cached && vec)
    layer_norm_forward_kernel<T, A, kVec, true><<<grid, threads, 0, stream>>>(s, xp, weight, bias, eps, yp, mean, rstd);
  else if (cached)
    layer_norm_forward_kernel<T, A, 1, true><<<grid, threads, 0, stream>>>(s, xp, weight, bias, eps, yp, mean, rstd);
  else
    layer_norm_forward_kernel<T, A, 1, false><<<grid, threads, 0, stream>>>(s, xp, weight, bias, eps, yp, mean, rstd);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OOPS_TA_OK : OOPS_TA_CUDA_ERROR;
}

template <typename T, typename A>
int backward_typed(const LnShape& s, const void* dy, const void* x, const void* weight, const float* mean, const float* rstd,
                   void* dx, void* dweight, void* dbias, float* workspace, cudaStream_t stream) {
  constexpr int kVec = 16 / int(sizeof(T));
  const bool vec = ln_vector_ok(kVec, s.width, {x, dy, dx}, {s.x_stride, s.dy_stride, s.dx_stride});
  const bool cached = s.width <= kLnCached;
  int grid = ln_grid(s.rows);
  const int threads = kLnWarps * 32;
  const bool parts_wanted = dweight != nullptr || dbias != nullptr;
  const int units = (s.width + kVec - 1) / kVec;
  const bool shared_rows = vec && units <= 128;  // several lanes (not always a whole warp) share a row
  const int lpr = units <= 8 ? 8 : units <= 16 ? 16 : 32;
  const bool staged = units <= 64;
  const LnLaunch launch = ln_launch(s.rows, lpr, ln_turn(units <= 32 ? 1 : units <= 64 ? 2 : 4, 2, staged), ln_ctas(2, sizeof(T), staged));
  if (shared_rows) grid = launch.grid;
  const int num_parts = cached ? grid : int(s.rows < kLnWideParts ? s.rows : kLnWideParts);
  float* dw_parts = dweight ? workspace : nullptr;
  float* db_parts = dbias ? workspace + int64_t(num_parts) * s.width : nullptr;
  const T* gp = reinterpret_cast<const T*>(dy);
  const T* xp = reinterpret_cast<const T*>(x);
  T* dp = reinterpret_cast<T*>(dx);
  const size_t smem = cached && parts_wanted ? size_t(kLnWarps) * s.width * sizeof(float) : 0;
  if (shared_rows) {
    const size_t parts_smem = parts_wanted ? size_t(kLnWarps) * (32 / lpr) * s.width * sizeof(float) : 0;
    auto rows = [&](auto groups_of, auto lanes, auto staged) {
      constexpr int GROUPS = decltype(groups_of)::value, LPR = decltype(lanes)::value;
      constexpr bool STAGED = decltype(staged)::value;
      LnShape shared = s;
      shared.share = launch.share;
      layer_norm_backward_rows_kernel<T, A, kVec, GROUPS, LPR, STAGED>
          <<<grid, threads, std::max(parts_smem, size_t(STAGED ? 2 * kLnStage : 0)), stream>>>(shared, gp, xp, weight, mean, rstd, dp, dw_parts,
                                                                                              db_parts);
    };
    using std::integral_constant;
    if (units <= 8) rows(integral_constant<int, 1>{}, integral_constant<int, 8>{}, std::true_type{});
    else if (units <= 16) rows(integral_constant<int, 1>{}, integral_constant<int, 16>{}, std::true_type{});
    else if (units <= 32) rows(integral_constant<int, 1>{}, integral_constant<int, 32>{}, std::true_type{});
    else if (units <= 64) rows(integral_constant<int, 2>{}, integral_constant<int, 32>{}, std::true_type{});
    else rows(integral_constant<int, 4>{}, integral_constant<int, 32>{}, std::false_type{});
  } else if (cached && vec)
    layer_norm_backward_kernel<T, A, kVec, true><<<grid, threads, smem, stream>>>(s, gp, xp, weight, mean, rstd, dp, dw_parts, db_parts);
  else if (cached)
    layer_norm_backward_kernel<T, A, 1, true><<<grid, threads, smem, stream>>>(s, gp, xp, weight, mean, rstd, dp, dw_parts, db_parts);
  else if (dx)
    layer_norm_backward_kernel<T, A, 1, false><<<grid, threads, 0, stream>>>(s, gp, xp, weight, mean, rstd, dp, nullptr, nullptr);
  if (cached || dx) count_launch();
  if (parts_wanted) {
    if (!cached) {
      const int64_t rows_per_part = (s.rows + num_parts - 1) / num_parts;
      layer_norm_wide_parts_kernel<T><<<dim3((s.width + 127) / 128, num_parts), 128, 0, stream>>>(s, gp, xp, mean, rstd, rows_per_part,
                                                                                                  dw_parts, db_parts);
      count_launch();
    }
    layer_norm_reduce_parts_kernel<A><<<dim3((s.width + 31) / 32, 2), 256, 0, stream>>>(
        dw_parts, db_parts, num_parts, s.width, reinterpret_cast<A*>(dweight), reinterpret_cast<A*>(dbias));
    count_launch();
  }
  return cudaGetLastError() == cudaSuccess ? OOPS_TA_OK : OOPS_TA_CUDA_ERROR;
}

// dtype of the activations and of the affine parameters: the same, or f32 parameters with 16-bit activations
template <typename F>
int ln_dispatch(int dtype, int affine_dtype, F&& run) {
  if (affine_dtype != dtype && affine_dtype != OOPS_TA_F32) return OOPS_TA_UNSUPPORTED_DTYPE;
  const bool master = affine_dtype == OOPS_TA_F32;
  switch (dtype) {
    case OOPS_TA_F32: return run(float{}, float{});
    case OOPS_TA_F16: return master ? run(__half{}, float{}) : run(__half{}, __half{});
    case OOPS_TA_BF16: return master ? run(__nv_bfloat16{}, float{}) : run(__nv_bfloat16{}, __nv_bfloat16{});
    default: return OOPS_TA_UNSUPPORTED_DTYPE;
  }
}

}  // namespace

uint64_t layer_norm_backward_workspace_bytes(int64_t rows, int width) {
  if (rows <= 0 || width <= 0) return 0;
  // cached rows: one partial row per CTA, and no launch has more CTAs than ln_grid of the row count
  const int64_t parts = width <= kLnCached ? ln_grid(rows) : (rows < kLnWideParts ? rows : kLnWideParts);
  return uint64_t(2) * uint64_t(parts) * uint64_t(width) * sizeof(float);
}

int layer_norm_max_width() { return kLnMaxWidth; }

int reduce_parameter_parts(int affine_dtype, const float* dw_parts, const float* db_parts, int num_parts, int width, void* dweight,
                           void* dbias, cudaStream_t stream) {
  return ln_dispatch(affine_dtype, affine_dtype, [&](auto, auto a) {
    using A = decltype(a);
    layer_norm_reduce_parts_kernel<A><<<dim3((width + 31) / 32, 2), 256, 0, stream>>>(
        dw_parts, db_parts, num_parts, width, reinterpret_cast<A*>(dweight), reinterpret_cast<A*>(dbias));
    count_launch();
    return check_launch("parameter gradient reduction");
  });
}

int layer_norm_forward(int dtype, int affine_dtype, int64_t rows, int width, const void* x, int64_t x_stride, const void* weight,
                       const void* bias, float eps, void* y, int64_t y_stride, float* mean, float* rstd, cudaStream_t stream) {
  if (rows == 0) return OOPS_TA_OK;
  const LnShape s{rows, width, x_stride, y_stride, 0, 0};
  return ln_dispatch(dtype, affine_dtype, [&](auto t, auto a) {
    return forward_typed<decltype(t), decltype(a)>(s, x, weight, bias, eps, y, mean, rstd, stream);
  });
}

int layer_norm_backward(int dtype, int affine_dtype, int64_t rows, int width, const void* dy, int64_t dy_stride, const void* x,
                        int64_t x_stride, const void* weight, const float* mean, const float* rstd, void* dx, int64_t dx_stride,
                        void* dweight, void* dbias, void* workspace, cudaStream_t stream) {
  if (rows == 0) return OOPS_TA_OK;
  const LnShape s{rows, width, x_stride, 0, dy_stride, dx_stride};
  return ln_dispatch(dtype, affine_dtype, [&](auto t, auto a) {
    return backward_typed<decltype(t), decltype(a)>(s, dy, x, weight, mean, rstd, dx, dweight, dbias,
                                                    reinterpret_cast<float*>(workspace), stream);
  });
}

}  // namespace oops_ta
