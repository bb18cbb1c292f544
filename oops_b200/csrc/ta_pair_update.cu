// Element-wise and normalisation passes of the triangle multiplicative update, between its library GEMMs (the reference
// composes them from single PyTorch operations: oops/pair/triangle_multiplication/triangle_multiplication.py:45-141).
//
// The projections want tokens as rows and channels contiguous ("token-major", (prefix * N * N, channels)); the O(N^3)
// contraction is one N x N product per channel and wants every channel as a plane ("channel-major",
// (prefix * hidden, Np, Np) with Np = N rounded up to 8, so that the GEMM rows stay 16-byte aligned for every N; the
// padding is written as zeros and contributes nothing).  Every pass below therefore moves between the two layouts
// through a shared-memory tile while it does its arithmetic, and reads and writes each operand once:
//   pair_gate_forward    left, right = mask * sigmoid(gate) * value            token-major -> channel-major
//   pair_gate_backward   the gradients of the four projections                channel-major -> token-major
//   channel_norm_forward layer norm over the channels of the update            channel-major -> token-major
//   channel_norm_backward its reverse pass and the parameter gradients         token-major -> channel-major
//   output_gate_*        out = values * sigmoid(gate) and its reverse pass     token-major
// All are bound by HBM.  A shared tile is 32 words wide: a word is two neighbouring tokens of a 16-bit type or one f32
// token, so that a warp's row of a plane is 128 contiguous bytes whatever the type, and a warp's token-major access is
// four lanes of 16 bytes on each of eight tokens; with 33 words between tile rows neither side has bank conflicts.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "ta_internal.h"

namespace oops_ta {
namespace {

constexpr int kPitch = 33;          // words between the rows of a shared tile
constexpr int kMaxHidden = 512;     // channels of a tile that holds whole tokens
constexpr int kNormThreads = 256;

template <typename T>
constexpr int tokens_per_word() { return sizeof(T) == 2 ? 2 : 1; }

struct PairShape {
  int prefix, tokens, padded, hidden;
  __host__ __device__ int64_t plane() const { return int64_t(padded) * padded; }
};

template <typename T>
__device__ __forceinline__ float sigmoid_of(float g) {
  // 16-bit results round far above the error of the fast exponential
  if constexpr (sizeof(T) == 4) return 1.f / (1.f + expf(-g));
  return __fdividef(1.f, 1.f + __expf(-g));
}

// Eight consecutive channels of a token; `n` of them exist.  VEC: all eight exist and the address is 16-byte aligned.
template <typename T, bool VEC>
__device__ __forceinline__ void load8(const T* p, int n, float (&out)[8]) {
  if constexpr (VEC && sizeof(T) == 2) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = float(e[i]);
  } else if constexpr (VEC) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
    out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = i < n ? float(p[i]) : 0.f;
  }
}

// The same as they were loaded, so that several can be under way without eight registers each (VEC; element by element, packing waits for each).
template <typename T, bool VEC>
struct Raw8 {
  uint4 words[sizeof(T) / 2];
  __device__ __forceinline__ void load(const T* p, int n, bool take) {
#pragma unroll
    for (int i = 0; i < int(sizeof(T) / 2); ++i) words[i] = take ? reinterpret_cast<const uint4*>(p)[i] : make_uint4(0, 0, 0, 0);
  }
  __device__ __forceinline__ float operator[](int i) const { return float(reinterpret_cast<const T*>(words)[i]); }
};
template <typename T>
struct Raw8<T, false> {
  float values[8];
  __device__ __forceinline__ void load(const T* p, int n, bool take) {
    if (take) {
      load8<T, false>(p, n, values);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) values[i] = 0.f;
    }
  }
  __device__ __forceinline__ float operator[](int i) const { return values[i]; }
};

template <typename T, bool VEC>
__device__ __forceinline__ void store8(T* p, int n, const float (&in)[8]) {
  if constexpr (VEC && sizeof(T) == 2) {
    uint4 v;
    T* e = reinterpret_cast<T*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = T(in[i]);
    *reinterpret_cast<uint4*>(p) = v;
  } else if constexpr (VEC) {
    reinterpret_cast<float4*>(p)[0] = make_float4(in[0], in[1], in[2], in[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(in[4], in[5], in[6], in[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n) p[i] = T(in[i]);
  }
}

// A tile word from the values of its tokens, and back.
template <typename T>
__device__ __forceinline__ uint32_t to_word(const float* tokens) {
  if constexpr (sizeof(T) == 4) {
    return __float_as_uint(tokens[0]);
  } else {
    const T pair[2] = {T(tokens[0]), T(tokens[1])};
    return *reinterpret_cast<const uint32_t*>(pair);
  }
}
template <typename T>
__device__ __forceinline__ void from_word(uint32_t word, float* tokens) {
  if constexpr (sizeof(T) == 4) {
    tokens[0] = __uint_as_float(word);
  } else {
    const T* pair = reinterpret_cast<const T*>(&word);
    tokens[0] = float(pair[0]);
    tokens[1] = float(pair[1]);
  }
}

// Token index (prefix element b included) of padded plane position `p`, or -1 in the padding.
__device__ __forceinline__ int64_t token_at(const PairShape& s, int b, int64_t p) {
  const uint32_t i = uint32_t(p) / uint32_t(s.padded), j = uint32_t(p) - i * uint32_t(s.padded);
  return i < uint32_t(s.tokens) && j < uint32_t(s.tokens) ? (int64_t(b) * s.tokens + i) * s.tokens + j : -1;
}

// ---------------------------------------------------------------------------------------------
// gated projections
// ---------------------------------------------------------------------------------------------
// Row m of `proj` holds [left gate | left value | right gate | right value | ...], `hidden` channels each.
// The channels of `left` and `right`, each rounded up to eight, form one axis.  CTA = (32 words of tokens, 64 of that axis,
// prefix element): a token's piece of a projection is then 128 contiguous bytes of a 16-bit type (64-byte pieces: 55 and
// 90 us forward and reverse at N = 384, 128 channels).  Pieces are kept as they were loaded until the arithmetic needs them: converted at
// once, a token's loads waited for those of the token before, and the reverse spilled 60 bytes a thread at five CTAs per SM (51.4 and 78.2 us;
// now 48.3 with eight CTAs and 62.2 with six, where a 16-bit thread spills 4, of 34.5 and 57.6 at the copy's rate); an f32 word is one token, whose forward pass gains nothing by it: N = 384, 64 channels, 42.9 us and 44.3).  The channel chunk is the
// fastest index: neighbouring CTAs touch a token's other pieces while their pages are open.

struct GateTile {  // rows = channels; rows 32 .. 63 stand four words on, so that a warp's eight channel groups miss each other's banks
  uint32_t words[64 * kPitch + 4];
  __device__ __forceinline__ uint32_t& at(int row, int word) { return words[row * kPitch + (row >> 5) * 4 + word]; }
};

// Where channel group `o` (the first of eight) of the common axis lies: its side, channel within the side, and how many of
// the eight exist.
struct GateGroup {
  int side, channel, n;
  __device__ GateGroup(const PairShape& s, int o) {
    const int rounded = (s.hidden + 7) / 8 * 8;
    side = o >= rounded;
    channel = o - side * rounded;
    n = o < 2 * rounded ? s.hidden - channel : 0;
  }
};
__host__ __device__ inline int gate_chunks(int hidden) { return (2 * ((hidden + 7) / 8 * 8) + 63) / 64; }

template <typename T, bool VEC>
__global__ void __launch_bounds__(256, 8) pair_gate_forward_kernel(PairShape s, const T* __restrict__ proj, int64_t ld,
                                                                const T* __restrict__ mask, uint32_t* __restrict__ left,
                                                                uint32_t* __restrict__ right) {
  constexpr int W = tokens_per_word<T>();
  __shared__ GateTile tile;
  const int chunks = gate_chunks(s.hidden), chunk = blockIdx.x % chunks, b = blockIdx.y;
  const int64_t first = int64_t(blockIdx.x / chunks) * 32;  // first word of the tile in a plane
  const int cg = threadIdx.x & 7, word = threadIdx.x >> 3;
  const GateGroup own(s, chunk * 64 + cg * 8);
  if constexpr (VEC && W == 2) {
    Raw8<T, VEC> gate[W], value[W];
    float weight[W];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const int64_t m = token_at(s, b, (first + word) * W + e);
      const bool there = m >= 0 && own.n > 0;
      const T* row = proj + m * ld + own.side * 2 * s.hidden + own.channel;
      gate[e].load(row, own.n, there);
      value[e].load(row + s.hidden, own.n, there);
      weight[e] = !there ? 0.f : mask ? float(mask[m]) : 1.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float both[2];
#pragma unroll
      for (int e = 0; e < W; ++e) both[e] = weight[e] * sigmoid_of<T>(gate[e][i]) * value[e][i];
      tile.at(cg * 8 + i, word) = to_word<T>(both);
    }
  } else {
    float out[W][8];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const int64_t m = token_at(s, b, (first + word) * W + e);
      float gate[8], value[8];
      if (m >= 0 && own.n > 0) {
        const T* row = proj + m * ld + own.side * 2 * s.hidden + own.channel;
        load8<T, VEC>(row, own.n, gate);
        load8<T, VEC>(row + s.hidden, own.n, value);
        const float weight = mask ? float(mask[m]) : 1.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) out[e][i] = weight * sigmoid_of<T>(gate[i]) * value[i];
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[e][i] = 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float both[2] = {out[0][i], out[W - 1][i]};
      tile.at(cg * 8 + i, word) = to_word<T>(both);
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t words = s.plane() / W;
#pragma unroll
  for (int i = 0; i < 8; ++i) {  // a warp's eight rows are one channel group
    const GateGroup group(s, chunk * 64 + (threadIdx.x >> 5) * 8);
    if (i < group.n)
      (group.side ? right : left)[(int64_t(b) * s.hidden + group.channel + i) * words + first + lane] =
          tile.at((threadIdx.x >> 5) * 8 + i, lane);
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(256, VEC ? 6 : 4) pair_gate_backward_kernel(PairShape s, const T* __restrict__ proj, int64_t ld,
                                                                 const T* __restrict__ mask, const uint32_t* __restrict__ dleft,
                                                                 const uint32_t* __restrict__ dright, T* __restrict__ dproj,
                                                                 int64_t ld_d) {
  constexpr int W = tokens_per_word<T>();
  __shared__ GateTile tile;
  const int chunks = gate_chunks(s.hidden), chunk = blockIdx.x % chunks, b = blockIdx.y;
  const int64_t first = int64_t(blockIdx.x / chunks) * 32;
  {
    const int lane = threadIdx.x & 31;
    const int64_t words = s.plane() / W;
    const GateGroup group(s, chunk * 64 + (threadIdx.x >> 5) * 8);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      tile.at((threadIdx.x >> 5) * 8 + i, lane) =
          i < group.n ? (group.side ? dright : dleft)[(int64_t(b) * s.hidden + group.channel + i) * words + first + lane] : 0u;
  }
  const int cg = threadIdx.x & 7, word = threadIdx.x >> 3;
  const GateGroup own(s, chunk * 64 + cg * 8);
  constexpr bool kWords = VEC || W == 1;
  Raw8<T, VEC> gate[W], value[W];
  float weight[W];
  int64_t at[W];
#pragma unroll
  for (int e = 0; e < W; ++e) {
    const int64_t m = own.n > 0 ? token_at(s, b, (first + word) * W + e) : -1;
    at[e] = m;
    const T* row = proj + m * ld + own.side * 2 * s.hidden + own.channel;
    if (kWords) {
      gate[e].load(row, own.n, m >= 0);
      value[e].load(row + s.hidden, own.n, m >= 0);
      weight[e] = m < 0 ? 0.f : mask ? float(mask[m]) : 1.f;
    } else if (m >= 0) {  // element by element one branch for all of a token's loads, which would otherwise be converted before the next ones
      gate[e].load(row, own.n, true);
      value[e].load(row + s.hidden, own.n, true);
      weight[e] = mask ? float(mask[m]) : 1.f;
    }
  }
  __syncthreads();
  float grad[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if constexpr (kWords) grad[i][0] = __uint_as_float(tile.at(cg * 8 + i, word));  // (a word, split where it is needed)
    else from_word<T>(tile.at(cg * 8 + i, word), grad[i]);
  }
#pragma unroll
  for (int e = 0; e < W; ++e) {
    if (at[e] < 0) continue;
    float dgate[8], dvalue[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float both[2];
      if constexpr (kWords) from_word<T>(__float_as_uint(grad[i][0]), both);
      else both[e] = grad[i][e];
      const float sg = sigmoid_of<T>(gate[e][i]), up = both[e] * weight[e];
      dvalue[i] = up * sg;
      dgate[i] = up * value[e][i] * sg * (1.f - sg);
    }
    T* row = dproj + at[e] * ld_d + own.side * 2 * s.hidden + own.channel;
    store8<T, VEC>(row, own.n, dgate);
    store8<T, VEC>(row + s.hidden, own.n, dvalue);
  }
}

// ---------------------------------------------------------------------------------------------
// layer norm over the channels of the update
// ---------------------------------------------------------------------------------------------
// A CTA holds 32 words of tokens with all their channels in shared memory.  Statistics: warp w sums channels w, w + 8, ...
// of the lane's word, the eight partial sums meet in shared memory; the variance is a second pass over centred values.

template <typename A>
__device__ __forceinline__ float affine_of(const void* p, int i, float missing) {
  return p ? float(reinterpret_cast<const A*>(p)[i]) : missing;
}

// Parameters c .. c + 7 (c is a multiple of eight).
template <typename A>
__device__ __forceinline__ void affine8(const void* p, int c, float missing, float (&out)[8]) {
  const A* from = reinterpret_cast<const A*>(p) + c;
  if (p && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    load8<A, true>(from, 8, out);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = p ? float(from[i]) : missing;
  }
}

// Sum over the eight warps of a per-(warp, lane) pair of values; every thread gets its lane's total.
template <int W>
__device__ __forceinline__ void sum_over_warps(float (&v)[W], float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
#pragma unroll
  for (int e = 0; e < W; ++e) scratch[(warp * W + e) * 32 + lane] = v[e];
  __syncthreads();
#pragma unroll
  for (int e = 0; e < W; ++e) {
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < kNormThreads / 32; ++w) total += scratch[(w * W + e) * 32 + lane];
    v[e] = total;
  }
}

template <typename T, typename A, bool VEC>
__global__ void __launch_bounds__(kNormThreads) channel_norm_forward_kernel(PairShape s, const uint32_t* __restrict__ update,
                                                                            const void* __restrict__ weight,
                                                                            const void* __restrict__ bias, float eps,
                                                                            T* __restrict__ y, float* __restrict__ mean_out,
                                                                            float* __restrict__ rstd_out) {
  constexpr int W = tokens_per_word<T>();
  extern __shared__ uint32_t norm_smem[];
  uint32_t* tile = norm_smem;                                                    // [hidden][kPitch]
  float* scratch = reinterpret_cast<float*>(tile + s.hidden * kPitch);           // [8][W][32]
  float* stats = scratch + 8 * W * 32;                                           // [2][W][32]: mean, rstd
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.y;
  const int64_t words = s.plane() / W;
  const uint32_t* src = update + int64_t(b) * s.hidden * words + int64_t(blockIdx.x) * 32 + lane;
  float sum[W];
#pragma unroll
  for (int e = 0; e < W; ++e) sum[e] = 0.f;
#pragma unroll 8
  for (int c = warp; c < s.hidden; c += 8) {
    const uint32_t word = src[int64_t(c) * words];
    tile[c * kPitch + lane] = word;
    float v[2];
    from_word<T>(word, v);
#pragma unroll
    for (int e = 0; e < W; ++e) sum[e] += v[e];
  }
  sum_over_warps<W>(sum, scratch);
  const float inv = 1.f / float(s.hidden);
  float sq[W];
#pragma unroll
  for (int e = 0; e < W; ++e) {
    sum[e] *= inv;
    sq[e] = 0.f;
  }
#pragma unroll 4
  for (int c = warp; c < s.hidden; c += 8) {
    float v[2];
    from_word<T>(tile[c * kPitch + lane], v);
#pragma unroll
    for (int e = 0; e < W; ++e) sq[e] += (v[e] - sum[e]) * (v[e] - sum[e]);
  }
  sum_over_warps<W>(sq, scratch);
  if (warp == 0) {
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const float rstd = rsqrtf(sq[e] * inv + eps);
      stats[e * 32 + lane] = sum[e];
      stats[(W + e) * 32 + lane] = rstd;
      const int64_t m = token_at(s, b, (int64_t(blockIdx.x) * 32 + lane) * W + e);
      if (m >= 0) {
        mean_out[m] = sum[e];
        rstd_out[m] = rstd;
      }
    }
  }
  __syncthreads();
  const int cg = threadIdx.x & 3, word = (threadIdx.x >> 2) & 31;
  int64_t at[W];
#pragma unroll
  for (int e = 0; e < W; ++e) at[e] = token_at(s, b, (int64_t(blockIdx.x) * 32 + word) * W + e);
  for (int c = (threadIdx.x >> 7) * 32 + cg * 8; c < s.hidden; c += 64) {
    float v[8][2], w[8], offset[8];  // parameters once for all of the word's tokens (fetched one by one for each: 23.5 us at N = 384, now 21.8)
    if constexpr (VEC) {
      affine8<A>(weight, c, 1.f, w);
      affine8<A>(bias, c, 0.f, offset);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (VEC || c + i < s.hidden) from_word<T>(tile[(c + i) * kPitch + word], v[i]);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      if (at[e] < 0) continue;
      const float mean = stats[e * 32 + word], rstd = stats[(W + e) * 32 + word];
      float out[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        out[i] = VEC || c + i < s.hidden
                     ? (v[i][e] - mean) * rstd * (VEC ? w[i] : affine_of<A>(weight, c + i, 1.f)) + (VEC ? offset[i] : affine_of<A>(bias, c + i, 0.f))
                     : 0.f;
      store8<T, VEC>(y + at[e] * s.hidden + c, s.hidden - c, out);
    }
  }
}

// Reverse pass: g = dy * weight, xhat = (u - mean) * rstd, du = rstd * (g - mean_c(g) - xhat * mean_c(g * xhat)).
// The CTA walks tiles so that a thread can carry the parameter gradients of its channels in registers (a thread owns up
// to four channels on one half of a tile's words); per-CTA partial rows are added in a fixed order by a second launch.
template <typename T, typename A, bool VEC>
__global__ void __launch_bounds__(kNormThreads, 4) channel_norm_backward_kernel(
    PairShape s, int64_t tiles_per_prefix, const T* __restrict__ dy, const uint32_t* __restrict__ update,
    const void* __restrict__ weight, const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
    uint32_t* __restrict__ dupdate, float* __restrict__ dw_parts, float* __restrict__ db_parts) {
  constexpr int W = tokens_per_word<T>(), kOwn = kMaxHidden / 128;
  extern __shared__ uint32_t norm_smem[];
  uint32_t* tile_u = norm_smem;                                                  // [hidden][kPitch]
  uint32_t* tile_g = tile_u + s.hidden * kPitch;                                 // [hidden][kPitch]: dy
  float* scratch = reinterpret_cast<float*>(tile_g + s.hidden * kPitch);         // [8][2 * W][32]
  float* stats = scratch + 8 * 2 * W * 32;                                       // [2][W][32]
  float* affine = stats + 2 * W * 32;                                            // [hidden] weight
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = s.plane() / W;
  const float inv = 1.f / float(s.hidden);
  float dw[kOwn], db[kOwn];
#pragma unroll
  for (int k = 0; k < kOwn; ++k) dw[k] = db[k] = 0.f;
  for (int c = threadIdx.x; c < s.hidden; c += kNormThreads) affine[c] = affine_of<A>(weight, c, 1.f);

  for (int64_t tile = blockIdx.x; tile < tiles_per_prefix * s.prefix; tile += gridDim.x) {
    const int b = int(tile / tiles_per_prefix);
    const int64_t first = (tile - int64_t(b) * tiles_per_prefix) * 32;  // first word of the tile in a plane
    __syncthreads();  // the previous tile's words are no longer read
    const int64_t plane_at = int64_t(b) * s.hidden * words + first + lane;
#pragma unroll 8
    for (int c = warp; c < s.hidden; c += 8) tile_u[c * kPitch + lane] = update[plane_at + int64_t(c) * words];
    {
      const int cg = threadIdx.x & 3, word = (threadIdx.x >> 2) & 31;
      int64_t at[W];
#pragma unroll
      for (int e = 0; e < W; ++e) at[e] = token_at(s, b, (first + word) * W + e);
      for (int c = (threadIdx.x >> 7) * 32 + cg * 8; c < s.hidden; c += 64) {
        float g[2][8];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (at[e] >= 0) {
            load8<T, VEC>(dy + at[e] * s.hidden + c, s.hidden - c, g[e]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) g[e][i] = 0.f;
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (VEC || c + i < s.hidden) {
            const float both[2] = {g[0][i], g[W - 1][i]};
            tile_g[(c + i) * kPitch + word] = to_word<T>(both);
          }
        }
      }
    }
    float mean[W], rstd[W], sums[2 * W];  // sums over the channels of g * xhat (first W) and of g
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const int64_t m = token_at(s, b, (first + lane) * W + e);
      mean[e] = m >= 0 ? mean_in[m] : 0.f;
      rstd[e] = m >= 0 ? rstd_in[m] : 0.f;
      sums[e] = sums[W + e] = 0.f;
      if (warp == 0) {
        stats[e * 32 + lane] = mean[e];
        stats[(W + e) * 32 + lane] = rstd[e];
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int c = warp; c < s.hidden; c += 8) {
      float u[2], g[2];
      from_word<T>(tile_u[c * kPitch + lane], u);
      from_word<T>(tile_g[c * kPitch + lane], g);
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const float gw = g[e] * affine[c];
        sums[e] += gw * (u[e] - mean[e]) * rstd[e];
        sums[W + e] += gw;
      }
    }
    sum_over_warps<2 * W>(sums, scratch);
#pragma unroll 4
    for (int c = warp; c < s.hidden; c += 8) {
      float u[2], g[2], out[2];
      from_word<T>(tile_u[c * kPitch + lane], u);
      from_word<T>(tile_g[c * kPitch + lane], g);
#pragma unroll
      for (int e = 0; e < W; ++e)
        out[e] = rstd[e] * (g[e] * affine[c] - sums[W + e] * inv - (u[e] - mean[e]) * rstd[e] * sums[e] * inv);
      dupdate[plane_at + int64_t(c) * words] = to_word<T>(out);
    }
    if (dw_parts || db_parts) {
      const int half = threadIdx.x >> 7;
#pragma unroll
      for (int k = 0; k < kOwn; ++k) {
        const int c = (threadIdx.x & 127) + 128 * k;
        if (c >= s.hidden) break;
#pragma unroll 4
        for (int w = half * 16; w < half * 16 + 16; ++w) {
          float u[2], g[2];
          from_word<T>(tile_u[c * kPitch + w], u);
          from_word<T>(tile_g[c * kPitch + w], g);
#pragma unroll
          for (int e = 0; e < W; ++e) {
            dw[k] += g[e] * (u[e] - stats[e * 32 + w]) * stats[(W + e) * 32 + w];
            db[k] += g[e];
          }
        }
      }
    }
  }
  if (dw_parts || db_parts) {
    float* halves = reinterpret_cast<float*>(tile_u);  // [2][hidden]: the sums of the upper half of the words
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
      const int c = (threadIdx.x & 127) + 128 * k;
      if (c < s.hidden && threadIdx.x >= 128) {
        halves[c] = dw[k];
        halves[s.hidden + c] = db[k];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
      const int c = (threadIdx.x & 127) + 128 * k;
      if (c < s.hidden && threadIdx.x < 128) {
        if (dw_parts) dw_parts[int64_t(blockIdx.x) * s.hidden + c] = dw[k] + halves[c];
        if (db_parts) db_parts[int64_t(blockIdx.x) * s.hidden + c] = db[k] + halves[s.hidden + c];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// output gate
// ---------------------------------------------------------------------------------------------
// One thread per eight channels of a token.

template <typename T, bool VEC>
__global__ void __launch_bounds__(256) output_gate_forward_kernel(int64_t rows, int channels, const T* __restrict__ values,
                                                                  const T* __restrict__ gate, int64_t gate_ld,
                                                                  T* __restrict__ out) {
  const int groups = (channels + 7) / 8;
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * groups) return;
  const int64_t row = i / groups;
  const int c = int(i - row * groups) * 8, n = channels - c;
  float v[8], g[8];
  load8<T, VEC>(values + row * channels + c, n, v);
  load8<T, VEC>(gate + row * gate_ld + c, n, g);
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] *= sigmoid_of<T>(g[e]);
  store8<T, VEC>(out + row * channels + c, n, v);
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(256) output_gate_backward_kernel(int64_t rows, int channels, const T* __restrict__ dout,
                                                                   const T* __restrict__ values, const T* __restrict__ gate,
                                                                   int64_t gate_ld, T* __restrict__ dvalues,
                                                                   T* __restrict__ dgate, int64_t dgate_ld) {
  const int groups = (channels + 7) / 8;
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * groups) return;
  const int64_t row = i / groups;
  const int c = int(i - row * groups) * 8, n = channels - c;
  float v[8], g[8], up[8];
  load8<T, VEC>(values + row * channels + c, n, v);
  load8<T, VEC>(gate + row * gate_ld + c, n, g);
  load8<T, VEC>(dout + row * channels + c, n, up);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float sg = sigmoid_of<T>(g[e]);
    g[e] = up[e] * v[e] * sg * (1.f - sg);
    up[e] *= sg;
  }
  store8<T, VEC>(dvalues + row * channels + c, n, up);
  store8<T, VEC>(dgate + row * dgate_ld + c, n, g);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int check_pair_shape(const PairShape& s) {
  if (s.prefix <= 0 || s.tokens <= 0 || s.hidden <= 0)
    return fail(OOPS_TA_INVALID_ARGUMENT, "empty dimension (prefix=%d tokens=%d hidden=%d)", s.prefix, s.tokens, s.hidden);
  if (s.padded < s.tokens || s.padded % 8 != 0)
    return fail(OOPS_TA_INVALID_ARGUMENT, "padded %d must be a multiple of 8 not below tokens %d", s.padded, s.tokens);
  if (s.prefix > 65535 || s.plane() > 0x7fffffffll || s.plane() / 32 * ceil_div(s.hidden, 32) > 0x7fffffffll)
    return fail(OOPS_TA_LIMIT_EXCEEDED, "prefix=%d padded=%d hidden=%d exceed a launch", s.prefix, s.padded, s.hidden);
  return OOPS_TA_OK;
}

template <typename F>
int by_type(int dtype, F&& run) {
  switch (dtype) {
    case OOPS_TA_F32: return run(float{});
    case OOPS_TA_F16: return run(__half{});
    case OOPS_TA_BF16: return run(__nv_bfloat16{});
    default: return fail(OOPS_TA_UNSUPPORTED_DTYPE, "dtype %d is not f32/f16/bf16", dtype);
  }
}

template <typename F>
int by_types(int dtype, int affine_dtype, F&& run) {
  if (affine_dtype != dtype && affine_dtype != OOPS_TA_F32)
    return fail(OOPS_TA_UNSUPPORTED_DTYPE, "parameter dtype %d with activations of dtype %d", affine_dtype, dtype);
  return by_type(dtype, [&](auto t) -> int {
    using T = decltype(t);
    return affine_dtype == OOPS_TA_F32 ? run(t, float{}) : run(t, T{});
  });
}

template <typename T>
size_t norm_smem_bytes(const PairShape& s, int tiles, bool affine) {
  constexpr int W = tokens_per_word<T>();
  return (size_t(tiles) * s.hidden * kPitch + 8 * tiles * W * 32 + 2 * W * 32 + (affine ? s.hidden : 0)) * 4;
}

int64_t norm_grid(const PairShape& s, int dtype) {
  const int64_t tiles = s.plane() / (dtype == OOPS_TA_F32 ? 32 : 64) * s.prefix;
  return std::min<int64_t>(tiles, 148 * 4);
}

}  // namespace

int channel_norm_max_width() { return kMaxHidden; }

int pair_gate_forward(int dtype, int prefix, int tokens, int padded, int hidden, const void* proj, int64_t ld, const void* mask,
                      void* left, void* right, cudaStream_t stream) {
  const PairShape s{prefix, tokens, padded, hidden};
  int status = check_pair_shape(s);
  if (status) return status;
  return by_type(dtype, [&](auto t) -> int {
    using T = decltype(t);
    constexpr int kVec = 16 / int(sizeof(T));
    const bool vec = hidden % 8 == 0 && ld % kVec == 0 && aligned16(proj);
    const dim3 grid((unsigned)(s.plane() / (32 * tokens_per_word<T>()) * gate_chunks(hidden)), (unsigned)prefix);
    auto kernel = vec ? pair_gate_forward_kernel<T, true> : pair_gate_forward_kernel<T, false>;
    kernel<<<grid, 256, 0, stream>>>(s, reinterpret_cast<const T*>(proj), ld, reinterpret_cast<const T*>(mask),
                                     reinterpret_cast<uint32_t*>(left), reinterpret_cast<uint32_t*>(right));
    count_launch();
    return check_launch("pair gate forward");
  });
}

int pair_gate_backward(int dtype, int prefix, int tokens, int padded, int hidden, const void* proj, int64_t ld, const void* mask,
                       const void* dleft, const void* dright, void* dproj, int64_t ld_d, cudaStream_t stream) {
  const PairShape s{prefix, tokens, padded, hidden};
  int status = check_pair_shape(s);
  if (status) return status;
  return by_type(dtype, [&](auto t) -> int {
    using T = decltype(t);
    constexpr int kVec = 16 / int(sizeof(T));
    const bool vec = hidden % 8 == 0 && ld % kVec == 0 && ld_d % kVec == 0 && aligned16(proj) && aligned16(dproj);
    const dim3 grid((unsigned)(s.plane() / (32 * tokens_per_word<T>()) * gate_chunks(hidden)), (unsigned)prefix);
    auto kernel = vec ? pair_gate_backward_kernel<T, true> : pair_gate_backward_kernel<T, false>;
    kernel<<<grid, 256, 0, stream>>>(s, reinterpret_cast<const T*>(proj), ld, reinterpret_cast<const T*>(mask),
                                     reinterpret_cast<const uint32_t*>(dleft), reinterpret_cast<const uint32_t*>(dright),
                                     reinterpret_cast<T*>(dproj), ld_d);
    count_launch();
    return check_launch("pair gate backward");
  });
}

int channel_norm_forward(int dtype, int affine_dtype, int prefix, int tokens, int padded, int hidden, const void* update,
                         const void* weight, const void* bias, float eps, void* y, float* mean, float* rstd, cudaStream_t stream) {
  const PairShape s{prefix, tokens, padded, hidden};
  int status = check_pair_shape(s);
  if (status) return status;
  return by_types(dtype, affine_dtype, [&](auto t, auto a) -> int {
    using T = decltype(t);
    using A = decltype(a);
    const bool vec = hidden % 8 == 0 && aligned16(y);
    const size_t smem = norm_smem_bytes<T>(s, 1, false);
    auto kernel = vec ? channel_norm_forward_kernel<T, A, true> : channel_norm_forward_kernel<T, A, false>;
    if (smem > 48 * 1024) {
      const int rc = reserve_dynamic_smem(reinterpret_cast<const void*>(kernel), int(smem));
      if (rc) return rc;
    }
    const dim3 grid((unsigned)(s.plane() / (32 * tokens_per_word<T>())), (unsigned)prefix);
    kernel<<<grid, kNormThreads, smem, stream>>>(s, reinterpret_cast<const uint32_t*>(update), weight, bias, eps,
                                                 reinterpret_cast<T*>(y), mean, rstd);
    count_launch();
    return check_launch("channel norm forward");
  });
}

uint64_t channel_norm_backward_workspace_bytes(int dtype, int prefix, int tokens, int padded, int hidden) {
  const PairShape s{prefix, tokens, padded, hidden};
  if (prefix <= 0 || padded <= 0 || hidden <= 0) return 0;
  return uint64_t(2) * norm_grid(s, dtype) * hidden * sizeof(float);
}

int channel_norm_backward(int dtype, int affine_dtype, int prefix, int tokens, int padded, int hidden, const void* dy,
                          const void* update, const void* weight, const float* mean, const float* rstd, void* dupdate,
                          void* dweight, void* dbias, float* workspace, cudaStream_t stream) {
  const PairShape s{prefix, tokens, padded, hidden};
  int status = check_pair_shape(s);
  if (status) return status;
  const int64_t grid = norm_grid(s, dtype);
  float* dw_parts = dweight ? workspace : nullptr;
  float* db_parts = dbias ? workspace + grid * hidden : nullptr;
  status = by_types(dtype, affine_dtype, [&](auto t, auto a) -> int {
    using T = decltype(t);
    using A = decltype(a);
    const bool vec = hidden % 8 == 0 && aligned16(dy);
    const size_t smem = norm_smem_bytes<T>(s, 2, true);
    auto kernel = vec ? channel_norm_backward_kernel<T, A, true> : channel_norm_backward_kernel<T, A, false>;
    if (smem > 48 * 1024) {
      const int rc = reserve_dynamic_smem(reinterpret_cast<const void*>(kernel), int(smem));
      if (rc) return rc;
    }
    kernel<<<(unsigned)grid, kNormThreads, smem, stream>>>(s, s.plane() / (32 * tokens_per_word<T>()),
                                                           reinterpret_cast<const T*>(dy), reinterpret_cast<const uint32_t*>(update),
                                                           weight, mean, rstd, reinterpret_cast<uint32_t*>(dupdate), dw_parts,
                                                           db_parts);
    count_launch();
    return check_launch("channel norm backward");
  });
  if (status || (!dweight && !dbias)) return status;
  return reduce_parameter_parts(affine_dtype, dw_parts, db_parts, int(grid), hidden, dweight, dbias, stream);
}

int output_gate_forward(int dtype, int64_t rows, int channels, const void* values, const void* gate, int64_t gate_ld, void* out,
                        cudaStream_t stream) {
  if (rows <= 0 || channels <= 0) return fail(OOPS_TA_INVALID_ARGUMENT, "empty output gate");
  return by_type(dtype, [&](auto t) -> int {
    using T = decltype(t);
    const bool vec = channels % 8 == 0 && gate_ld % (16 / int(sizeof(T))) == 0 && aligned16(values) && aligned16(gate) && aligned16(out);
    const int64_t blocks = ceil_div(rows * ceil_div(channels, 8), 256);
    if (blocks > 0x7fffffffll) return fail(OOPS_TA_LIMIT_EXCEEDED, "output gate of %lld rows", (long long)rows);
    auto kernel = vec ? output_gate_forward_kernel<T, true> : output_gate_forward_kernel<T, false>;
    kernel<<<(unsigned)blocks, 256, 0, stream>>>(rows, channels, reinterpret_cast<const T*>(values), reinterpret_cast<const T*>(gate),
                                                 gate_ld, reinterpret_cast<T*>(out));
    count_launch();
    return check_launch("output gate forward");
  });
}

int output_gate_backward(int dtype, int64_t rows, int channels, const void* dout, const void* values, const void* gate,
                         int64_t gate_ld, void* dvalues, void* dgate, int64_t dgate_ld, cudaStream_t stream) {
  if (rows <= 0 || channels <= 0) return fail(OOPS_TA_INVALID_ARGUMENT, "empty output gate");
  return by_type(dtype, [&](auto t) -> int {
    using T = decltype(t);
    constexpr int kVec = 16 / int(sizeof(T));
    const bool vec = channels % 8 == 0 && gate_ld % kVec == 0 && dgate_ld % kVec == 0 && aligned16(dout) && aligned16(values) &&
                     aligned16(gate) && aligned16(dvalues) && aligned16(dgate);
    const int64_t blocks = ceil_div(rows * ceil_div(channels, 8), 256);
    if (blocks > 0x7fffffffll) return fail(OOPS_TA_LIMIT_EXCEEDED, "output gate of %lld rows", (long long)rows);
    auto kernel = vec ? output_gate_backward_kernel<T, true> : output_gate_backward_kernel<T, false>;
    kernel<<<(unsigned)blocks, 256, 0, stream>>>(rows, channels, reinterpret_cast<const T*>(dout), reinterpret_cast<const T*>(values),
                                                 reinterpret_cast<const T*>(gate), gate_ld, reinterpret_cast<T*>(dvalues),
                                                 reinterpret_cast<T*>(dgate), dgate_ld);
    count_launch();
    return check_launch("output gate backward");
  });
}

}  // namespace oops_ta
